"""Host batches whose page-locked buffers change from call to call: the copies
of the captured graph follow them, and every call gives the bytes of a batch
whose buffers it sees for the first time."""
import numpy as np
import pytest

from cudadecon_gb300 import synth

pytestmark = pytest.mark.gpu

SHAPES = [(16, 48, 64), (12, 60, 135), (20, 36, 150)]


@pytest.mark.parametrize("n_iters", [0, 3])
def test_host_batch_follows_its_buffers(cdx, torch_cuda, n_iters):
    torch = torch_cuda
    otf = synth.gaussian_otf_table(65, 32, 1.3, 2.5)

    def stacks(seed):
        rng = np.random.default_rng(seed)
        return [dict(raw=torch.from_numpy(rng.integers(90, 900, s, dtype=np.uint16)).pin_memory(), otf=otf, dr=0.104,
                     dz=0.3, dr_psf=0.104, dz_psf=0.25, background=100.0) for s in SHAPES]

    def outs():
        return [torch.full(cdx.batch_grid(s), -1.0).pin_memory() for s in SHAPES]

    sets = [stacks(seed) for seed in range(3)]
    want = []
    for st in sets:
        cdx.lib().cdx_batch_release()
        want.append([o.clone() for o in cdx.rl_batch_host(st, n_iters=n_iters, results=outs())])
    # other inputs, other results, only one of them, in and out of a device batch
    a, b = outs(), outs()
    for which, res in ((0, a), (1, a), (1, b), (2, b), (0, a)):
        for o in res:
            o.fill_(-1.0)
        got = cdx.rl_batch_host(sets[which], n_iters=n_iters, results=res)
        assert all(torch.equal(g, w) for g, w in zip(got, want[which]))
    dev = [dict(d, raw=d["raw"].cuda()) for d in sets[2]]
    got = cdx.rl_batch(dev, n_iters=n_iters)
    torch.cuda.synchronize()
    assert all(torch.equal(g.cpu(), w) for g, w in zip(got, want[2]))
    got = cdx.rl_batch_host(sets[1], n_iters=n_iters, results=b)
    assert all(torch.equal(g, w) for g, w in zip(got, want[1]))
    cdx.lib().cdx_batch_release()
