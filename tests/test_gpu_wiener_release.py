"""The Wiener filter's kept workspaces give way: with the rest of the card's
memory taken, a Richardson-Lucy call whose buffers do not fit beside them gets
their memory and gives the same numbers as with the card free."""

import numpy as np
import pytest

from cudadecon_gb300 import synth

pytestmark = pytest.mark.gpu


def test_kept_workspaces_give_way_to_rl(cdx, torch_cuda, tmp_path):
    torch = torch_cuda
    path = tmp_path / "otf.tif"
    synth.write_otf(path, synth.gaussian_otf_table(65, 32, 1.3, 2.5))
    shape, kw = (64, 512, 512), dict(dr=0.104, dz=0.3, dr_psf=0.104, dz_psf=0.2)
    raw = np.random.default_rng(1).integers(90, 400, shape, dtype=np.uint16)
    cdx.rl_init(shape, path, **kw)
    want = cdx.rl_decon(raw, background=100.0, n_iters=2)
    cdx.rl_cleanup()

    cdx.rl_init(shape, path, **kw)
    v = torch.rand((128, 512, 1024), device="cuda") * 500 + 90
    first = cdx.wiener(v, background=100.0, wiener=0.05, NA=1.1, wavelength=0.525)
    with_them = torch.cuda.mem_get_info()[0]
    cdx.rl_cleanup()
    assert torch.cuda.mem_get_info()[0] - with_them > 400 << 20  # two spectra of 32 Mi complex numbers
    cdx.rl_init(shape, path, **kw)
    assert torch.equal(cdx.wiener(v, background=100.0, wiener=0.05, NA=1.1, wavelength=0.525), first)
    torch.cuda.empty_cache()
    # less is left than the call needs (five volumes of floats, the raw stack and a
    # spectrum: 0.4 GB), more than that with the workspaces
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (256 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = cdx.rl_decon(raw, background=100.0, n_iters=2)
    finally:
        del filler
        torch.cuda.empty_cache()
    assert np.array_equal(got, want)
    assert torch.equal(cdx.wiener(v, background=100.0, wiener=0.05, NA=1.1, wavelength=0.525), first)
    cdx.rl_cleanup()
