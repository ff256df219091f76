"""The Wiener filter's kept workspaces: a call gives the same bytes whatever
sizes and streams came before it, and after they were given back."""
import pytest

from cudadecon_gb300 import synth

pytestmark = pytest.mark.gpu

SHAPES = [(32, 64, 64), (100, 128, 150), (21, 50, 64), (64, 96, 128), (32, 64, 64)]


def test_wiener_after_other_sizes(cdx, torch_cuda, tmp_path):
    torch = torch_cuda
    path = tmp_path / "otf.tif"
    synth.write_otf(path, synth.gaussian_otf_table(65, 32, 1.3, 2.5))

    def init(shape):
        cdx.rl_init(shape, path, dr=0.104, dz=0.3, dr_psf=0.104, dz_psf=0.2, deskew_angle=0.0, rotation_angle=0.0)

    gen = torch.Generator(device="cuda").manual_seed(7)
    stacks = [torch.rand(s, device="cuda", generator=gen) * 500 + 90 for s in SHAPES]
    alone = []
    for v in stacks:
        init(v.shape)
        alone.append(cdx.wiener(v, background=100.0, wiener=0.05, NA=1.1, wavelength=0.525))
        cdx.rl_cleanup()
    init(SHAPES[0])
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for i, v in enumerate(stacks * 2):
        with torch.cuda.stream(streams[i % 2]):
            got = cdx.wiener(v, background=100.0, wiener=0.05, NA=1.1, wavelength=0.525)
        torch.cuda.synchronize()
        assert torch.equal(got, alone[i % len(SHAPES)])
    cdx.rl_cleanup()


@pytest.mark.parametrize("shape", [(16, 36, 128), (9, 35, 135), (10, 27, 150), (12, 50, 64)])
def test_wiener_background_in_the_x_pass(cdx, torch_cuda, tmp_path, shape):
    """A background given to the filter equals one taken off before, bit for
    bit: heights whose second half has fewer rows, an odd one, and a width
    that the paired passes do not take."""
    torch = torch_cuda
    path = tmp_path / "otf.tif"
    synth.write_otf(path, synth.gaussian_otf_table(65, 32, 1.3, 2.5))
    cdx.rl_init(shape, path, dr=0.104, dz=0.3, dr_psf=0.104, dz_psf=0.2, deskew_angle=0.0, rotation_angle=0.0)
    gen = torch.Generator(device="cuda").manual_seed(sum(shape))
    v = torch.rand(shape, device="cuda", generator=gen) * 500 + 90
    kw = dict(wiener=0.05, NA=1.1, wavelength=0.525)
    assert torch.equal(cdx.wiener(v, background=100.3, **kw), cdx.wiener(v - 100.3, background=0.0, **kw))
    cdx.rl_cleanup()
