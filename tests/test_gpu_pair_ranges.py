"""The paired plans at the ends of their ranges and where their form changes.

* 3D transform against numpy in float64, relative L2 <= 2e-6 (the bound the
  other plain transforms are held to): heights of 8 to 31 and above 1024, odd
  ones of two wide and of three radices, with and without room for whole slot
  blocks (189, 225), beside even and odd depths; heights left to the generic
  engine; depths above 256 and of two wide radices.
* The convolution, which takes the columns in the order the forward y pass
  leaves them, with a radial and with a full 3D OTF: same bound.
* RL at 875 columns (three pairs a block) on rows whose last block starts and
  ends on 16 bytes: relative L2 <= 5e-6, the bound of the other paired loops.
"""

import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from cudadecon_gb300 import synth

pytestmark = pytest.mark.gpu

SHAPES = [(6, 8, 128), (5, 9, 135), (4, 12, 128), (7, 14, 128), (3, 10, 140), (6, 15, 128), (5, 27, 150),
          (4, 28, 128), (3, 30, 128), (3, 189, 128), (2, 225, 128), (5, 375, 128), (3, 525, 135),
          (2, 875, 128), (3, 1029, 128), (2, 1080, 128), (3, 1225, 128), (2, 1458, 128), (1, 1875, 128),
          (2, 2025, 128), (3, 2048, 128), (2, 2160, 128), (147, 12, 128), (175, 9, 128), (343, 8, 128),
          (500, 9, 128), (512, 8, 128), (525, 8, 128)]


def _dev(torch, x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


@pytest.mark.parametrize("shape", SHAPES)
def test_transform_and_convolution(cdx, oracle, torch_cuda, tmp_path, shape):
    torch = torch_cuda
    nz, ny, nx = shape
    tab = synth.gaussian_otf_table(65, 32, 1.3, 2.5)
    tab = (tab * np.exp(0.3j * np.arange(32))[None, :]).astype(np.complex64)
    p = tmp_path / "otf.tif"
    synth.write_otf(p, tab)
    cdx.rl_init((32, 32, 128), p, dr=0.1, dz=0.3, dr_psf=0.104, dz_psf=0.25)
    x = np.random.default_rng(nz + 7 * ny + nx).random(shape).astype(np.float32)
    d = _dev(torch, x)
    out = torch.empty_like(d)
    spec = torch.empty((nz, ny, nx // 2 + 1), dtype=torch.complex64, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    L = cdx.lib()
    assert L.cdx_rfft3d_device(ptr(d), ptr(spec), nx, ny, nz, None) == 1, L.cdx_last_error()
    assert L.cdx_conv3d_device(ptr(d), ptr(out), nx, ny, nz, 1, None) == 1, L.cdx_last_error()
    torch.cuda.synchronize()
    cdx.rl_cleanup()
    S = np.fft.rfftn(x.astype(np.float64))
    assert rel_l2(spec.cpu().numpy(), S) < 2e-6
    st = oracle.rl_init(128, 32, 32, 0.1, 0.3, 0.104, 0.25, 0.0, 0.0, 0, False,
                        synth.otf_table_to_image(tab))
    H = np.asarray(oracle.otf_on_grid(st, nx, ny, nz, dtype=np.float32)).reshape(S.shape)
    want = np.fft.irfftn(S * np.conj(H), s=shape, axes=(0, 1, 2))
    assert rel_l2(out.cpu().numpy(), want) < 2e-6


@pytest.mark.parametrize("shape", [(8, 27, 128), (6, 36, 135), (5, 10, 128), (3, 189, 128), (4, 225, 128),
                                   (300, 9, 128), (8, 50, 128)])
@pytest.mark.parametrize("conj", [0, 1])
def test_convolution_with_a_3d_otf(cdx, oracle, torch_cuda, tmp_path, shape, conj):
    torch = torch_cuda
    nz, ny, nx = shape
    grid = np.meshgrid(*[np.fft.fftfreq(n) * n - s for n, s in ((32, 0.3), (64, -0.2), (64, 0.25))],
                       indexing="ij")
    psf = np.exp(-0.5 * sum((g / s) ** 2 for g, s in zip(grid, (2.5, 1.4, 1.4))))
    otf = np.fft.rfftn(psf / psf.sum()).astype(np.complex64)
    img = np.ascontiguousarray(otf).view(np.float32).reshape(32, 64, -1)
    p = tmp_path / "otf3d.tif"
    synth.write_tiff(p, img)
    cdx.rl_init((32, 32, 128), p, dr=0.104, dz=0.3, dr_psf=0.1, dz_psf=0.25)
    x = np.random.default_rng(nz + 7 * ny + nx).random(shape).astype(np.float32)
    d = _dev(torch, x)
    out = torch.empty_like(d)
    L = cdx.lib()
    assert L.cdx_conv3d_device(ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(out.data_ptr()), nx, ny, nz,
                               conj, None) == 1, L.cdx_last_error()
    torch.cuda.synchronize()
    cdx.rl_cleanup()
    st = oracle.rl_init(128, 32, 32, 0.104, 0.3, 0.1, 0.25, 0.0, 0.0, 0, False, img)
    S = np.fft.rfftn(x.astype(np.float64))
    H = np.asarray(oracle.otf_on_grid(st, nx, ny, nz, dtype=np.float32)).reshape(S.shape)
    want = np.fft.irfftn(S * (np.conj(H) if conj else H), s=shape, axes=(0, 1, 2))
    assert rel_l2(out.cpu().numpy(), want) < 2e-6


@pytest.mark.parametrize("shape", [(8, 32, 875), (6, 27, 875), (5, 30, 875)])
def test_rl_with_three_pairs_a_block(cdx, oracle, torch_cuda, tmp_path, shape):
    raw = synth.bead_stack(shape, n_beads=60, psf_sigma_xy=1.3, psf_sigma_z=2.0, seed=sum(shape))
    tab = synth.gaussian_otf_table(65, 32, 1.3, 2.5)
    p = tmp_path / "otf.tif"
    synth.write_otf(p, tab)
    kw = dict(dr=0.104, dz=0.3, dr_psf=0.104, dz_psf=0.25)
    cdx.rl_init(raw.shape, p, **kw)
    assert cdx.decon_grid() == shape
    mine = cdx.rl_decon(raw, background=100.0, n_iters=5)
    cdx.rl_cleanup()
    nz, ny, nx = shape
    st = oracle.rl_init(nx, ny, nz, kw["dr"], kw["dz"], kw["dr_psf"], kw["dz_psf"], 0.0, 0.0, 0,
                        False, synth.otf_table_to_image(tab))
    X0 = oracle.bgsub(raw.astype(np.float32), 100.0)
    want = oracle.rl_iterations(X0, X0, oracle.otf_on_grid(st, nx, ny, nz, dtype=np.float64), 5,
                                dtype=np.float64)
    assert rel_l2(mine, want) < 5e-6
