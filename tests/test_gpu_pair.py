"""The paired passes of the plain form (csrc/fft_pair.cuh, decon_p[xyz].cuh) at
the sizes where their dispatch changes or their tiles have remainders.

* 3D transform against numpy in float64, relative L2 <= 2e-6 (the bound the
  other plain transforms are held to): y heights divisible by 4, even, odd, and
  without a plan (generic engine); odd depths (a slice pair of one); depths
  with 8 and 16 column tiles and without a plan; x lengths at both ends of the
  plans and with the twiddles in global memory (1620).
* RL loop against the float64 oracle, relative L2 <= 5e-6 after 5 iterations
  (the unpaired loop stays below 1e-6 there), on rows that start on 4, 8 and 16
  bytes.
* Operands that the ratio's fast division does not take (zeros, a blurred
  estimate far below 1e-18) against the same oracle.
"""

import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from cudadecon_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [
    (16, 32, 128), (18, 1024, 128), (5, 6, 135), (9, 30, 140), (6, 126, 150), (7, 27, 144),
    (15, 75, 147), (8, 1000, 128), (256, 12, 128), (270, 10, 160), (2, 2, 128), (3, 3, 189),
    (4, 36, 1620), (3, 20, 2048), (162, 14, 175), (25, 243, 128)])
def test_paired_rfft3d_matches_numpy(cdx, torch_cuda, shape):
    torch = torch_cuda
    nz, ny, nx = shape
    x = np.random.default_rng(nz + 7 * ny + nx).standard_normal(shape).astype(np.float32)
    d = torch.from_numpy(x).cuda()
    out = torch.empty((nz, ny, nx // 2 + 1), dtype=torch.complex64, device="cuda")
    ok = cdx.lib().cdx_rfft3d_device(ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                     nx, ny, nz, None)
    assert ok == 1, cdx.lib().cdx_last_error()
    torch.cuda.synchronize()
    assert rel_l2(out.cpu().numpy(), np.fft.rfftn(x.astype(np.float64))) < 2e-6


def _rl(cdx, oracle, tmp_path, raw, n_iters, sxy=1.3, sz=2.5):
    tab = synth.gaussian_otf_table(65, 32, sxy, sz)
    p = tmp_path / "otf.tif"
    synth.write_otf(p, tab)
    kw = dict(dr=0.104, dz=0.3, dr_psf=0.104, dz_psf=0.25)
    cdx.rl_init(raw.shape, p, **kw)
    gz, gy, gx = cdx.decon_grid()
    mine = cdx.rl_decon(raw, background=100.0, n_iters=n_iters)
    cdx.rl_cleanup()
    nz, ny, nx = raw.shape
    st = oracle.rl_init(nx, ny, nz, kw["dr"], kw["dz"], kw["dr_psf"], kw["dz_psf"], 0.0, 0.0, 0,
                        False, synth.otf_table_to_image(tab))
    X0 = oracle.bgsub(raw[:gz, :gy, :gx].astype(np.float32), 100.0)
    fp64 = oracle.rl_iterations(X0, X0, oracle.otf_on_grid(st, gx, gy, gz, dtype=np.float64), n_iters,
                                dtype=np.float64)
    return mine, fp64


@pytest.mark.parametrize("shape", [(12, 36, 135), (11, 34, 150), (10, 35, 128), (9, 27, 175),
                                   (8, 50, 756), (6, 28, 1620), (33, 10, 243)])
def test_paired_rl_matches_fp64(cdx, oracle, torch_cuda, tmp_path, shape):
    raw = synth.bead_stack(shape, n_beads=60, psf_sigma_xy=1.3, psf_sigma_z=2.0, seed=sum(shape))
    mine, fp64 = _rl(cdx, oracle, tmp_path, raw, 5)
    assert mine.shape == fp64.shape
    assert rel_l2(mine, fp64) < 5e-6


def test_paired_ratio_outside_the_fast_range(cdx, oracle, torch_cuda, tmp_path):
    """An empty stack (every blurred value 0) and one bead in an empty stack,
    whose estimate far from the bead falls below the fast division's range."""
    shape = (16, 40, 128)
    raw = np.full(shape, 100, np.uint16)
    mine, fp64 = _rl(cdx, oracle, tmp_path, raw, 4)
    assert np.array_equal(mine, np.zeros_like(mine)) and not fp64.any()
    raw[8, 20, 64] = 40000
    mine, fp64 = _rl(cdx, oracle, tmp_path, raw, 4)
    assert np.isfinite(mine).all()
    assert rel_l2(mine, fp64) < 5e-6


def test_paired_rl_large_ragged_rows(cdx, oracle, torch_cuda, tmp_path):
    """Rows of no whole 16-byte units in a volume past the L2 cache: the update
    pass reads Y and G through shared memory there (an odd height leaves rows
    of the last blocks empty).  Same bound as the smaller volumes'."""
    raw = synth.bead_stack((98, 375, 350), n_beads=200, psf_sigma_xy=1.3, psf_sigma_z=2.0, seed=11)
    mine, fp64 = _rl(cdx, oracle, tmp_path, raw, 3)
    assert mine.shape == (98, 375, 350)
    assert rel_l2(mine, fp64) < 5e-6
