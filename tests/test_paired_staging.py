"""The x update's row copies in shared memory (PX::kStaged, csrc/decon_px.cuh).

* On the CPU: the shared memory that every x pass of every plan asks for, as the
  headers compute it, fits a block (227 KB with the kernels' static arrays).
* On the GPU: RL past 12 << 20 voxels, where the copies are used, against the
  float64 oracle: the plans of 4 pairs a block whose two copies do not fit, and
  none, one and two copies.  Relative L2 <= 5e-6 after 2 iterations, the bound
  of the other paired loops.
* A call that CUDA refuses leaves no error behind for the next one.
"""

import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from conftest import rel_l2
from cudadecon_gb300 import synth

CSRC = Path(__file__).resolve().parents[1] / "cudadecon_gb300" / "csrc"
PROGRAM = """
#include <cstdio>
#include "decon_px.cuh"
#include "pair_plans_gen.cuh"
using namespace cdx;
#define ROW(L, N, V, A, B, C)                                                       \\
  {                                                                                 \\
    using P = PX<PPX##L, V>;                                                        \\
    printf("%d %d %d %zu %zu %zu %zu\\n", L, P::T, P::kStaged, P::smem(0), P::smem(1), \\
           P::smem(P::kStaged), P::smem_fwd(2));                                    \\
  }
int main() { CDX_PX_PLANS(ROW) }
"""


def test_every_x_plan_fits_a_block(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    (tmp_path / "px.cu").write_text(PROGRAM)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-I", str(CSRC),
                    "-o", str(tmp_path / "px"), str(tmp_path / "px.cu")], check=True)
    rows = subprocess.run([str(tmp_path / "px")], check=True, capture_output=True, text=True).stdout
    rows = [[int(v) for v in r.split()] for r in rows.splitlines()]
    assert len(rows) > 130 and {r[2] for r in rows} == {0, 1, 2}
    for L, threads, staged, *smem in rows:
        assert threads <= 1024 and max(smem) + 512 <= 227 * 1024, L


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(36, 256, 1372), (36, 243, 1458), (32, 256, 1568), (64, 320, 625),
                                   (64, 256, 800), (96, 256, 525)])
def test_rl_past_the_staging_line(cdx, oracle, torch_cuda, tmp_path, shape):
    assert np.prod(shape) >= 12 << 20
    raw = synth.bead_stack(shape, n_beads=200, psf_sigma_xy=1.3, psf_sigma_z=2.0, seed=sum(shape))
    tab = synth.gaussian_otf_table(65, 32, 1.3, 2.5)
    p = tmp_path / "otf.tif"
    synth.write_otf(p, tab)
    kw = dict(dr=0.104, dz=0.3, dr_psf=0.104, dz_psf=0.25)
    cdx.rl_init(shape, p, **kw)
    assert cdx.decon_grid() == shape
    mine = cdx.rl_decon(raw, background=100.0, n_iters=2)
    cdx.rl_cleanup()
    nz, ny, nx = shape
    st = oracle.rl_init(nx, ny, nz, kw["dr"], kw["dz"], kw["dr_psf"], kw["dz_psf"], 0.0, 0.0, 0,
                        False, synth.otf_table_to_image(tab))
    X0 = oracle.bgsub(raw.astype(np.float32), 100.0)
    want = oracle.rl_iterations(X0, X0, oracle.otf_on_grid(st, nx, ny, nz, dtype=np.float64), 2,
                                dtype=np.float64)
    assert rel_l2(mine, want) < 5e-6


@pytest.mark.gpu
def test_a_refused_call_leaves_no_error_behind(cdx, torch_cuda):
    """A transform whose spectrum (about 0.5 TB) no card holds is refused; the
    call after it works."""
    torch = torch_cuda
    x = torch.randn((4, 8, 128), device="cuda")
    out = torch.empty((4, 8, 65), dtype=torch.complex64, device="cuda")
    args = [ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(out.data_ptr())]
    L = cdx.lib()
    assert L.cdx_rfft3d_device(*args, 2048, 8192, 7680, None) == 0
    assert b"memory" in L.cdx_last_error()
    assert L.cdx_rfft3d_device(*args, 128, 8, 4, None) == 1, L.cdx_last_error()
    want = np.fft.rfftn(x.cpu().numpy().astype(np.float64))
    assert rel_l2(out.cpu().numpy(), want) < 2e-6
