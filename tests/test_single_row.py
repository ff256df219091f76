"""Volumes of one row (ny = 1): the paired layout puts rows 2m and 2m + 1 in one
slot and needs both, so these take the plain passes.

* On the CPU: at every height that may use the layout, a slot's rows of the
  first half exist and the halves cover the volume.
* On the GPU: forward transform and convolution of single-row volumes against
  numpy in float64, relative L2 <= 2e-6, in buffers whose guard elements on
  either side stay as they were.
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
#include "pair_layout.cuh"
int main() {
  for (int ny = 1; ny <= 4096; ++ny)
    printf("%d %d %d %d\\n", ny, cdx::pair_rows(ny) ? 1 : 0, cdx::pair_split(ny), cdx::pair_half(ny));
}
"""


def test_paired_rows_exist(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    (tmp_path / "rows.cu").write_text(PROGRAM)
    subprocess.run([nvcc, "-std=c++17", "-I", str(CSRC), "-o", str(tmp_path / "rows"),
                    str(tmp_path / "rows.cu")], check=True)
    out = subprocess.run([str(tmp_path / "rows")], check=True, capture_output=True, text=True).stdout
    for ny, ok, split, half in (map(int, r.split()) for r in out.splitlines()):
        assert bool(ok) == (ny >= 2)
        if ok:
            assert split % 2 == 0 and split <= ny <= 2 * split and 2 * half >= split


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(5, 1, 128), (1, 1, 756), (32, 1, 320), (7, 1, 1620)])
def test_single_row_transform_and_convolution(cdx, oracle, torch_cuda, tmp_path, shape):
    torch = torch_cuda
    nz, ny, nx = shape
    tab = synth.gaussian_otf_table(65, 32, 1.3, 2.5)
    p = tmp_path / "otf.tif"
    synth.write_otf(p, tab)
    cdx.rl_init((32, 32, 128), p, dr=0.104, dz=0.3, dr_psf=0.104, dz_psf=0.25)
    x = np.random.default_rng(nz + nx).random(shape).astype(np.float32)
    n, guard = x.size, 4096
    src = torch.full((n + 2 * guard,), 7.0, device="cuda")
    src[guard:guard + n] = torch.from_numpy(x.ravel()).cuda()
    dst = torch.full((n + 2 * guard,), 9.0, device="cuda")
    spec = torch.empty((nz, ny, nx // 2 + 1), dtype=torch.complex64, device="cuda")
    at = lambda t: ctypes.c_void_p(t.data_ptr() + 4 * guard)  # noqa: E731
    L = cdx.lib()
    assert L.cdx_rfft3d_device(at(src), ctypes.c_void_p(spec.data_ptr()), nx, ny, nz, None) == 1
    assert L.cdx_conv3d_device(at(src), at(dst), nx, ny, nz, 0, None) == 1
    torch.cuda.synchronize()
    cdx.rl_cleanup()
    S = np.fft.rfftn(x.astype(np.float64))
    assert rel_l2(spec.cpu().numpy(), S) < 2e-6
    st = oracle.rl_init(128, 32, 32, 0.104, 0.3, 0.104, 0.25, 0.0, 0.0, 0, False,
                        synth.otf_table_to_image(tab))
    H = oracle.otf_on_grid(st, nx, ny, nz, dtype=np.float32)  # table positions are 32-bit
    want = np.fft.irfftn(S * np.asarray(H).reshape(S.shape), s=shape, axes=(0, 1, 2))
    assert rel_l2(dst[guard:guard + n].cpu().numpy().reshape(shape), want) < 2e-6
    for t, v in ((src, 7.0), (dst, 9.0)):
        assert bool((t[:guard] == v).all()) and bool((t[guard + n:] == v).all())
