"""Transforms with an axis of length 1, on which they are the identity: the
generic engine's single stage of radix 1.  The forward transform and the
convolution against numpy in float64 (relative L2 <= 2e-6, the bound of the
other lengths), with guard elements around the buffers that must keep their
values.
"""

import ctypes

import numpy as np
import pytest

from conftest import rel_l2
from cudadecon_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 36, 756), (1, 27, 128), (1, 40, 100), (3, 4, 1), (1, 2, 2)])
def test_axis_of_one(cdx, oracle, torch_cuda, tmp_path, shape):
    torch = torch_cuda
    nz, ny, nx = shape
    tab = synth.gaussian_otf_table(65, 32, 1.3, 2.5)
    p = tmp_path / "otf.tif"
    synth.write_otf(p, tab)
    cdx.rl_init((32, 32, 128), p, dr=0.104, dz=0.3, dr_psf=0.104, dz_psf=0.25)
    x = np.random.default_rng(nz + ny + nx).random(shape).astype(np.float32)
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
