"""Deskew, rotation and maximum projections at the sizes where their kernels'
row batches, lane tiles and split columns have remainders, against the same
formulas in 64 bits (deskew_kernel and rotate_kernel, geometryTransform.cu:
4-88; MaxIntProj, linearDecon.cpp:1434-1473)."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# (nz, ny, nx): rows 1, one below / at / above a batch, two thread blocks;
# columns below, at and above a warp and a block
SIZES = [(1, 1, 2), (3, 15, 17), (2, 16, 128), (5, 17, 129), (33, 33, 65), (70, 100, 260), (9, 257, 31)]


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _stack(shape):
    rng = np.random.default_rng(sum(shape))
    return rng.random(shape, dtype=np.float32)


@pytest.mark.parametrize("shape", SIZES)
def test_deskew_rows(shape):
    from cudadecon_gb300 import lib

    nz, ny, nx = shape
    v, wide, factor, pad = _stack(shape), nx + 13, 0.8371, 7.0
    d = torch.from_numpy(v).cuda()
    out = torch.full((nz, ny, wide), -1.0, device="cuda")
    assert lib().cdx_deskew_device(_p(d), nx, ny, nz, factor, _p(out), wide, 0, pad, _stream()) == 1
    got = out.cpu().numpy()
    x = np.arange(wide) - wide / 2.0
    xin = (x[None] - factor * (np.arange(nz)[:, None] - nz / 2.0) + nx / 2.0)
    inside = (xin >= 0) & (xin < nx - 1)
    # coordinates below 512 are rounded to 2^-16 at most and the slope is at
    # most 1; the blend adds three roundings of values below 1
    tol = 2.0 ** -16 + 3 * 2.0 ** -24
    edge = (np.abs(xin) < 2.0 ** -14) | (np.abs(xin - (nx - 1)) < 2.0 ** -14)
    i = np.clip(np.floor(xin).astype(int), 0, max(nx - 2, 0))
    f = xin - i
    for z in range(nz):
        want = np.where(inside[z], (1 - f[z]) * v[z][:, i[z]].astype(np.float64) + f[z] * v[z][:, i[z] + 1], pad)
        ok = ~edge[z]
        assert np.abs(got[z] - want)[:, ok].max(initial=0.0) <= tol


@pytest.mark.parametrize("shape", SIZES)
@pytest.mark.parametrize("angle", [0.0, 31.5, -128.0])
def test_rotate_rows(shape, angle):
    from cudadecon_gb300 import lib

    nz, ny, nx = shape
    v, nz_o, nx_o = _stack(shape), nz + 6, nx + 5
    c, s = math.cos(math.radians(angle)), math.sin(math.radians(angle))
    rot = np.array([c, s, -s, c], np.float32)
    d = torch.from_numpy(v).cuda()
    out = torch.full((nz_o, ny, nx_o), -1.0, device="cuda")
    assert lib().cdx_rotate_device(_p(d), nx, ny, nz, rot.ctypes.data_as(ctypes.POINTER(ctypes.c_float)), _p(out),
                                   nx_o, nz_o, _stream()) == 1
    got = out.cpu().numpy()[::-1]
    q = rot.astype(np.float64)
    xc, zc = np.arange(nx_o)[None] - nx_o / 2.0, np.arange(nz_o)[:, None] - nz_o / 2.0
    zin = q[0] * zc + q[1] * xc + nz / 2.0
    xin = q[2] * zc + q[3] * xc + nx / 2.0
    near = lambda a, b: np.abs(a - b) < 2.0 ** -13
    edge = near(xin, 0) | near(xin, nx - 1) | near(zin, 0) | near(zin, nz - 1)
    inside = (xin >= 0) & (xin < nx - 1) & (zin >= 0) & (zin < nz - 1)
    ix, iz = np.clip(np.floor(xin).astype(int), 0, nx - 2), np.clip(np.floor(zin).astype(int), 0, max(nz - 2, 0))
    iz1 = np.minimum(iz + 1, nz - 1)
    fx, fz = (xin - ix)[:, None], (zin - iz)[:, None]
    w = v.astype(np.float64).transpose(0, 2, 1)  # (z, x, y)
    g = lambda k, j: w[k, j].transpose(0, 2, 1)  # (z out, y, x out)
    want = (1 - fz) * ((1 - fx) * g(iz, ix) + fx * g(iz, ix + 1)) + fz * ((1 - fx) * g(iz1, ix) + fx * g(iz1, ix + 1))
    want = np.where(inside[:, None], want, 0.0)
    # three roundings of a coordinate below 512 in each of two axes, and the blends'
    tol = 2 * 3 * 2.0 ** -16 + 9 * 2.0 ** -24
    err = np.abs(got - want).transpose(0, 2, 1)[~edge]
    assert err.max(initial=0.0) <= tol


@pytest.mark.parametrize("shape", SIZES + [(7, 3, 400), (130, 600, 700)])
def test_projections_split(shape):
    import cudadecon_gb300 as cdx

    v = _stack(shape) - 0.5
    v.reshape(-1)[:: 7] = np.nan
    v.reshape(-1)[:: 11] = -np.inf
    v[0, 0, :] = -np.inf
    want = np.where(np.isnan(v) | (v < -1e10), np.float32(-1e10), v)
    d = torch.from_numpy(v).cuda()
    for axis, reduced in ((0, 2), (1, 1), (2, 0)):
        got = cdx.mip(d, axis).cpu().numpy()
        assert np.array_equal(got, want.max(axis=reduced))
