"""Rounding of the RL loop on mostly dark stacks (csrc/decon_px.cuh: the ratio
goes through the second convolution less its mean).

A few beads whose background lies below what is subtracted leave 99% of the
voxels at 0 and a ratio near 0 there; a constant of 1 taken off it would be what
the transforms round.  The error against 64 bits is set against that of the
oracle's float32 loop, which takes nothing off.  The ratio of the two errors
scatters by a factor of about 1.55 from stack to stack (an ill-conditioned loop),
so the geometric mean of 32 stacks by about 8%: it lies near 1 and is held to
1.45; with the constant of 1 it was 2.0 to 2.3.
"""

import math

import numpy as np
import pytest

from cudadecon_gb300 import synth

pytestmark = pytest.mark.gpu
PIX = dict(dr=0.104, dz=0.3, dr_psf=0.104, dz_psf=0.3)


def _dark(shape, seed):
    r = np.random.default_rng(seed)
    nz, ny, nx = shape
    obj = np.zeros(shape)
    for _ in range(5):
        obj[r.integers(nz), r.integers(ny), r.integers(nx)] = \
            (500 + 4500 * r.random()) * (2 * math.pi) ** 1.5 * 1.3 * 1.3 * 3.0
    f = [np.fft.fftfreq(nz)[:, None, None] * 3.0, np.fft.fftfreq(ny)[None, :, None] * 1.3,
         np.fft.rfftfreq(nx)[None, None] * 1.3]
    blur = np.exp(-2 * math.pi ** 2 * (f[0] ** 2 + f[1] ** 2 + f[2] ** 2))
    img = np.clip(np.fft.irfftn(np.fft.rfftn(obj) * blur, s=shape, axes=(0, 1, 2)), 0, None)
    return r.poisson(img + 100).astype(np.uint16)


def test_dark_stacks_keep_the_plain_loops_error(cdx, oracle, torch_cuda, tmp_path):
    tab = synth.gaussian_otf_table(65, 32, 1.3, 3.0)
    p = tmp_path / "otf.tif"
    synth.write_otf(p, tab)
    logs = []
    for shape in ((24, 48, 128), (27, 45, 150)):
        nz, ny, nx = shape
        st = oracle.rl_init(nx, ny, nz, *PIX.values(), 0.0, 0.0, 0, False, synth.otf_table_to_image(tab))
        H = {d: oracle.otf_on_grid(st, nx, ny, nz, dtype=d) for d in (np.float64, np.float32)}
        cdx.rl_init(shape, p, **PIX)
        for seed in range(16):
            raw = _dark(shape, seed)
            iters = 10 + seed % 8
            X0 = oracle.bgsub(raw.astype(np.float32), 140.0)
            assert 0.97 < (X0 == 0).mean() < 1.0
            mine = cdx.rl_decon(raw, background=140.0, n_iters=iters)
            want, plain = (oracle.rl_iterations(X0, X0, H[d], iters, dtype=d) for d in H)
            logs.append(math.log(np.linalg.norm(mine - want) / np.linalg.norm(plain - want)))
        cdx.rl_cleanup()
    assert math.exp(np.mean(logs)) < 1.45
