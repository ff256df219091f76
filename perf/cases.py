"""The work a user has this library do, as cases that can be timed and checked.

Every case is one pass through the package's public entry points on the sizes
the library is used with: Richardson-Lucy deconvolution of single stacks
(smallest to time-lapse volume), with and without deskew and rotation, from
device and from host memory, batches of uneven stacks, y-tiled stacks, the
one-step Wiener filter, and the preview of a raw stage-scan stack (deskew,
rotate, projections).  All volumes are synthetic: sparse beads blurred by a
Gaussian PSF on a 100-count background with Poisson noise, as uint16.

The library keeps one RL session per process, so the OTF belongs to the case
and only the images come from the seed.
"""

import ctypes
import math
import os
import tempfile

import numpy as np
import torch

import cudadecon_gb300 as cdx
from cudadecon_gb300 import synth

BACKGROUND = 100.0
EPS32 = float(np.finfo(np.float32).eps)


# ---------------------------------------------------------------- the cases
def _rl(name, shape, iters, entry="device", angle=0.0, dz=0.3, sxy=1.3, sz=3.0, napodize=0, nzblend=0,
        mirror=False, camcor=False):
    nz, ny, nx = shape
    d = dict(kind="rl", nz=nz, ny=ny, nx=nx, iters=iters, entry=entry, angle=angle, dz=dz, sxy=sxy, sz=sz,
             napodize=napodize, nzblend=nzblend, mirror=mirror, camcor=camcor)
    return dict(d, name=name) if name else d


def listed():
    return [
        # a cropped cell or a single bead: the smallest stacks of a batch, launch-bound
        _rl("rl_32x128x128", (32, 128, 128), 10, sxy=1.5, sz=4.0),
        # an ordinary camera crop without deskew, resident on the GPU
        _rl("rl_64x256x256", (64, 256, 256), 10, sxy=1.5, sz=4.0),
        # a ragged crop from host memory with the conditioning options: odd sizes
        # (63 x 189 x 324 after the crop to FFT-friendly sizes), edge taper, z blend
        # and the mirrored stack
        _rl("rl_ragged_options_host", (63, 190, 333), 10, entry="host", napodize=15, nzblend=3, mirror=True),
        # one stage-scan light-sheet stack through the reference's own entry point,
        # numpy in and numpy out: deskew to 100 x 256 x 756, 15 iterations, rotate
        _rl("stage_scan_host", (101, 256, 512), 15, entry="host", angle=31.5),
        # the stack of the reference's published timing: 186 x 613 x 313 raw at 32.8
        # degrees, deconvolved on 180 x 600 x 810, rotated
        _rl("published_stack", (186, 613, 313), 15, angle=32.8, dz=0.36),
        # a large plain stack
        _rl("rl_128x512x1024", (128, 512, 1024), 20, sxy=1.5, sz=4.0),
        # one volume of a two-channel time lapse: camera correction, deskew to
        # 256 x 1024 x 1620, 20 iterations, rotate
        _rl("timelapse_volume", (256, 1024, 1024), 20, angle=31.5, camcor=True),
        # timepoints, channels and tiles of uneven shape in one call, each with its
        # own OTF, resident on the GPU
        dict(name="batch_16_uneven", kind="batch", entry="device", stacks=16, shapes=1003, zmax=160, ymax=512,
             xmax=1024, iters=10),
        # small crops from and into page-locked host memory in one call
        dict(name="batch_12_small_host", kind="batch", entry="host", stacks=12, shapes=17, zmax=64, ymax=256,
             xmax=384, iters=10),
        # a tall stack cut into y tiles, host memory
        dict(name="tiled_100x512x512", kind="tiled", nz=100, ny=512, nx=512, tile=128, overlap=30, iters=10),
        # the one-step filter a user tries before iterating
        dict(name="wiener_100x256x756", kind="wiener", nz=100, ny=256, nx=756),
        # looking at a raw stage-scan stack: deskew, rotate, three projections
        dict(name="preview_101x256x512", kind="preview", nz=101, ny=256, nx=512, angle=31.5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rl", "rl", "rl", "deskewed", "deskewed", "batch", "batch", "tiled", "wiener", "preview"])
    z, y, x = _log(rng, 32, 200), _log(rng, 128, 640), _log(rng, 128, 1024)
    iters = rng.randint(8, 20)
    if kind == "rl":
        opt = rng.random() < 0.3
        return _rl(None, (z, y, x), iters, entry=rng.choice(["device", "device", "host"]),
                   sxy=round(rng.uniform(1.0, 1.8), 2), sz=round(rng.uniform(2.4, 4.8), 2),
                   napodize=rng.randint(5, 20) if opt else 0, nzblend=rng.randint(0, 4) if opt else 0,
                   mirror=opt and z <= 80)
    if kind == "deskewed":
        return _rl(None, (z, y, min(x, 640)), iters, entry=rng.choice(["device", "host"]),
                   angle=round(rng.uniform(29.0, 34.0), 1), dz=round(rng.uniform(0.2, 0.4), 2),
                   camcor=rng.random() < 0.3)
    if kind == "batch":
        entry = rng.choice(["device", "host"])
        return dict(kind="batch", entry=entry, stacks=rng.randint(4, 16), shapes=rng.randint(1, 10 ** 6),
                    zmax=_log(rng, 48, 160), ymax=_log(rng, 192, 512), xmax=_log(rng, 192, 1024), iters=iters)
    if kind == "tiled":
        return dict(kind="tiled", nz=min(z, 120), ny=_log(rng, 300, 640), nx=min(x, 640), tile=rng.choice([96, 128, 160]),
                    overlap=rng.randint(16, 40), iters=iters)
    if kind == "wiener":
        s = synth.smooth_sizes(32, 1024)
        near = lambda v: max(n for n in s if n <= v)  # noqa: E731 - the entry point takes FFT-friendly sizes
        return dict(kind="wiener", nz=near(z), ny=near(y), nx=near(x))
    return dict(kind="preview", nz=z, ny=y, nx=min(x, 640), angle=round(rng.uniform(29.0, 34.0), 1))


# ---------------------------------------------------------------- inputs
def _stack(shape, seed, sxy, sz, density=1.0 / 40000):
    """uint16 CUDA stack of sparse beads blurred by the PSF, with Poisson noise."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    n = math.prod(shape)
    k = max(8, int(n * density))
    at = torch.randint(0, n, (k,), generator=g, device="cuda")
    amp = (500.0 + 4500.0 * torch.rand(k, generator=g, device="cuda")) * (2 * math.pi) ** 1.5 * sxy * sxy * sz
    obj = torch.zeros(n, dtype=torch.float32, device="cuda").scatter_reduce_(0, at, amp, "amax").view(shape)
    f = [torch.fft.fftfreq(shape[0], device="cuda")[:, None, None] * sz,
         torch.fft.fftfreq(shape[1], device="cuda")[None, :, None] * sxy,
         torch.fft.rfftfreq(shape[2], device="cuda")[None, None, :] * sxy]
    blur = torch.exp(-2 * math.pi ** 2 * (f[0] ** 2 + f[1] ** 2 + f[2] ** 2))
    img = torch.fft.irfftn(torch.fft.rfftn(obj) * blur, s=shape).clamp_(min=0.0).add_(BACKGROUND)
    return torch.poisson(img, generator=g).clamp_(0, 65535).to(torch.int32).to(torch.uint16)


def _camera(ny, nx, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 7)
    p = torch.rand((3, ny, nx), generator=g, device="cuda")
    p[:2] *= 0.02
    p[2] = 90.0 + 20.0 * p[2]
    return p.contiguous()


def _pixels(case):
    """Pixel sizes (dr, dz, dr_psf, dz_psf) of a case."""
    return 0.104, case.get("dz", 0.3), 0.104, 0.2 if case.get("angle") else 0.3


def _table(case):
    return synth.gaussian_otf_table(129, 64, case.get("sxy", 1.3), case.get("sz", 3.0))


def _session(case, shape):
    dr, dz, dr_psf, dz_psf = _pixels(case)
    fd, path = tempfile.mkstemp(suffix=".tif")
    os.close(fd)
    try:
        synth.write_otf(path, _table(case))
        a = case.get("angle", 0.0)
        cdx.rl_init(shape, path, dr=dr, dz=dz, dr_psf=dr_psf, dz_psf=dz_psf, deskew_angle=a, rotation_angle=a)
    finally:
        os.unlink(path)


def _batch_shapes(case):
    r = np.random.default_rng(case["shapes"])
    out = []
    for _ in range(case["stacks"]):
        shape = [int(r.integers(lo, hi + 1)) for lo, hi in ((32, case["zmax"]), (128, case["ymax"]), (128, case["xmax"]))]
        j = r.uniform(0.8, 1.2, 2)
        out.append((tuple(shape), 1.5 * float(j[0]), 4.0 * float(j[1])))
    return out


def prepare(case, seed):
    k = case["kind"]
    if k == "batch":
        stacks = []
        for i, (shape, sxy, sz) in enumerate(_batch_shapes(case)):
            raw = _stack(shape, seed * 1000 + i, sxy, sz)
            stacks.append(dict(raw=raw if case["entry"] == "device" else raw.cpu().pin_memory(),
                               otf=synth.gaussian_otf_table(129, 64, sxy, sz), dr=0.104, dz=0.3, dr_psf=0.104,
                               dz_psf=0.3, background=BACKGROUND))
        s = dict(case=case, stacks=stacks)
        if case["entry"] == "host":
            s["out"] = [torch.empty(cdx.batch_grid(tuple(d["raw"].shape)), dtype=torch.float32).pin_memory()
                        for d in stacks]
        return s
    shape = (case["nz"], case["ny"], case["nx"])
    s = dict(case=case, raw=_stack(shape, seed, case.get("sxy", 1.3), case.get("sz", 3.0)))
    if k == "rl":
        _session(case, shape)
        if case["camcor"]:
            s["camera"] = _camera(shape[1], shape[2], seed)
            s["corrected"] = torch.empty_like(s["raw"])
            if case["entry"] == "host":
                cdx.camcor_init(shape, s["camera"].cpu().numpy())
        if case["entry"] == "host":
            s["raw"] = s["raw"].cpu().numpy()
        else:
            s["out"] = torch.empty(cdx.output_shape(), dtype=torch.float32, device="cuda")
    elif k == "tiled":
        _session(case, (shape[0], case["tile"], shape[2]))
        s["raw"] = s["raw"].cpu().numpy()
    elif k == "wiener":
        _session(case, shape)
        s["raw"] = s["raw"].to(torch.float32)
    else:
        g = _geometry(case)
        s["raw"] = s["raw"].to(torch.float32)
        s["deskewed"] = torch.empty((shape[0], shape[1], g["width"]), dtype=torch.float32, device="cuda")
        s["rotated"] = torch.empty((g["nz_r"], shape[1], g["nx_r"]), dtype=torch.float32, device="cuda")
        s["geometry"] = g
    return s


# ---------------------------------------------------------------- one pass
def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _ok(rc, what):
    if rc != 1:
        raise RuntimeError("%s: %s" % (what, cdx.lib().cdx_last_error().decode()))


def run(state):
    case = state["case"]
    k = case["kind"]
    if k == "batch":
        if case["entry"] == "device":
            return cdx.rl_batch(state["stacks"], n_iters=case["iters"])
        return cdx.rl_batch_host(state["stacks"], n_iters=case["iters"], results=state["out"])
    if k == "tiled":
        return cdx.rl_tiled(state["raw"], tile=case["tile"], tile_overlap=case["overlap"], background=BACKGROUND,
                            n_iters=case["iters"])
    if k == "wiener":
        return cdx.wiener(state["raw"], background=BACKGROUND, wiener=0.05, NA=1.1, wavelength=0.525)
    if k == "rl" and case["entry"] == "host":
        raw = cdx.camcor(state["raw"]) if case["camcor"] else state["raw"]
        return cdx.rl_decon(raw, background=BACKGROUND, n_iters=case["iters"], napodize=case["napodize"],
                            nzblend=case["nzblend"], dup_rev_stack=case["mirror"])
    L = cdx.lib()
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    raw = state["raw"]
    nz, ny, nx = raw.shape
    if k == "rl":
        if case["camcor"]:
            _ok(L.cdx_camcor_device(_p(raw), nx, ny, nz, _p(state["camera"]), _p(state["corrected"]), st), "camcor")
            raw = state["corrected"]
        _ok(L.cdx_RL_device(_p(raw), nx, ny, nz, _p(state["out"]), None, BACKGROUND, False, False, case["iters"], 0,
                            case["napodize"], case["nzblend"], 0.0, case["mirror"], False, st), "RL")
        return state["out"]
    g = state["geometry"]
    rot = (ctypes.c_float * 4)(*g["rot"])
    _ok(L.cdx_deskew_device(_p(raw), nx, ny, nz, g["factor"], _p(state["deskewed"]), g["width"], 0, 0.0, st), "deskew")
    _ok(L.cdx_rotate_device(_p(state["deskewed"]), g["width"], ny, nz, rot, _p(state["rotated"]), g["nx_r"], g["nz_r"],
                            st), "rotate")
    return [state["deskewed"], state["rotated"]] + [cdx.mip(state["rotated"], a) for a in (0, 1, 2)]


# ---------------------------------------------------------------- sizes and work
def _smooth(n):
    while n > 1:
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n -= 1
    return n


def _geometry(case):
    """Deskew factor and width, rotation matrix (float32) and rotated sizes of a case."""
    f = np.float32
    dr, dz = f(_pixels(case)[0]), f(_pixels(case)[1])
    nz, a = case["nz"], float(f(case.get("angle", 0.0)))
    grid_z = _smooth(nz) if case["kind"] != "preview" else nz
    if not a:
        return dict(factor=0.0, width=_smooth(case["nx"]), rot=None, dz=dz)
    rad = a * math.pi / 180.0
    factor = math.cos(rad) * float(dz) / float(dr)
    width = _smooth(case["nx"] + int(math.floor(float(f(grid_z) * dz) * abs(math.cos(rad)) / float(dr))))
    dz = f(float(dz) * abs(math.sin(rad)))
    r = f(rad)
    c, s, stretch = f(math.cos(float(r))), f(math.sin(float(r))), dr / dz
    rot = [float(c * stretch), float(s * stretch), float(-s), float(c)]
    q = [f(v) for v in rot]
    return dict(factor=factor, width=width, rot=rot, dz=dz, nz_r=int(f(grid_z) * q[3] / q[0]),
                nx_r=int(f(width) * q[3] + f(grid_z) * q[2] * q[2] / abs(q[1])))


def _tiles(case):
    """(tile size, count, overlap, deconvolved rows) of a tiled case."""
    ny, size = case["ny"], min(case["tile"], case["ny"])
    n = math.ceil(ny / (size - case["overlap"]))
    return size, n, math.floor((size * n - ny) / (n - 1)) if n > 1 else 0, _smooth(size)


def _rl_work(voxels, iters):
    # one iteration streams 56 bytes a voxel: four 3D transforms read and write
    # 8 each, the ratio reads the image (4) and the update and prediction read
    # two and write three float volumes; 4 real transforms of 2.5 N log2 N
    # operations and about 30 elementwise ones
    return 56.0 * voxels * iters, iters * (10.0 * voxels * math.log2(voxels) + 30.0 * voxels)


def work(case):
    k = case["kind"]
    if k == "batch":
        b = fl = 0.0
        for shape, _, _ in _batch_shapes(case):
            v = math.prod(_smooth(n) for n in shape)
            w = _rl_work(v, case["iters"])
            b, fl = b + w[0] + 2.0 * math.prod(shape) + 4.0 * v, fl + w[1]
        return {"bytes": b, "flops": fl}
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    raw = nz * ny * nx
    if k == "tiled":
        size, n, _, rows = _tiles(case)
        w = _rl_work(_smooth(nz) * rows * _smooth(nx), case["iters"])
        return {"bytes": n * w[0] + 2.0 * raw + 4.0 * _smooth(nz) * ny * _smooth(nx), "flops": n * w[1]}
    if k == "wiener":
        return {"bytes": 4.0 * raw + 4.0 * raw + 16.0 * raw, "flops": 5.0 * raw * math.log2(raw) + 30.0 * raw}
    g = _geometry(case)
    if k == "preview":
        d, r = nz * ny * g["width"], g["nz_r"] * ny * g["nx_r"]
        return {"bytes": 4.0 * (raw + d + r) + 4.0 * (ny * g["nx_r"] + g["nz_r"] * (ny + g["nx_r"])),
                "flops": 3.0 * d + 9.0 * r + 3.0 * r}
    zz, yy = _smooth(nz), _smooth(ny)
    v = zz * yy * g["width"]
    b, fl = _rl_work(v * (2 if case["mirror"] else 1), case["iters"])
    out = g["nz_r"] * yy * g["nx_r"] if case["angle"] else v
    return {"bytes": b + 2.0 * raw + 4.0 * out, "flops": fl + 20.0 * raw + 9.0 * out}


# ---------------------------------------------------------------- 64-bit values
# Coordinates (table positions, shear and rotation offsets) are defined in 32
# bits and are computed in 32 bits here too; every value is computed in 64.
def _f32(v):
    return torch.as_tensor(v, dtype=torch.float32, device="cuda")


def _fma(a, b, c):
    """float32 a * b + c with one rounding (the product of two floats is exact in 64 bits)."""
    return (a.double() * b.double() + c.double()).float()


def _otf_grid(shape, table, dr, dz, dr_psf, dz_psf):
    """OTF on the rfft grid of shape (nz, ny, nx), complex128: bilinear in (kr, kz), kz wrapping."""
    nz, ny, nx = shape
    f = np.float32
    nr, nzo = table.shape
    step = f(1) / (f((nr - 1) * 2) * f(dr_psf))
    sx = f(1.0 / float(f(dr) * f(nx))) / step
    sy = f(1.0 / float(f(dr) * f(ny))) / step
    sz = f(1.0 / float(f(dz) * f(nz))) / (f(1) / (f(nzo) * f(dz_psf)))
    t = torch.as_tensor(table, device="cuda").to(torch.complex128)
    z = torch.arange(nz, device="cuda")
    fz = torch.where(z > nz // 2, z - nz, z).float() * _f32(float(sz))
    kz = torch.where(fz < 0, fz + float(nzo), fz)
    inside = (kz < nzo) & (kz >= 0)
    kz = torch.where(inside, kz, torch.zeros_like(kz))
    iz = kz.floor().long()
    az = kz.double() - iz
    tz = (t[:, iz] * (1 - az) + t[:, (iz + 1) % nzo] * az) * inside  # (nr, nz)
    y = torch.arange(ny, device="cuda")
    fy = torch.where(y > ny // 2, y - ny, y).float() * _f32(float(sy))
    fx = torch.arange(nx // 2 + 1, device="cuda").float() * _f32(float(sx))
    kr = _fma(fx[None], fx[None], (fy * fy)[:, None].expand(ny, nx // 2 + 1)).sqrt()
    ok = kr < nr - 1
    ir = torch.where(ok, kr, torch.zeros_like(kr)).floor().long()
    ar = torch.where(ok, kr.double() - ir, torch.zeros_like(kr, dtype=torch.float64))
    H = torch.empty((nz, ny, nx // 2 + 1), dtype=torch.complex128, device="cuda")
    for i in range(nz):
        c = tz[:, i]
        H[i] = (c[ir] * (1 - ar) + c[(ir + 1).clamp_(max=nr - 1)] * ar) * ok
    return H


def _conv(v, H, conj=False):
    S = torch.fft.rfftn(v)
    S *= H.conj() if conj else H
    return torch.fft.irfftn(S, s=v.shape)


def _rl64(X, H, iters):
    raw, Xm, G, lam = X.clone(), None, None, 0.0
    for k in range(iters):
        Y = X if k < 2 else (X + lam * (X - Xm)).clamp_(min=0.0)
        c = _conv(Y, H)
        c = torch.where(c != 0, c, torch.full_like(c, EPS32))
        r = (raw / c + EPS32).clamp_(-10.0, 10.0)
        new = (_conv(r, H, True) * Y).clamp_(min=0.0)
        g = new - Y
        if k >= 1:
            lam = min(max(float((g * G).sum() / ((G * G).sum() + EPS32)), 0.0), 1.0)
        X, Xm, G = new, X, g
    return X


def _deskew64(v, factor, width):
    nz, ny, nx = v.shape
    x = torch.arange(width, dtype=torch.float64, device="cuda") - width / 2.0
    z = torch.arange(nz, dtype=torch.float64, device="cuda") - nz / 2.0
    at = (x[None] - factor * z[:, None] + nx / 2.0).float()
    ok = (at >= 0) & (at < nx - 1)
    at = torch.where(ok, at, torch.zeros_like(at))
    i = at.floor().long()
    w = at.double() - i
    out = torch.empty((nz, ny, width), dtype=torch.float64, device="cuda")
    for k in range(nz):
        out[k] = (v[k][:, i[k]] * (1 - w[k]) + v[k][:, (i[k] + 1).clamp(max=nx - 1)] * w[k]) * ok[k]
    return out


def _rotate64(v, rot, nx_r, nz_r):
    nz, ny, nx = v.shape
    q = [_f32(r) for r in rot]
    xc = (torch.arange(nx_r, dtype=torch.float64, device="cuda") - nx_r / 2.0).float()[None]
    zc = (torch.arange(nz_r, dtype=torch.float64, device="cuda") - nz_r / 2.0).float()[:, None].expand(nz_r, nx_r)
    zi = (_fma(q[0], zc, (q[1] * xc).expand(nz_r, nx_r)).double() + nz / 2.0).float()
    xi = (_fma(q[2], zc, (q[3] * xc).expand(nz_r, nx_r)).double() + nx / 2.0).float()
    ok = (xi >= 0) & (xi < nx - 1) & (zi >= 0) & (zi < nz - 1)
    zi, xi = torch.where(ok, zi, torch.zeros_like(zi)), torch.where(ok, xi, torch.zeros_like(xi))
    z0, x0 = zi.floor().long(), xi.floor().long()
    wz, wx = zi.double() - z0, xi.double() - x0
    z1, x1 = (z0 + 1).clamp(max=nz - 1), (x0 + 1).clamp(max=nx - 1)
    out = torch.empty((nz_r, ny, nx_r), dtype=torch.float64, device="cuda")
    for k in range(nz_r):  # the output is flipped in z
        a = v[z0[k], :, x0[k]] * (1 - wx[k])[:, None] + v[z0[k], :, x1[k]] * wx[k][:, None]
        b = v[z1[k], :, x0[k]] * (1 - wx[k])[:, None] + v[z1[k], :, x1[k]] * wx[k][:, None]
        out[nz_r - 1 - k] = ((a * (1 - wz[k])[:, None] + b * wz[k][:, None]) * ok[k][:, None]).T
    return out


def _conditioned(case, v):
    """Background, edge taper, z blend and mirrored stack as the options of a case say."""
    n = case["napodize"]
    if n:
        w = 1.0 - torch.sin((torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) / n * math.pi * 0.5)
        d = (v[:, -1, :] - v[:, 0, :]) / 2.0
        v[:, :n, :] += d[:, None, :] * w[None, :, None]
        v[:, -n:, :] -= d[:, None, :] * w.flip(0)[None, :, None]
        d = (v[:, :, -1] - v[:, :, 0]) / 2.0
        v[:, :, :n] += d[:, :, None] * w[None, None, :]
        v[:, :, -n:] -= d[:, :, None] * w.flip(0)[None, None, :]
    return (v - BACKGROUND).clamp_(min=0.0)


def _exact_rl(case, seed):
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    if case["camcor"]:
        return None  # the camera correction truncates to whole numbers, on either side of those it falls next to
    raw = _stack((nz, ny, nx), seed, case["sxy"], case["sz"])
    g = _geometry(case)
    zz, yy = _smooth(nz), _smooth(ny)
    xx = nx if case["angle"] else _smooth(nx)
    v = _conditioned(case, raw[:zz, :yy, :xx].to(torch.int32).double())
    if case["angle"]:
        v = _deskew64(v, g["factor"], g["width"])
    n = case["nzblend"]
    if n:
        step = (v[-1] - v[0]) * (1.0 - math.sin(1.5 / n * math.pi * 0.5))
        for _ in range(n):
            v[1] += step
            v[-2] -= step
    if case["mirror"]:
        v = torch.cat([v, v.flip(0)])
    dr, _, dr_psf, dz_psf = _pixels(case)
    X = _rl64(v, _otf_grid(v.shape, _table(case), dr, float(g["dz"]), dr_psf, dz_psf), case["iters"])
    X = X[:zz]
    return _rotate64(X, g["rot"], g["nx_r"], g["nz_r"]) if case["angle"] else X


def _exact_tiled(case, seed):
    nz, ny, nx = case["nz"], case["ny"], case["nx"]
    raw = _stack((nz, ny, nx), seed, 1.3, 3.0).to(torch.int32).double()
    size, n, overlap, rows = _tiles(case)
    zz, xx = _smooth(nz), _smooth(nx)
    if n == 1:
        return None
    dr, dz, dr_psf, dz_psf = _pixels(case)
    H = _otf_grid((zz, rows, xx), _table(case), dr, dz, dr_psf, dz_psf)
    out = torch.zeros((zz, ny, xx), dtype=torch.float64, device="cuda")
    for t in range(n):
        at = int(math.floor(t * (size - overlap)))
        src = (torch.arange(size, device="cuda") + at).clamp_(0, ny - 1)
        X = _rl64((raw[:, src][:zz, :rows, :xx] - BACKGROUND).clamp_(min=0.0), H, case["iters"])
        lo = 0 if t == 0 else int(math.floor(overlap / 2.0))
        hi = rows if t == n - 1 else int(math.floor(rows - overlap / 2.0))
        hi = min(hi, ny - at)
        out[:, at + lo:at + hi] = X[:, lo:hi]
    return out


def exact(case, seed):
    k = case["kind"]
    if k == "batch":
        out = []
        for i, (shape, sxy, sz) in enumerate(_batch_shapes(case)):
            raw = _stack(shape, seed * 1000 + i, sxy, sz)
            grid = tuple(_smooth(n) for n in shape)
            v = (raw[:grid[0], :grid[1], :grid[2]].to(torch.int32).double() - BACKGROUND).clamp_(min=0.0)
            H = _otf_grid(grid, synth.gaussian_otf_table(129, 64, sxy, sz), 0.104, 0.3, 0.104, 0.3)
            out.append(_rl64(v, H, case["iters"]))
        return out
    if k == "tiled":
        return _exact_tiled(case, seed)
    if k == "rl":
        return _exact_rl(case, seed)
    shape = (case["nz"], case["ny"], case["nx"])
    v = _stack(shape, seed, case.get("sxy", 1.3), case.get("sz", 3.0)).to(torch.int32).double()
    if k == "preview":
        g = _geometry(case)
        d = _deskew64(v, g["factor"], g["width"])
        r = _rotate64(d, g["rot"], g["nx_r"], g["nz_r"])
        return [d, r, r.amax(2), r.amax(1), r.amax(0)]
    dr, dz, dr_psf, dz_psf = _pixels(case)
    H = _otf_grid(shape, _table(case), dr, dz, dr_psf, dz_psf)
    f = np.float32
    cut = float(f(2) * f(1.1) / f(0.525))
    dx, dy = f(1.0 / float(f(dr) * f(shape[2]))), f(1.0 / float(f(dr) * f(shape[1])))
    ky = torch.fft.fftfreq(shape[1], 1.0 / shape[1], device="cuda", dtype=torch.float64)[:, None] * float(dy)
    kx = torch.arange(shape[2] // 2 + 1, device="cuda", dtype=torch.float64)[None] * float(dx)
    kr = (ky * ky + kx * kx).sqrt()
    W = (H.conj() / (H.abs() ** 2 + float(f(0.05) * f(0.05)))) * ((1 - kr / cut) * (kr <= cut))
    return _conv(v - BACKGROUND, W)
