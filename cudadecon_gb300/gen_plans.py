"""Generate the compile-time FFT plans for every 2,3,5,7-smooth length of
the batched workloads' stack sizes that the hand-tuned registry in
csrc/static_plans.cuh does not already hold: x in [128, 1024], y in
[128, 512], z in [32, 160].

Writes csrc/static_plans_gen.cuh (those plan lists), and for the paired passes
of the plain form (csrc/fft_pair.cuh; x in [128, 2048], y in [8, 2048], z in
[16, 512]) csrc/pair_plans_gen.cuh (the plans), csrc/x_gen_dispatch.h (their
dispatch) and csrc/decon_{x,y,z}_gen_<k>.cu (their kernels, spread over several
units so that the build compiles them in parallel).

Each length has a short list of candidate plans (radix order, pencil batch
-- rows, row pairs or columns per block -- the register budget behind the
launch bounds, and for three-radix row plans the padding of the layouts
between the stages); candidate 0 is the heuristic choice:

  y, z : the most balanced pair of radices of at most 32 points (in
         registers), larger radix first; three radices when no such pair
         exists (343 = 7*7*7).  y blocks take 2048 // L rows, z blocks 16
         columns.  Candidates: half the rows (or 8 columns), the reversed
         radix order, twice the rows (or 32 columns) where the block stays
         within 1024 threads, 16 more registers per thread, and three
         radices (the most balanced triple) with the full and half batch:
         an unbalanced pair such as 125 = 25*5 leaves most threads idle in
         its large-radix stage.
  x    : (neither tuned nor compiled: the paired passes took over every x
         length of a plan)
         the most balanced three radices, smallest last (the fused epilogues
         of the x passes run in the last stage, which then has a thread for
         every butterfly), with the generic engine's row pairs per block.
         Candidates: half the row pairs, the two larger radices swapped, the
         most balanced two-radix plan where its padded middle array fits the
         tile, 16 more registers per thread, a quarter of the row pairs, and
         the swapped radices with half the row pairs.

Padding (x and y plans of three radices): each layout between two stages
can get one float2 of padding after every B, with B in PAD_CHOICES picked
by a model of the shared-memory bank conflicts of the stage that writes it
and the stage that reads it (smem_pads); one candidate per length carries
the model's padding where the model finds one.

autotune.py times the y and z candidates on the GPU, in the mixed-precision
form that runs them, and records the fastest per axis and length in
tuned_plans.json, which this script then follows.

    python cudadecon_gb300/gen_plans.py               (tuned, else candidate 0)
    python cudadecon_gb300/gen_plans.py --column k    (candidate k everywhere,
                                                       for the tuning builds)
"""

from __future__ import annotations

import argparse
import functools
import json
from pathlib import Path

import numpy as np

HERE = Path(__file__).resolve().parent
OUT = HERE / "csrc" / "static_plans_gen.cuh"
XDISPATCH = HERE / "csrc" / "x_gen_dispatch.h"
TUNED = HERE / "tuned_plans.json"
X_UNITS = 20
Y_UNITS = 8
Z_UNITS = 8
N_COLUMNS = 8
REGX = 16
PAD_CHOICES = (0, 16, 32, 64, 128)
PAD_MIN_GAIN = 0.7

REGISTERED = {32, 64, 100, 128, 256, 512, 756, 1024, 1620}
X_RANGE = (128, 1024)
Y_RANGE = (128, 512)
Z_RANGE = (32, 160)
Z_COLS = 16
MAX_THREADS = 1024


def smooth(n: int) -> bool:
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def lengths() -> dict[str, list[int]]:
    def rng(r):
        return [n for n in range(r[0], r[1] + 1) if smooth(n) and n not in REGISTERED]
    return {"x": rng(X_RANGE), "y": rng(Y_RANGE), "z": rng(Z_RANGE)}


def radices2(L: int) -> list[int] | None:
    """The most balanced pair of radices <= 32 (larger first), or None."""
    best = None
    for a in range(2, 33):
        b, r = divmod(L, a)
        if r == 0 and 2 <= b <= 32 and (best is None or max(a, b) < max(best)):
            best = (max(a, b), min(a, b))
    return list(best) if best else None


def radices3(L: int) -> list[int]:
    """The most balanced triple of radices <= 32, in descending order."""
    best = None
    for a in range(2, 33):
        if L % a:
            continue
        for b in range(2, 33):
            c, r = divmod(L // a, b)
            if (L // a) % b == 0 and 2 <= c <= 32:
                t = sorted((a, b, c), reverse=True)
                key = (t[0], -t[2])
                if best is None or key < best[0]:
                    best = (key, t)
    if best is None:
        raise ValueError(f"no three-radix plan for {L}")
    return best[1]


def radices(L: int) -> list[int]:
    """y/z plans: a pair where one exists, else three radices."""
    return radices2(L) or radices3(L)


def x_pairs(nx: int) -> int:
    """Row pairs per x tile of the generic engine (x_pairs, decon_common.cuh)."""
    p = min(8, 8192 // nx)
    if nx >= 512:
        p = min(p, 4)
    return max(p, 1)


def threads(L: int, rad: list[int], batch: int) -> int:
    """Threads of a block (splan_threads, fft_static.cuh)."""
    t = batch * (L // min(rad))
    return (t + 31) // 32 * 32


def spad_size(n: int) -> int:
    return n + (n >> 4) + 1


def x_fits(L: int, rad: list[int], P: int) -> bool:
    """A two-radix plan's padded middle array must fit the padded row tile
    the x launchers allocate (splan_rows_fit, fft_static.cuh)."""
    if threads(L, rad, P) > MAX_THREADS:
        return False
    if len(rad) == 2:
        return P * rad[1] * (rad[0] + 1) <= spad_size(P * L)
    return True


def _wavefronts64(addr: np.ndarray) -> int:
    """Shared-memory wavefronts of 8-byte accesses: addr (..., 32) float2
    indices of one warp's threads (-1: inactive); each half-warp is one
    request whose wavefronts are the most distinct words on one bank."""
    a = addr.reshape(-1, 16)
    act = np.concatenate([a >= 0, a >= 0], axis=1)
    words = np.where(act, np.concatenate([2 * a, 2 * a + 1], axis=1), -1)
    words.sort(axis=1)
    uniq = np.ones_like(words, dtype=bool)
    uniq[:, 1:] = words[:, 1:] != words[:, :-1]
    uniq &= words >= 0
    g = np.broadcast_to(np.arange(words.shape[0])[:, None], words.shape)
    cnt = np.zeros((words.shape[0], 32), dtype=np.int64)
    np.add.at(cnt, (g[uniq], words[uniq] % 32), 1)
    return int(cnt.max(axis=1).sum())


def _wavefronts128(addr: np.ndarray) -> int:
    """Wavefronts of 16-byte accesses: addr (..., 32) float4 indices (-1:
    inactive); each quarter-warp is one request."""
    a = addr.reshape(-1, 8)
    act = np.concatenate([a >= 0] * 4, axis=1)
    words = np.where(act, np.concatenate([4 * a + i for i in range(4)], axis=1), -1)
    words.sort(axis=1)
    uniq = np.ones_like(words, dtype=bool)
    uniq[:, 1:] = words[:, 1:] != words[:, :-1]
    uniq &= words >= 0
    g = np.broadcast_to(np.arange(words.shape[0])[:, None], words.shape)
    cnt = np.zeros((words.shape[0], 32), dtype=np.int64)
    np.add.at(cnt, (g[uniq], words[uniq] % 32), 1)
    return int(cnt.max(axis=1).sum())


def boundary_wavefronts(L: int, rad: list[int], V: int, s: int, B: int) -> int:
    """Wavefronts of the stores of stage s and the loads of stage s + 1 of a
    row plan (sstage in fft_static.cuh: thread b owns butterfly j of vector
    v; loads at j + r L/Q, stores at (j - k) Q + k + r Ns with k = j mod
    Ns) through the layout padded every B float2s.  The first stage's stores
    into the natural layout (B = 0) go out as 16-byte pairs when its radix is
    even (sstage's pair path)."""
    T = threads(L, rad, V)
    b = np.arange(T)
    ns = int(np.prod(rad[:s])) if s else 1
    tot = 0
    for kind, Q, nsk in (("st", rad[s], ns), ("ld", rad[s + 1], ns * rad[s])):
        LR = L // Q
        v, j = np.divmod(b, LR)
        if kind == "st" and nsk == 1 and Q % 2 == 0 and B == 0:
            r2 = np.arange(0, Q, 2)[:, None]
            t = (v[None, :] * L + j[None, :] * Q + r2) // 2
            t = np.where(b[None, :] < V * LR, t, -1)
            tot += _wavefronts128(t.reshape(len(r2), -1, 32))
            continue
        r = np.arange(Q)[:, None]
        if kind == "ld":
            e = j[None, :] + r * LR
        else:
            k = j % nsk
            e = ((j - k) * Q + k)[None, :] + r * nsk
        t = v[None, :] * L + e
        if B:
            t = t + t // B
        t = np.where(b[None, :] < V * LR, t, -1)
        tot += _wavefronts64(t.reshape(Q, -1, 32))
    return tot


def smem_pads(L: int, rad: list[int], V: int) -> list[int]:
    """Padding periods (powers of two: the padded index is a shift and an
    add) of the two layouts between the stages of a three-radix row plan:
    per boundary the fewest modelled wavefronts, kept where they save a
    quarter of that boundary's, and none at all unless the plan's two
    boundaries together drop below PAD_MIN_GAIN of the natural layout's.
    Measured on the GB300 against float2 stores in the natural layout:
    plans whose model dropped below half ran 5-13% faster padded (radix 8
    first, B = 16); those between 0.58 and 0.97 ran up to 8% slower.  The
    first stage now stores 16-byte pairs into the natural layout, which
    removes most of what the padding did, so the padded plan is one
    candidate among the others for the tuner to measure."""
    return list(_smem_pads(L, tuple(rad), V))


@functools.lru_cache(maxsize=None)
def _smem_pads(L: int, rad: tuple[int, ...], V: int) -> tuple[int, int]:
    if len(rad) != 3:
        return (0, 0)
    nat = [boundary_wavefronts(L, list(rad), V, s, 0) for s in range(2)]
    pads, cost = [], []
    for s in range(2):
        c = {B: boundary_wavefronts(L, list(rad), V, s, B) for B in PAD_CHOICES}
        best = min(c, key=lambda B: (c[B], B))
        if c[best] > 0.75 * nat[s]:
            best = 0
        pads.append(best)
        cost.append(c[best])
    # the padded index costs instructions of its own: pad only where the
    # model removes more than PAD_MIN_GAIN of the two boundaries' wavefronts
    if sum(cost) > PAD_MIN_GAIN * sum(nat):
        return (0, 0)
    return tuple(pads)


def candidates(axis: str, L: int) -> list[tuple[list[int], int, int, list[int]]]:
    """Candidate (radices, batch, extra registers, paddings) of one length,
    candidate 0 first."""
    out: list[tuple[list[int], int, int, list[int]]] = []

    def add(rad, b, rx=0, padded=False):
        rad = list(rad)
        if axis == "x" and not x_fits(L, rad, b):
            return
        if axis != "x" and threads(L, rad, b) > MAX_THREADS:
            return
        pads = smem_pads(L, rad, b) if padded and axis != "z" else [0, 0]
        if padded and pads == [0, 0]:
            return
        c = (rad, b, rx, pads)
        if c not in out:
            out.append(c)

    if axis == "x":
        base, P = radices3(L), x_pairs(L)
        swapped = [base[1], base[0], base[2]]
        add(base, P)
        add(base, max(1, P // 2))
        add(swapped, P)
        pair = radices2(L)
        if pair:
            add(pair, P)
        add(base, P, REGX)
        add(base, max(1, P // 4))
        add(swapped, max(1, P // 2))
        add(base, max(1, P // 2), padded=True)
    else:
        base = radices(L)
        b = max(1, 2048 // L) if axis == "y" else Z_COLS
        add(base, b)
        add(base, max(1, b // 2))
        add(list(reversed(base)), b)
        add(base, 2 * b)
        add(base, b, REGX)
        if len(base) == 2:
            try:
                tri = radices3(L)
            except ValueError:
                tri = None
            if tri:
                add(tri, b)
                add(tri, max(1, b // 2))
                add(tri, b, padded=True)
    assert out, f"no plan within {MAX_THREADS} threads for {axis} length {L}"
    return out


def choose(axis: str, L: int, column: int | None,
           tuned: dict) -> tuple[list[int], int, int, list[int]]:
    c = candidates(axis, L)
    if column is not None:
        return c[column] if column < len(c) else c[0]
    t = tuned.get(axis, {}).get(str(L))
    if t:
        pick = (t["radices"], t["batch"], t.get("regx", 0), t.get("pads", [0, 0]))
        if pick in c:
            return pick
    return c[0]


# ---------------------------------------------------------------- paired plans
PAIR_X_RANGE = (128, 2048)
PAIR_Y_RANGE = (8, 2048)
PAIR_Z_RANGE = (16, 512)
PAIR_MAX_RADIX = 16
PAIR_Y_RADIX = 18  # y 324 as 18 9 took 30-37 us a pass on 108 x 324 x 525, as 6 9 3 35-44 us
PAIR_X_RADIX = 12  # x 256 as 4 8 8 took 17 us in x ratio, as 16 16 30 us
PAIR_THREE_RADIX = 27
# odd heights: two radices to 35 where three need one above 9 (each round trip costs
# an odd height more: 525 as 25 21 took 30 us a pass on 64 x 525 x 384, as 7 15 5 45)
PAIR_WIDE_RADIX = 35
PAIRP = HERE / "csrc" / "pair_plans_gen.cuh"


def pair_two(L: int, most: int) -> tuple[int, int, int] | None:
    """The most balanced two radices of at most `most` points, larger first."""
    c = [(a, 1, L // a) for a in range(2, most + 1) if L % a == 0 and 2 <= L // a <= a]
    return min(c, default=None)


def pair_lengths() -> dict[str, list[int]]:
    def rng(r, points):
        return [n for n in range(r[0], r[1] + 1) if smooth(n) and pair_radices(*points(n))]
    return {"x": rng(PAIR_X_RANGE, lambda n: (n, False)), "y": rng(PAIR_Y_RANGE, pair_y_points),
            "z": rng(PAIR_Z_RANGE, lambda n: (n, False))}


def pair_y_points(L: int) -> tuple[int, bool]:
    """Points of the y transform of height L, and whether it starts even."""
    return (L // 2, L % 4 == 0) if L % 2 == 0 else (L, False)


def pair_radices(L: int, even_first: bool, most: int = PAIR_MAX_RADIX) -> tuple[int, int, int] | None:
    """Radices (Q0, Q1, Q2) of a paired plan, Q1 = 1 for two.  Two radices of at
    most `most` points where they exist (one shared round trip less), else the most
    balanced three; the smallest last (stage C holds the rows' values too), the
    largest in the middle (stage B touches no global memory).  even_first: Q0
    is even.  Radices up to `most` or 16 and then 27 where that leaves no plan (625 = 5 25 5); None
    where that does not either (1715 = 5 7^3)."""
    best = None
    for a in range(2, PAIR_THREE_RADIX + 1):
        if L % a:
            continue
        for b in range(1, PAIR_THREE_RADIX + 1):
            if (L // a) % b:
                continue
            c = L // a // b
            if not 2 <= c <= PAIR_THREE_RADIX or (even_first and a % 2):
                continue
            two, m = b == 1, max(a, b, c)
            key = (m > most, m > max(most, PAIR_MAX_RADIX), not two, m, 0 if two else -min(a, b, c), c, -b)
            if best is None or key < best[0]:
                best = (key, (a, b, c))
    return best[1] if best else None


def _slots(addr: np.ndarray) -> int:
    """Wavefronts of one 16-byte access per thread: addr (threads,) float4
    indices, quarter-warps of 8 threads, 8 slots of 16 bytes a wavefront."""
    a = addr[: len(addr) // 8 * 8].reshape(-1, 8)
    cnt = np.zeros((len(a), 8), dtype=np.int64)
    np.add.at(cnt, (np.arange(len(a))[:, None], a % 8), 1)
    return int(cnt.max(axis=1).sum())


@functools.lru_cache(maxsize=None)
def pair_strides(L: int, rad: tuple[int, int, int], V: int, axis: str, odd: bool) -> tuple[int, int]:
    """Strides (S0 of the first digit, VS of a vector) of the shared tile with
    the fewest modelled wavefronts over the three stages' accesses, smallest
    first.  x: stage A's threads run over the vectors first.  y: the threads
    of stages A and C run over 4 butterflies, then the vectors; odd heights:
    those of stage A over a vector, those that regroup rows over 4 pairs of
    rows, then the vectors."""
    q0, q1, q2 = rad
    ka, kb, kc = q1 * q2, q0 * q2, q0 * q1
    best = None
    def runs(n):  # 4 consecutive, then the vectors
        i = np.arange(V * (n // 4) * 4)
        return i // (4 * V) * 4 + i % 4, i // 4 % V

    for s0 in range(ka, ka + 8):
        for vs in range((q0 - 1) * s0 + ka, (q0 - 1) * s0 + ka + (8 if V > 1 else 1)):
            i = np.arange(V * ka)
            if axis == "x":
                j, v = i // V, i % V
            elif odd:
                j, v = i % ka, i // ka
            else:
                j, v = runs(ka)
            cost = q0 * _slots(v * vs + j)
            if odd:
                m, v = runs(L // 4)
                for e in (2 * m, 2 * m + 1):
                    cost += 2 * _slots(v * vs + e // ka * s0 + e % ka)
            if q1 > 1:
                i = np.arange(V * kb)
                v, w = i // kb, i % kb
                cost += q1 * _slots(v * vs + w // q2 * s0 + w % q2)
            if axis == "x":
                i = np.arange(V * kc)
                v, k = i // kc, i % kc
            else:
                k, v = runs(kc)
            cost += q2 * _slots(v * vs + k % q0 * s0 + k // q0 * q2)
            key = (cost, vs)
            if best is None or key < best[0]:
                best = (key, (s0, vs))
    return best[1]


def pair_threads(rad, V: int) -> int:
    q0, q1, q2 = rad
    k = max(q1 * q2, q0 * q1, q0 * q2 if q1 > 1 else 0)
    return (V * k + 31) // 32 * 32


def pair_x_warps(L: int, rad, V: int) -> int:
    """Resident warps per SM of the x passes with V pairs a block: max(4 max(rad)
    + 24, 8 rad[2] + 12) registers a thread; stage B's twiddles, tile and one copy of the rows in
    shared memory (227 KB an SM, 1 KB of it kept per block)."""
    t = pair_threads(rad, V)
    if t > 1024:
        return 0
    smem = 16 * V * (L + 32) + 16 * V * L + 8 * rad[0] * rad[1] + 1024
    return min(65536 // (t * max(4 * max(rad) + 24, 8 * rad[2] + 12)), 227 * 1024 // smem) * t // 32


def pair_z_warps(L: int, rad, V: int) -> int:
    """Resident warps per SM of the z pass with V column pairs a block: 4
    max(rad) + 56 registers a thread, twiddles and two tiles in shared memory."""
    t = pair_threads(rad, V)
    return min(65536 // (t * (4 * max(rad) + 56)), 227 * 1024 // (8 * L + 32 * V * L + 1024)) * t // 32


def pair_y_odd_kx(L: int, two: bool) -> int:
    """Neighbouring kx per block of an odd height: few, since every round trip
    ends at a barrier (64 x 441 x 384: 23 us a pass with 2, 25 with 4, 31 with 8),
    but more where two radices leave few threads per kx (225: 16 us with 4, 19
    with 2) and one where three radices make a block of many (1215: 35 with 1, 41
    with 2 on 32 x 1215 x 384)."""
    if L < 100:
        return 8
    if L <= (384 if two else 180):
        return 4
    return 2 if two or L < 1000 else 1


def pair_plan(axis: str, L: int) -> tuple[int, int, tuple[int, int, int], int, int]:
    """(transform length, vectors per block, radices, S0, VS) of one length.
    x: 2 pairs (half a slot block of the layout), 4 where that
    keeps more warps on an SM (810 at 180 slices of 600 rows: x ratio 308 us
    with 4, 390 with 2; 1024: 282 and 234); y: neighbouring kx for about 128 threads
    at even heights; z: 16 column pairs
    (256-byte runs), 8 past 144 slices (210: 47 us a pass with 8, 51 with 16 and 55 with
    4 on 210 x 256 x 384) or where that keeps more warps on an SM, 4 where 8 do not fit."""
    if axis == "x":
        rad = pair_radices(L, False, PAIR_X_RADIX)
        if max(rad) > 16 and rad[1] > 1 and (pair_two(L, PAIR_WIDE_RADIX) or (0, 0, 99))[2] <= 25:
            # 875 as 35 25 with 3 pairs: 548 us an iteration of 100 x 225 x 875; as 7 25 5
            # 600 to 650 us (one block an SM), as 35 25 with 2 or 4 pairs 580 and 570 us
            rad = pair_two(L, PAIR_WIDE_RADIX)
            return (L, 3, rad, *pair_strides(L, rad, 3, "x", False))
        V = 4 if pair_x_warps(L, rad, 4) > 1.1 * pair_x_warps(L, rad, 2) else 2
        return (L, V, rad, *pair_strides(L, rad, V, "x", False))
    if axis == "y":
        n, even = pair_y_points(L)
        rad = pair_radices(n, even, PAIR_Y_RADIX)
        if n == L:
            if max(rad) > 9 and rad[1] > 1:
                rad = pair_two(n, PAIR_WIDE_RADIX) or rad
            V = pair_y_odd_kx(n, rad[1] == 1)
        else:
            # two where four take more than 256 threads (810: 50 and 38 us a pass
            # against 51 and 45 on 64 x 810 x 384; 1024, 256 threads: 47 us with 4, 49 with 2)
            V = max(4, round(128 / pair_threads(rad, 8) * 8)) & ~1
            if pair_threads(rad, V) > 256:
                V = 2
        return (n, V, rad, *pair_strides(n, rad, V, "y", n == L))
    rad = pair_radices(L, False)
    # two radices to 24 (25 past 300) where three leave few columns a block: 147 as
    # 21 7 took 41 us on 147 x 256 x 384, as 7 7 3 51 us; 384 as 24 16 82, as 8 8 6
    # 111; but 175 as 25 7 62, as 5 7 5 50
    if rad[1] > 1:
        rad = pair_two(L, 25 if L > 300 else 24) or rad
    V = 8 if L > 144 or pair_z_warps(L, rad, 8) > 1.2 * pair_z_warps(L, rad, 16) else 16
    if not pair_z_warps(L, rad, V):
        V = 4
    return (L, V, rad, rad[1] * rad[2], L)


def _unit(axis: str, k: int, lens: list[int], body: list[str], header: str) -> None:
    out = ["// Generated by cudadecon_gb300/gen_plans.py (do not edit): paired "
           f"{axis}-pass kernels",
           f"// of the lengths {', '.join(map(str, lens))}.",
           f'#include "{header}"', '#include "pair_plans_gen.cuh"', '#include "x_gen_dispatch.h"', "",
           "namespace cdx {", ""] + body + ["}  // namespace cdx", ""]
    (HERE / "csrc" / f"decon_{axis}_gen_{k}.cu").write_text("\n".join(out))


def pair_units() -> dict:
    """Write the paired plans, their kernels' units and the dispatch."""
    lens = pair_lengths()
    plans = {a: {L: pair_plan(a, L) for L in lens[a]} for a in lens}
    kinds = {
        "x": {
            "pxgen_fwd": ("const PairGeom& g, const float2* tw, const float* X, float* Xm1, "
                          "const float* lam, int predict, float bg, float2* S", "px_fwd_go", X_UNITS),
            "pxgen_ratio": ("const PairGeom& g, const float2* tw, float2* S, const float* raw, "
                            "const float* mean, float eps", "px_ratio_go", X_UNITS),
            "pxgen_update": ("const PairGeom& g, const float2* tw, const float2* S, const float* Y, "
                             "float* Xout, float* G, int dots, RLWork* w, float* lam_next, "
                             "float eps", "px_update_go", X_UNITS),
        },
        "y": {"pygen": ("const PairGeom& g, const float2* tw, float2* S, bool inv", None, Y_UNITS)},
        "z": {"pzgen": ("const PairGeom& g, const float2* tw, float2* S, const OtfDev& otf, "
                        "bool conj", "pz_mode", Z_UNITS)},
    }
    size = {"x": "g.nx", "y": "g.ny", "z": "g.nz"}
    decl, disp = [], []
    for axis, ks in kinds.items():
        tail = "cudaStream_t st, bool fwd_only, bool* done" if axis == "z" else "cudaStream_t st, bool* done"
        units: dict[int, list[str]] = {}
        for name, (args, go, n) in ks.items():
            names = [a.split()[-1].lstrip("*&") for a in (args + ", " + tail).split(", ")]
            for k in range(n):
                decl.append(f"int {name}_{k}({args}, {tail});")
                body = units.setdefault(k, [])
                body.append(f"int {name}_{k}({args}, {tail}) {{")
                body.append(f"  switch ({size[axis]}) {{")
                for L in lens[axis][k::n]:
                    V = plans[axis][L][1]
                    fn = go or ("py_eo_go" if L % 2 == 0 else "py_zz_go")
                    body.append(f"    case {L}:")
                    body.append("      *done = true;")
                    body.append(f"      return {fn}<PP{axis.upper()}{L}, {V}>({', '.join(names[:-1])});")
                body += ["    default:", "      return 0;", "  }", "}", ""]
            calls = "\n".join(f"  if ((rc = {name}_{k}({', '.join(names)})) || *done) return rc;"
                              for k in range(n))
            disp.append(f"inline int {name}({args}, {tail}) {{\n  int rc = 0;\n  *done = false;\n"
                        f"{calls}\n  return 0;\n}}")
        hdr = {"x": "decon_px.cuh", "y": "decon_py.cuh", "z": "decon_pz.cuh"}[axis]
        for k, body in units.items():
            _unit(axis, k, lens[axis][k::len(units)], body, hdr)
    XDISPATCH.write_text(
        "// Generated by cudadecon_gb300/gen_plans.py (do not edit): dispatch of the\n"
        "// paired passes to the units decon_{x,y,z}_gen_<k>.cu.  Each function sets\n"
        "// *done when its length has a plan.\n"
        "#pragma once\n\n#include \"pair_layout.cuh\"\n\nnamespace cdx {\n\n" + "\n".join(decl) +
        "\n\n" + "\n\n".join(disp) + "\n\n}  // namespace cdx\n")
    out = ["// Generated by cudadecon_gb300/gen_plans.py (do not edit): plans of the paired",
           "// passes, PP<axis><length> = PPlan<points, Q0, Q1, Q2, S0, VS> (fft_pair.cuh).  A",
           "// y plan of an even height transforms half of it.",
           "#pragma once", "", '#include "fft_pair.cuh"', "", "namespace cdx {", ""]
    for axis in "xyz":
        for L, (n, V, rad, s0, vs) in plans[axis].items():
            out.append(f"using PP{axis.upper()}{L} = PPlan<{n}, {rad[0]}, {rad[1]}, {rad[2]}, {s0}, {vs}>;")
        out += ["", f"// length, points, vectors per block, radices of the {axis} plans",
                f"#define CDX_P{axis.upper()}_PLANS(F) \\"]
        out += [f"  F({L}, {n}, {V}, {rad[0]}, {rad[1]}, {rad[2]}) \\"
                for L, (n, V, rad, s0, vs) in plans[axis].items()]
        out += [""]
    out += ["}  // namespace cdx", ""]
    (HERE / "csrc" / PAIRP.name).write_text("\n".join(out))
    return plans


def generate(column: int | None = None) -> dict:
    """Write the generated sources; returns the chosen plans per axis."""
    tuned = json.loads(TUNED.read_text()) if column is None and TUNED.exists() else {}
    lens = lengths()
    plans = {a: {L: choose(a, L, column, tuned) for L in lens[a]} for a in lens}
    src = "tuned_plans.json" if tuned else ("candidate column %d" % column if column is not None
                                             else "candidate 0")
    lines = [
        "// Generated by cudadecon_gb300/gen_plans.py (do not edit): compile-time",
        "// plans for the 2,3,5,7-smooth x lengths in [128, 1024], y lengths in",
        "// [128, 512] and z lengths in [32, 160] outside the hand-tuned registry of",
        "// static_plans.cuh; x plans are types SPX<L>, z plans SPZ<L>, y plans",
        f"// SP<L>.  Plans from {src}.",
        "#pragma once",
        "",
    ]

    def block(name, items):
        return [f"#define {name}(F) \\"] + [f"  F({i}) \\" for i in items] + [""]

    lines += block("CDX_GEN_SPLANS", [f"{L}, {', '.join(map(str, c[0]))}"
                                      for L, c in plans["y"].items()])
    lines += block("CDX_GEN_Z_SPLANS", [f"{L}, {', '.join(map(str, c[0]))}"
                                        for L, c in plans["z"].items()])
    lines += block("CDX_GEN_Y_PLANS", [f"{L}, {c[1]}, {c[2]}, {c[3][0]}, {c[3][1]}"
                                       for L, c in plans["y"].items()])
    lines += block("CDX_GEN_Z_PLANS", [f"{L}, {c[1]}, {c[2]}" for L, c in plans["z"].items()])
    OUT.write_text("\n".join(lines) + "\n")
    pair_units()
    return plans


def main() -> None:
    ap = argparse.ArgumentParser(description=__doc__.split("\n\n")[0])
    ap.add_argument("--column", type=int, default=None,
                    help="use candidate COLUMN for every length (tuning builds)")
    a = ap.parse_args()
    plans = generate(a.column)
    print(f"{OUT}: {len(plans['y'])} y, {len(plans['z'])} z and {len(plans['x'])} x plans")


if __name__ == "__main__":
    main()
