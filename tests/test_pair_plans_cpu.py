"""The generated plans of the paired passes, on the CPU: radices, strides,
threads and shared memory of every length."""

import sys
from pathlib import Path

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "cudadecon_gb300"))
import gen_plans as G  # noqa: E402


def test_paired_plans_fit_their_tiles():
    lens = G.pair_lengths()
    assert {128, 756, 1620}.issubset(lens["x"]) and {32, 225, 1024}.issubset(lens["y"])
    # every length the batched workloads' ranges hold
    for axis, old in G.lengths().items():
        assert set(old).issubset(lens[axis])
    for axis, ls in lens.items():
        for L in ls:
            n, V, (q0, q1, q2), s0, vs = G.pair_plan(axis, L)
            assert n == (L // 2 if axis == "y" and L % 2 == 0 else L)
            assert q0 * q1 * q2 == n and min(q0, q2) >= 2 and max(q0, q1, q2) <= G.PAIR_WIDE_RADIX
            if axis == "y" and L % 4 == 0:
                assert q0 % 2 == 0
            # positions b0 s0 + b1 q2 + a2 are distinct and inside a vector
            pos = {a * s0 + b * q2 + c for a in range(q0) for b in range(q1) for c in range(q2)}
            assert len(pos) == n and max(pos) < vs
            assert 32 <= G.pair_threads((q0, q1, q2), V) <= 1024
            # twiddles, tile (z: two) and, on x, one copy of the rows beside it
            # or two in its place
            tile, rows = 16 * V * vs, 16 * V * n
            data = {"x": max(tile + rows, 2 * rows), "y": tile, "z": 2 * tile}[axis]
            assert (16 if axis == "y" else 8) * n + 8 + data <= 227 * 1024, (axis, L)
