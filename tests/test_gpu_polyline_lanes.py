"""The polyline kernel that shares a line between eight lanes against the
float64 restatement of MagTool.py and against the one-lane kernel (taken from
3000 lines on): every stored point equal, for line counts that fill a warp's
groups partly, seeds on nodes, faces and outside, a field with zero,
subnormal and large values, and a step that is no power of two."""
import numpy as np
import pytest

from oracle import magtool as M

pytestmark = pytest.mark.gpu


def _field(kind):
    g = np.random.default_rng(4)
    B = [np.asfortranarray(g.uniform(-1.0, 1.0, (20, 17, 13)).astype(np.float32)) for _ in range(3)]
    if kind == "zeros":       # a sample of zero field ends the line (NaN)
        for b in B:
            b[10:, :, :] = 0.0
    elif kind == "extreme":   # subnormal, tiny and large node values, zero components
        B[0] = np.asfortranarray((B[0] * np.float32(1e-41)).astype(np.float32))
        B[1][::2] *= np.float32(1e30)
        B[2][:, ::3] = 0.0
    return B


SEEDS = np.array([[3.0, 4.0, 5.0], [0.0, 0.0, 0.0], [-0.0, 2.5, 3.25], [19.0, 16.0, 12.0], [20.0, 8.0, 6.0],
                  [9.75, 8.1, 6.6], [-1.0, 3.0, 3.0], [5.0, 17.5, 12.9], [5.3, 6.1, 14.0], [21.0, 1.0, 1.0],
                  [1e-9, 1e-12, 12.999999], [12.4, 3.3, 7.7], [6.0, 16.0, 12.0]])


def _same(a, b):
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(a[~np.isnan(a)], b[~np.isnan(b)])


@pytest.mark.parametrize("kind,n,dr", [("plain", 13, 0.25), ("plain", 1, 0.3), ("plain", 5, 0.7), ("zeros", 13, 0.25),
                                       ("extreme", 13, 0.25)])
def test_lanes_equal_the_restatement(cuda, kind, n, dr):
    from fastqsl_gb300.fastqslpy import MagTool as mt
    B = _field(kind)
    got = mt.TraceBlines(*B, SEEDS[:n], maxstep=120, dr=dr)
    for s in range(n):
        ref = [np.full(120, np.nan, np.float32) for _ in range(3)]
        for rng, step in ((range(60, 120), dr), (range(60, 0, -1), -dr)):
            with np.errstate(all="ignore"):
                try:
                    M.rk4_bline(B, SEEDS[s].copy(), *ref, rng, step)
                except (IndexError, ValueError, ZeroDivisionError):
                    ref = None  # a zero field sample: the restatement raises
                    break
        for a, b in zip(got, ref or ()):
            assert _same(a[s], b), (kind, s)


def test_lanes_equal_one_lane_per_line(cuda):
    from fastqsl_gb300.fastqslpy import MagTool as mt
    B = _field("plain")
    g = np.random.default_rng(9)
    seeds = g.uniform(-0.5, 20.5, (3001, 3))
    few = [np.concatenate(v) for v in zip(*(mt.TraceBlines(*B, part, maxstep=60) for part in
                                            (seeds[:7], seeds[7:1500], seeds[1500:])))]
    many = mt.TraceBlines(*B, seeds, maxstep=60)
    for a, b in zip(few, many):
        assert _same(a, b)
