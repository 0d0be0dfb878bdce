"""Polylines where the float64 restatement of MagTool.py stops with an
exception (a zero field sample divides by zero, a NaN has no cell): the GPU
stores the point the exception came at and ends the line there, in the
kernel that shares a line between eight lanes as in the one-lane kernel; and
both kernels' points are the same on either side of the number of runs at
which one takes over from the other."""
import numpy as np
import pytest

from oracle import magtool as M

pytestmark = pytest.mark.gpu


def _field():
    g = np.random.default_rng(4)
    B = [np.asfortranarray(g.uniform(-1.0, 1.0, (20, 17, 13)).astype(np.float32)) for _ in range(3)]
    for b in B:
        b[10:, :, :] = 0.0  # no field in half of the box
    return B


def _line(B, seed, maxstep, dr, monkeypatch):
    """The restatement with a failed sample giving NaN instead of raising."""
    plain = M.bnorm

    def bnorm(B, vec):
        try:
            return plain(B, vec)
        except (ZeroDivisionError, ValueError):
            return [float("nan")] * 3

    out = [np.full(maxstep, np.nan, np.float32) for _ in range(3)]
    with monkeypatch.context() as m:
        m.setattr(M, "bnorm", bnorm)
        for rng, step in ((range(maxstep // 2, maxstep), dr), (range(maxstep // 2, 0, -1), -dr)):
            M.rk4_bline(B, seed, *out, rng, step)
    return out


def _seeds(n):
    g = np.random.default_rng(12)
    s = g.uniform([0.0, 0.5, 0.5], [11.5, 16.0, 12.0], (n, 3))
    s[:4] = [[9.75, 8.1, 6.6], [9.0, 5.5, 4.5], [12.4, 3.3, 7.7], [-0.0, 2.5, 3.25]]
    return s


def _same_bits(a, b):
    assert np.array_equal(np.isnan(a), np.isnan(b))
    assert np.array_equal(a[~np.isnan(a)].view(np.int32), b[~np.isnan(b)].view(np.int32))


# 40 lines: eight lanes each; 9100: one lane each (their first 40 are compared)
@pytest.mark.parametrize("n", [40, 9100])
def test_a_zero_sample_ends_the_line(cuda, n, monkeypatch):
    from fastqsl_gb300.fastqslpy import MagTool as mt
    B, maxstep, dr = _field(), 120, 0.25
    seeds = _seeds(40)
    got = mt.TraceBlines(*B, np.concatenate([seeds, np.tile(seeds[:1], (n - 40, 1))]), maxstep=maxstep, dr=dr)
    at_zero = 0
    for s in range(40):
        ref = _line(B, seeds[s], maxstep, dr, monkeypatch)
        stored = ~np.isnan(ref[0])
        assert stored[maxstep // 2]  # every line has its seed
        for rng in (range(maxstep // 2, maxstep), range(maxstep // 2, 0, -1)):
            last = [i for i in rng if stored[i]][-1]
            at_zero += bool(ref[0][last] > 9.0) and last not in (rng[-1], rng[0])
        for a, b in zip(got, ref):
            _same_bits(a[s], b)
    assert at_zero >= 5  # lines that run into the zero half and end there


@pytest.mark.parametrize("both", [True, False])
def test_the_kernels_agree_where_one_takes_over(cuda, both):
    import torch
    from fastqsl_gb300 import _lib
    lib = _lib.load()
    g = np.random.default_rng(4)
    B = [torch.from_numpy(g.uniform(-1.0, 1.0, (13, 17, 20)).astype(np.float32)).cuda() for _ in range(3)]
    n0 = 4500 if both else 9000  # 9000 runs: eight lanes each; more: one lane each
    seeds = torch.from_numpy(np.random.default_rng(9).uniform(-0.5, 20.5, (n0 + 1, 3))).cuda()
    outs = []
    for n in (n0, n0 + 1):
        out = torch.full((3, n, 24), float("nan"), device="cuda")
        args = [*[b.data_ptr() for b in B], 20, 17, 13, seeds.data_ptr(), n]
        o = [out[k].data_ptr() for k in range(3)]
        _lib.check(lib.qsl_trace_path_both(*args, 12, 0.25, *o, 24, None) if both else
                   lib.qsl_trace_path(*args, 0, 24, 1, 0.25, *o, 24, None), "trace path")
        outs.append(out[:, :n0].cpu().numpy())
    assert np.isfinite(outs[0]).mean() > 0.2
    _same_bits(outs[0], outs[1])
