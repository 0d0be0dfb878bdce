"""Windows of a batch's line space at any first and last line: a window
traces its own lines and no other, whatever the jobs' boundaries (a job's
range is padded to a multiple of 32 lines), and windows that cover the batch
give what one launch of it gives."""
import numpy as np
import pytest
import torch

from fastqsl_gb300 import params as P

pytestmark = pytest.mark.gpu

COUNTS = (50, 77, 1, 300)  # padded to 64, 96, 32 and 320 lines


@pytest.fixture(scope="module")
def batch(cuda):
    from fastqsl_gb300 import api, synthetic as S
    store = api.FieldStore(*[torch.from_numpy(b).cuda() for b in S.make_field(S.bipole4_64(3))], layout="h4b")
    g = torch.Generator(device="cuda").manual_seed(1)
    jobs = []
    for n in COUNTS:
        s = [(61.0 * torch.rand(n, generator=g, device="cuda") + 1.0).contiguous() for _ in range(3)]
        jobs.append(dict(field=store, xs=s[0], ys=s[1], zs=s[2], params=P.absolute_rkf45(tol=1e-3), s_len=0.25,
                         out=api.alloc_trace_outputs(n, status=True)))
    return api.BatchPlan(jobs), jobs


def _clear(jobs):
    for j in jobs:
        for v in j["out"].values():
            if v is not None:
                v.fill_(-7)


def _outputs(jobs):
    return [{k: v.cpu().numpy().copy() for k, v in j["out"].items() if v is not None} for j in jobs]


# max_blocks 1 and 2: more lines than the launch has lanes (one lane to a
# line, several turns of a warp); 0: up to eight lanes to a line
@pytest.mark.parametrize("max_blocks", [0, 1, 2])
@pytest.mark.parametrize("lo,hi", [(40, -1), (41, 70), (63, 65), (1, 400), (50, 64), (33, 34), (95, 481), (0, 47)])
def test_a_window_traces_its_lines(batch, lo, hi, max_blocks):
    plan, jobs = batch
    plan.launch()
    whole = _outputs(jobs)
    _clear(jobs)
    plan.launch(lo=lo, hi=hi, max_blocks=max_blocks)
    got = _outputs(jobs)
    begin = 0
    for n, a, b in zip(COUNTS, got, whole):
        line = begin + np.arange(n)
        inside = (line >= lo) & ((line < hi) | (hi < 0))
        for k in a:
            assert np.array_equal(a[k][inside], b[k][inside], equal_nan=a[k].dtype.kind == "f"), (k, lo, hi)
            assert (a[k][~inside] == -7).all(), (k, lo, hi)
        begin += (n + 31) // 32 * 32


@pytest.mark.parametrize("step", [13, 37, 100])
def test_windows_of_any_step_cover_the_batch(batch, step):
    plan, jobs = batch
    plan.launch()
    whole = _outputs(jobs)
    _clear(jobs)
    for lo in range(0, plan.window_lines, step):
        plan.launch(lo=lo, hi=lo + step)
    for a, b in zip(_outputs(jobs), whole):
        for k in a:
            assert np.array_equal(a[k], b[k], equal_nan=a[k].dtype.kind == "f"), (k, step)
