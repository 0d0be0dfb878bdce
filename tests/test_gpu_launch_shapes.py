"""Every way a launch shares its lanes out, one after the other by the number
of lines: four lanes to a line and the directions on warp pairs, two, one,
and from there a lane to a line, several turns or the work queue.  Each
line's outputs equal those of one launch of all lines, for the fast and the
exact kernels, static and queue, and for a count that only the device knows."""
import numpy as np
import pytest
import torch

from test_gpu_lockstep import CASES, N_ALL, _run, field, seeds  # noqa: F401  (fixtures)

pytestmark = pytest.mark.gpu

# lanes of the grids: 152 SMs x 4-7 blocks of 128 = 77,824-136,192; four lanes
# up to an eighth of that, two up to a quarter, one up to half
LINES = (9001, 15001, 17999, 25001, 37001, 60001, 90001)


@pytest.mark.parametrize("name", list(CASES))
def test_every_shape_gives_the_same_lines(field, seeds, name):  # noqa: F811
    from fastqsl_gb300 import api
    layout, prm, twist = CASES[name]
    store = api.FieldStore(*field, layout=layout)
    cur = [api.as_xfast(b.roll(1, 0).contiguous()) for b in field] if twist else None
    whole = _run(store, prm, seeds, cur, N_ALL, schedule="static")

    def check(out, n):
        for k, v in out.items():
            a, b = v[:n].cpu().numpy(), whole[k][:n].cpu().numpy()
            assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), (k, n)

    for n in LINES:
        for schedule in ("static", "queue"):
            check(_run(store, prm, seeds, cur, n, schedule=schedule), n)
            cnt = torch.tensor([n], dtype=torch.int64, device="cuda")
            check(_run(store, prm, seeds, cur, N_ALL, schedule=schedule, n_dev=cnt), n)


@pytest.mark.parametrize("n", LINES)
def test_batches_give_the_same_lines(field, seeds, n):  # noqa: F811
    from fastqsl_gb300 import api
    layout, prm, _ = CASES["h4b"]
    store = api.FieldStore(*field, layout=layout)
    whole = _run(store, prm, seeds, None, n, schedule="static", occupancy=6)
    s = [a[:n].contiguous() for a in seeds]
    for limit in (0, 1 << 30, 64):
        out = api.alloc_trace_outputs(n, status=True)
        cut = n // 3
        jobs = [dict(field=store, xs=s[0][p], ys=s[1][p], zs=s[2][p], params=prm, s_len=0.25,
                     out={k: None if v is None else v[p] for k, v in out.items()})
                for p in (slice(0, cut), slice(cut, n))]
        api.BatchPlan(jobs).launch(max_blocks=limit)
        for k, v in whole.items():
            assert np.array_equal(out[k].cpu().numpy(), v.cpu().numpy(), equal_nan=v.is_floating_point()), (k, limit)
