"""The work-queue schedule on lines of very different lengths within a warp:
lanes whose lines have ended take new ones, however many lines the caller
lets a warp take at a time, so the time is not that of each warp's longest
line.  Outputs equal the static schedule's."""
import numpy as np
import pytest
import torch

from fastqsl_gb300 import params as P

pytestmark = pytest.mark.gpu

N = 200000


@pytest.fixture(scope="module")
def ropes(cuda):
    """A rope of closed lines (3 % of the box, traced to the length limit)
    in a field of straight ones; seeds anywhere."""
    shape = (160, 160, 128)
    x, y, _ = torch.meshgrid(*[torch.arange(k, device="cuda", dtype=torch.float32) for k in shape], indexing="ij")
    r = (0.03 * shape[0] * shape[1] / np.pi) ** 0.5
    dx, dy = x - shape[0] / 2, y - shape[1] / 2
    w = torch.sigmoid((r - (dx * dx + dy * dy).sqrt()) * 2.0)
    field = [-dy / r * 4 * w, dx / r * 4 * w, 1.0 - w + 0.02]
    g = torch.Generator(device="cuda").manual_seed(3)
    seeds = [((k - 1) * torch.rand(N, generator=g, device="cuda")).contiguous() for k in shape]
    return [b.contiguous() for b in field], seeds


def _time(f):
    f()
    best = float("inf")
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("layout", ["h4b", "f4"])
def test_uneven_lines(ropes, layout):
    """The chunks' times lie within 1.3 of one another (2.6 where a warp traces
    its chunk 32 lines at a time) and the queue takes less than 0.75 of the
    static schedule's time (0.8 so, 0.55 with refills)."""
    from fastqsl_gb300 import api
    field, seeds = ropes
    store = api.FieldStore(*field, layout=layout)
    prm = P.absolute_rkf45(tol=1e-4)
    ref = api.alloc_trace_outputs(N)
    static = _time(lambda: api.trace(store, *seeds, prm, s_len=0.25, out=ref, schedule="static"))
    times = {}
    for chunk in (0, 8, 32, 48, 256):
        out = api.alloc_trace_outputs(N)
        times[chunk] = _time(lambda: api.trace(store, *seeds, prm, s_len=0.25, out=out, chunk=chunk))
        for k, v in out.items():
            assert v is None or np.array_equal(v.cpu().numpy(), ref[k].cpu().numpy(),
                                               equal_nan=v.is_floating_point()), (k, chunk)
    assert max(times.values()) <= 1.3 * min(times.values()), times
    assert max(times.values()) <= 0.75 * static, (times, static)


@pytest.mark.parametrize("twist", [False, True])
@pytest.mark.parametrize("n", [77825, 100001, N])
def test_exact_outputs_equal_the_static_schedule(ropes, n, twist):
    """The drop-in arithmetic, from just above the lanes of the twist kernel's
    grid (its queue starts there) to several refills of a warp."""
    from fastqsl_gb300 import api
    field, seeds = ropes
    store = api.FieldStore(*field, layout="soa")
    cur = [api.as_xfast(b.roll(1, 0).contiguous()) for b in field] if twist else None
    prm = P.reference_rk4().copy(max_steps=400)
    s = [a[:n].contiguous() for a in seeds]
    a, b = (api.trace(store, *s, prm, s_len=0.25, curB=cur, schedule=k, status=True) for k in ("static", "queue"))
    for k, v in a.items():
        assert v is None or np.array_equal(v.cpu().numpy(), b[k].cpu().numpy(), equal_nan=v.is_floating_point()), k


def test_samples_and_order_do_not_depend_on_refills(ropes):
    from fastqsl_gb300 import api
    field, seeds = ropes
    store = api.FieldStore(*field, layout="h4b")
    prm = P.absolute_rkf45(tol=1e-3)
    order = torch.randperm(N, device="cuda").to(torch.int32)
    runs = []
    for schedule in ("static", "queue"):
        count = torch.zeros(1, dtype=torch.int64, device="cuda")
        out = api.trace(store, *seeds, prm, s_len=0.25, schedule=schedule, order=order, samples=count)
        runs.append((int(count.item()), out["LineLen"].cpu().numpy(), out["end_x"].cpu().numpy()))
    assert runs[0][0] == runs[1][0]
    assert all(np.array_equal(x, y) for x, y in zip(runs[0][1:], runs[1][1:]))


@pytest.mark.parametrize("layout", ["soa", "h4b"])
def test_neighbours_and_others_in_one_launch(ropes, layout):
    """Warps whose seeds are neighbours (rows of a plane) wait for their last
    line, others refill; a warp may change from one to the other."""
    from fastqsl_gb300 import api
    field, seeds = ropes
    k = torch.arange(N // 2, device="cuda", dtype=torch.float32)
    rows = [0.25 * (k % 600) + 2.0, 0.9 * (k // 600) + 2.0, torch.full_like(k, 3.0)]
    s = [torch.cat([r, a[:N // 2]]).contiguous() for r, a in zip(rows, seeds)]
    store = api.FieldStore(*field, layout=layout)
    prm = P.reference_rkf45() if layout == "soa" else P.absolute_rkf45(tol=1e-4)
    a, b = (api.trace(store, *s, prm, s_len=0.25, schedule=q, status=True) for q in ("static", "queue"))
    for name, v in a.items():
        assert v is None or np.array_equal(v.cpu().numpy(), b[name].cpu().numpy(),
                                           equal_nan=v.is_floating_point()), name
