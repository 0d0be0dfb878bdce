"""A line's results do not depend on how its launch shares the lines out: one
thread per line or a warp per direction (chosen from the number of lines
against the GPU's resident threads), static or queue schedule, any chunk,
partly filled warps, a device-side count, a batch.  Every output of every
line is compared for equality with one launch of all lines."""
import numpy as np
import pytest
import torch

from fastqsl_gb300 import params as P
from fastqsl_gb300 import synthetic as S

pytestmark = pytest.mark.gpu

N_ALL = 1 << 18  # more lines than any kernel keeps resident threads for


@pytest.fixture(scope="module")
def field(cuda):
    spec = S.bipole4_64(3)
    return [torch.from_numpy(a).cuda().contiguous() for a in S.make_field(spec)]


@pytest.fixture(scope="module")
def seeds(cuda):
    g = torch.Generator(device="cuda").manual_seed(5)
    u = torch.rand(3, N_ALL, generator=g, device="cuda")
    z = torch.where(torch.arange(N_ALL, device="cuda") % 3 == 0, torch.zeros_like(u[2]), 20.0 * u[2])
    return [(63.0 * u[0]).contiguous(), (63.0 * u[1]).contiguous(), z.contiguous()]


CASES = {
    "soa-exact-rkf45": ("soa", P.reference_rkf45(), True),
    "soa-exact-rk4": ("soa", P.reference_rk4().copy(max_steps=300), True),
    "h4b": ("h4b", P.absolute_rkf45(tol=1e-3), False),
    "f4-twist": ("f4", P.absolute_rkf45(tol=1e-3), True),
}


def _run(store, prm, seeds, cur, n, **kw):
    from fastqsl_gb300 import api
    s = [a[:n].contiguous() for a in seeds]
    out = api.trace(store, *s, prm, s_len=0.25, curB=cur, status=True, **kw)
    return {k: v for k, v in out.items() if v is not None}


@pytest.mark.parametrize("name", list(CASES))
def test_outputs_do_not_depend_on_the_launch(field, seeds, name):
    from fastqsl_gb300 import api
    layout, prm, twist = CASES[name]
    store = api.FieldStore(*field, layout=layout)
    cur = [b.roll(1, 0).contiguous() for b in field] if twist else None
    cur = [api.as_xfast(c) for c in cur] if cur else None
    whole = _run(store, prm, seeds, cur, N_ALL, schedule="static")

    def check(out, n):
        for k, v in out.items():
            a, b = v[:n].cpu().numpy(), whole[k][:n].cpu().numpy()
            assert np.array_equal(a, b, equal_nan=a.dtype.kind == "f"), (k, n)

    for n in (1, 31, 32, 33, 64, 65, 127, 4097):
        check(_run(store, prm, seeds, cur, n, schedule="static"), n)
        check(_run(store, prm, seeds, cur, n, schedule="queue"), n)
    check(_run(store, prm, seeds, cur, N_ALL, schedule="queue"), N_ALL)
    check(_run(store, prm, seeds, cur, N_ALL, schedule="queue", chunk=96), N_ALL)
    # a device-side count below the arrays' length, few and many lines
    for n in (45, 200001):
        cnt = torch.tensor([n], dtype=torch.int64, device="cuda")
        for schedule in ("static", "queue"):
            check(_run(store, prm, seeds, cur, N_ALL, schedule=schedule, n_dev=cnt), n)


@pytest.mark.parametrize("n", [1, 33, 5000, N_ALL])
def test_batch_equals_one_launch(field, seeds, n):
    from fastqsl_gb300 import api
    store = api.FieldStore(*field, layout="h4b")
    prm = P.absolute_rkf45(tol=1e-3)
    whole = _run(store, prm, seeds, None, n, schedule="static")
    s = [a[:n].contiguous() for a in seeds]
    out = api.alloc_trace_outputs(n, status=True)
    plan = api.BatchPlan([dict(field=store, xs=s[0], ys=s[1], zs=s[2], params=prm, s_len=0.25, out=out)])
    plan.launch()
    for k, v in whole.items():
        assert torch.equal(out[k], v) or np.array_equal(out[k].cpu().numpy(), v.cpu().numpy(), equal_nan=True), k


@pytest.mark.parametrize("twist", [False, True])
def test_wide_blocks_equal_narrow_ones(field, twist):
    """Launches of many waves on bricks run in blocks of 256 threads at the
    6-block budget; the 7-block budget keeps blocks of 128."""
    from fastqsl_gb300 import api
    n = 1200037  # over 8 waves of 6 x 128 threads on every SM, last warp partly filled
    g = torch.Generator(device="cuda").manual_seed(8)
    s = [(63.0 * torch.rand(n, generator=g, device="cuda")).contiguous() for _ in range(3)]
    store = api.FieldStore(*field, layout="h4b")
    cur = [api.as_xfast(b.roll(1, 0).contiguous()) for b in field] if twist else None
    prm = P.absolute_rkf45(tol=1e-2)
    a, b = (api.trace(store, *s, prm, s_len=0.5, curB=cur, schedule="static", occupancy=k) for k in (6, 7))
    for k, v in a.items():
        assert v is None or np.array_equal(v.cpu().numpy(), b[k].cpu().numpy(), equal_nan=v.is_floating_point()), k
