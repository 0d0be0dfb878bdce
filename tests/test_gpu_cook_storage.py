"""CookPseudoLine's 25 results: each an allocation of its own, contiguous and
aligned as the allocator aligns, with the compacted seeds and Bz in it and
zeros in the outputs, down to no pixel at all."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _cook(sel):
    from fastqsl_gb300.fastqslpy.FastQSL import CookPseudoLine
    n = sel.size
    g = np.random.default_rng(6)
    f = lambda: torch.from_numpy(g.uniform(1.0, 9.0, n).astype(np.float32)).cuda()  # noqa: E731
    i = lambda: torch.from_numpy(g.integers(1, 7, n).astype(np.int32)).cuda()  # noqa: E731
    xe, ye, ze, fe, xs, ys, zs, fs = f(), f(), f(), i(), f(), f(), f(), i()
    b = [f() for _ in range(7)]
    flag = torch.from_numpy(sel.astype(np.int32)).cuda()
    out = CookPseudoLine(xe, ye, ze, fe, xs, ys, zs, fs, *b[:6], b[6], flag, 0.1)
    return out, (xs, ys, zs), b


@pytest.mark.parametrize("n,every", [(1, 1), (37, 5), (1024, 3), (1500, 1), (5000, 7), (300, 0)])
def test_results_own_their_memory(cuda, n, every):
    sel = (np.arange(n) % every == 0) if every else np.zeros(n, bool)
    k = int(sel.sum())
    out, seeds, b = _cook(sel)
    assert len(out) == 25
    for a in out:
        assert a.is_contiguous() and a.storage_offset() == 0
        assert a.untyped_storage().nbytes() == a.numel() * a.element_size()
        assert a.data_ptr() % 256 == 0
    assert len({a.untyped_storage().data_ptr() for a in out if a.numel()}) == sum(a.numel() > 0 for a in out)
    for a in out[:21]:
        assert a.shape == (4 * k,)
    assert int(out[21].item()) == 4 * k and out[22].dtype == torch.float64 and out[22].shape == (4 * k,)
    for a in (*out[3:21], out[22]):
        assert not a.any()
    assert [a.dtype for a in (out[6], out[10], out[14])] == [torch.int32] * 3
    # (Bz at the start and end footpoints of the selected pixels)
    assert torch.equal(out[23].cpu(), b[2].cpu()[torch.from_numpy(sel)])
    assert torch.equal(out[24].cpu(), b[5].cpu()[torch.from_numpy(sel)])
    # a pixel's four seeds lie evenly about its start footpoint (each coordinate
    # a rounded sum of numbers below 16: within 2^-21 of it)
    for a, c in zip(out[:3], seeds):
        mean = a.double().view(-1, 4).mean(1).cpu()
        assert (mean - c.cpu()[torch.from_numpy(sel)].double()).abs().max().item() <= 2.0 ** -21 if k else mean.numel() == 0
