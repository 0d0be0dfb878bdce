"""Compaction of flagged pixels where its dispatch and its tiles can go
wrong: up to 1024 tiles of 1024 pixels a tile's block forms its own offset
from the counts, above that a scan kernel does.  The oracle is numpy; indexes
and copies are exact, the seeds are one FP32 addition each, so every
comparison is for equality."""
import numpy as np
import pytest
import torch

from fastqsl_gb300 import _lib, api, params as P

pytestmark = pytest.mark.gpu

T = 1024


@pytest.mark.parametrize("n", [1, T - 1, T, T + 1, T * T - 1, T * T, T * T + 1, 2 * T * T + 77])
@pytest.mark.parametrize("density", [0.0, 0.1, 1.0])
def test_cook_offsets(cuda, n, density):
    lib = _lib.load()
    g = np.random.default_rng(n)
    flag = np.where(g.random(n) < density, 1, 0).astype(np.int32)
    if density == 0.1:
        flag[0] = flag[-1] = 1
    face = g.integers(0, 8, n).astype(np.int32)
    xyz = g.random((3, n), dtype=np.float32) * 50
    bz = g.random((2, n), dtype=np.float32)
    d = [torch.as_tensor(a).cuda() for a in (flag, xyz[0], xyz[1], xyz[2], face, bz[0], bz[1])]
    cut = torch.full((3, 4 * n), -1, dtype=torch.float32, device="cuda")
    b0 = torch.full((2, n), -1, dtype=torch.float32, device="cuda")
    pix = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    count = torch.full((2,), 99, dtype=torch.int64, device="cuda")
    nb = lib.qsl_cook_workspace_bytes(n)
    work = torch.empty(nb, dtype=torch.uint8, device="cuda")
    stride = np.float32(0.3)
    p = [api.ptr(t) for t in d]
    _lib.check(lib.qsl_cook_pseudo_line(p[0], p[1], p[2], p[3], p[4], p[5], p[6], n, 0, 0, 0, float(stride),
                                        api.ptr(cut[0]), api.ptr(cut[1]), api.ptr(cut[2]), api.ptr(b0[0]),
                                        api.ptr(b0[1]), api.ptr(pix), api.ptr(count), api.ptr(work), nb,
                                        api.stream_handle(None)), "qsl_cook_pseudo_line")
    k = np.flatnonzero(flag == 1)
    assert count.tolist() == [k.size, 4 * k.size]
    np.testing.assert_array_equal(pix.cpu().numpy(), np.concatenate([k, np.full(n - k.size, -1)]))
    np.testing.assert_array_equal(b0.cpu().numpy()[:, :k.size], bz[:, k])
    # +u, +v, -u, -v along the axes of the face, (x, y), (x, z) or (y, z)
    want = np.repeat(xyz[:, k, None], 4, axis=2)
    for axis, (u, v) in {0: (1, 2), 1: (0, 2), 2: (0, 1)}.items():
        on = ((face[k] - 1) // 2 == axis) & (face[k] >= 1) & (face[k] <= 6)
        want[u, on, 0] += stride
        want[u, on, 2] -= stride
        want[v, on, 1] += stride
        want[v, on, 3] -= stride
    np.testing.assert_array_equal(cut.cpu().numpy()[:, :4 * k.size], want.reshape(3, -1))
    assert torch.all(cut[:, 4 * k.size:] == -1)


@pytest.mark.parametrize("rows", [(512, 512), (512, 513)])
def test_batch_tiles(cuda, rows):
    """Two plane jobs of 1024 tiles together, and of 1025: each Q map equals
    that of the job in a batch of its own."""
    from fastqsl_gb300 import serving
    fs = serving.make_fields(n_fields=1, shape=(24, 24, 20), seed=5)
    n, u, v = serving.plane_axes((0.0, 0.0, 1.0))
    jobs = [dict(field=fs["f0"], params=P.absolute_rkf45(tol=1e-2), center=(11.5, 11.5, 2.0 + k), normal=n, u=u, v=v,
                 spacing=0.02, n0=r, n1=T) for k, r in enumerate(rows)]
    both = api.PlaneQBatch(jobs)
    both.run()
    for k, j in enumerate(jobs):
        one = api.PlaneQBatch([j])
        one.run()
        torch.cuda.synchronize()
        a, b = both.Q[k], one.Q[0]
        assert torch.equal(torch.isnan(a), torch.isnan(b))
        assert torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
        one.close()
    both.close()
    for f in fs.values():
        f.close()


@pytest.mark.parametrize("n0,n1", [(3, 3), (9, 31), (33, 130), (120, 200)])
def test_shared_launches(cuda, n0, n1):
    """A batch that shares the GPU (grids capped at one thread per line, the
    pseudo-lines' at fewer) gives the Q maps of one that spreads its lines
    over idle lanes, bit for bit: a few lines, one block, several."""
    from fastqsl_gb300 import serving
    fs = serving.make_fields(n_fields=1, shape=(40, 36, 32), seed=9)
    n, u, v = serving.plane_axes((0.2, 0.1, 0.97))
    job = dict(field=fs["f0"], params=P.absolute_rkf45(tol=1e-4), center=(19.0, 17.0, 6.0), normal=n, u=u, v=v,
               spacing=0.1, n0=n0, n1=n1)
    got = []
    for share in (False, True):
        qb = api.PlaneQBatch([job, dict(job, center=(21.0, 16.0, 4.0))])
        qb.run_main(share=share)
        qb.run_post(share=share)
        torch.cuda.synchronize()
        got.append([q.clone() for q in qb.Q])
        qb.close()
    for a, b in zip(*got):
        assert torch.equal(torch.isnan(a), torch.isnan(b))
        assert torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
    for f in fs.values():
        f.close()
