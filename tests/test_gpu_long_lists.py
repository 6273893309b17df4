"""Lists of records that go into more chunks than the few-point FP64 form has warps (4 096): s shells, every
quartet a record of its own.

Reference: the record formula over the records read back, in numpy. Tolerance: a term is rounded (10 + 3 y)
times on either side (y its exponent) and a sum of n terms n times, 2^-53 each.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrec,npts", [(131073, 3), (400000, 1), (400000, 128)])
def test_few_points_of_a_long_list(nrec, npts):
    import torch
    from inca_parallel_gb300 import Context, build
    build.build()
    rng = np.random.default_rng(nrec)
    n = 40
    with Context(0) as c:
        c.set_primitives(np.linspace(0.3, 1.2, n), np.zeros((n, 3), dtype=np.int32), 0.5 * rng.normal(size=(n, 3)))
        i, k = np.triu_indices(n)
        q = rng.permutation(len(i) ** 2)[:nrec]
        a, b = q // len(i), q % len(i)
        c.set_quartets((np.stack([i[a], i[b], k[a], k[b]], 1) + 1).astype(np.int32), rng.normal(size=nrec))
        c.prepare(1e-18)
        rec = c.records()
        assert len(rec["A"]) > 131072  # more than 4 096 chunks of 32
        pts = rng.normal(size=(npts, 3))
        c.grid_points(pts)
        before = torch.cuda.mem_get_info()[0]
        got = c.eval(mode=0)
        assert before - torch.cuda.mem_get_info()[0] <= 10 << 20  # 4 MB of partial sums, tables, sums
        np.testing.assert_array_equal(c.eval(mode=0), got)
        A = rec["A"] * rec["C"][:, :, 0].prod(1)
        for g in range(0, npts, max(1, npts // 4)):
            y = ((rec["sqe"][:, None] * (pts[g] + rec["d"])) ** 2).sum(1)
            t = A * np.exp(-y)
            allowed = 2 * 2.0 ** -53 * (np.abs(t) * (len(A) + 10 + 3 * y)).sum()
            assert abs(got[g] - t.sum()) <= allowed
