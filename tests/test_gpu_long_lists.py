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


def test_more_shells_than_sort_keys():
    """70 000 primitives of different shells: the pairs of shell pairs do not fit a sort key, so quartets are not
    merged. The few of them that the list uses, alone, are; both give the same intracule."""
    from inca_parallel_gb300 import Context, build
    build.build()
    rng = np.random.default_rng(4)
    n, used = 70000, 12
    at = np.sort(rng.permutation(n)[:used])
    tmn = np.zeros((n, 3), dtype=np.int32)
    tmn[:, 0] = np.arange(n) % 2
    alpha, xyz = np.linspace(0.3, 1.2, n), 0.5 * rng.normal(size=(n, 3))
    ijkl = rng.integers(0, used, size=(5000, 4))
    v = rng.normal(size=len(ijkl))
    v[rng.random(len(v)) < 0.3] = 0.0  # (these fail the first screening and sort last)
    pts = rng.normal(size=(200, 3))
    got = []
    with Context(0) as c:
        for a, t, x, q in ((alpha, tmn, xyz, at[ijkl]), (alpha[at], tmn[at], xyz[at], ijkl)):
            c.set_primitives(a, t, x)
            c.set_quartets((q + 1).astype(np.int32), v)
            assert c.prepare(1e-30)[2] == (v != 0).sum()
            c.grid_points(pts)
            got.append((c.eval(mode=0), c.eval(mode=1, tol=1e-10), c.records()))
    for k in ("A", "sqe", "d", "L", "C"):
        np.testing.assert_array_equal(got[0][2][k], got[1][2][k])
    scale = np.abs(got[1][0]).max()
    assert np.abs(got[0][0] - got[1][0]).max() <= 1e-13 * scale
    assert np.abs(got[0][1] - got[1][1]).max() <= 1e-10 * scale
