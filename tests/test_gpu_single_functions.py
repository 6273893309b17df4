"""Shells of one function each: every subgroup is one quartet, whose polynomials are held by themselves instead of
in a table over all powers. Lists of one block and beyond, against the oracle; and the same list twice at half the
values, whose subgroups have two quartets and take the table: the same bits.

Tolerances of the evaluations as in test_gpu_merged.py.
"""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_merged import ctx, majorant  # noqa: F401

pytestmark = pytest.mark.gpu

POWERS = [(0, 0, 0), (1, 0, 0), (0, 2, 0), (0, 1, 2), (4, 0, 0), (1, 1, 1), (0, 0, 3)]


@pytest.mark.parametrize("powers", [POWERS, POWERS[:2], POWERS[:1], [(4, 4, 4)]])
@pytest.mark.parametrize("n", [1, 9, 14])  # 1, 1 035 and 5 565 quartets
def test_one_function_a_shell(ctx, n, powers):  # noqa: F811
    rng = np.random.default_rng(n)
    i, k = np.triu_indices(n)
    a, b = np.triu_indices(len(i))
    s = {"alpha": np.linspace(0.4, 1.5, n), "tmn": np.array([powers[p % len(powers)] for p in range(n)], dtype=np.int32),
         "xyz": 0.7 * rng.normal(size=(n, 3)),
         "ijkl": np.stack([i[a], i[b], k[a], k[b]], 1).astype(np.int32) + 1, "v": rng.normal(size=len(a))}
    ctx.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    ctx.set_quartets(s["ijkl"], s["v"])
    counts = ctx.prepare(1e-10)
    ref = O.prepare(s, 1e-10, records=True)
    assert list(counts) == ref["counts"].tolist()
    flags, s1, s2 = ctx.screening()
    np.testing.assert_array_equal(flags, ref["flags"])
    rec = ctx.records()
    for key in ("A", "sqe", "d", "L", "C"):
        np.testing.assert_array_equal(rec[key], ref[key], err_msg=key)
    pts = np.concatenate([np.zeros((1, 3)), rng.normal(size=(20, 3))])
    want, _ = O.intracule(s, 1e-10, pts)
    M, F = majorant(ref, pts)
    ctx.grid_points(pts)
    i64, imix = ctx.eval(mode=0), ctx.eval(mode=1, tol=1e-10)
    assert (np.abs(i64 - want) <= 2 * 2.0 ** -53 * M).all()
    assert (np.abs(imix - want) <= 1e-10 * np.abs(want) + 2.0 ** -42 * M + F).all()
    # twice at half the values
    ctx.set_quartets(np.repeat(s["ijkl"], 2, 0), np.repeat(s["v"] / 2, 2))
    assert ctx.prepare(0.5e-10) == tuple(2 * x for x in counts)
    two = ctx.screening()
    np.testing.assert_array_equal(two[0], np.repeat(flags, 2))
    np.testing.assert_array_equal(2 * two[1], np.repeat(s1, 2))
    np.testing.assert_array_equal(2 * two[2], np.repeat(s2, 2))
    assert (np.abs(ctx.eval(mode=0) - want) <= 3 * 2.0 ** -53 * M).all()
