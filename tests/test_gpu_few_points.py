"""Grids of few points: the FP64 form's kernel for them (up to 128 points) and the mixed form with every
term in double-float (up to 640 points, explicit points up to 2 047 at tight tolerances), at the edges of
their tiles and ranges, against the oracle and the FP64 form.

Tolerances as in test_gpu_merged: 2 x 2^-53 M between two FP64 evaluations, 2^-42 M + F and the tolerance
itself for the mixed form.
"""
import numpy as np
import pytest

import oracle_lib as O
from test_gpu_merged import ctx, majorant, system  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["p", "d", "beyond"])
@pytest.mark.parametrize("npts", [1, 2, 31, 32, 33, 127, 128, 129, 640, 641, 2047, 2048])
def test_points(ctx, name, npts):  # noqa: F811
    s = system(name)
    ctx.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    ctx.set_quartets(s["ijkl"], s["v"])
    ctx.prepare(1e-12)
    ref = O.prepare(s, 1e-12, records=True)
    pts = 2.0 * np.random.default_rng(npts).normal(size=(npts, 3))
    ctx.grid_points(pts)
    some = slice(0, None, max(1, npts // 24))
    M, F = majorant(ref, pts[some])
    want = O.intracule(s, 1e-12, pts[some])[0]
    assert (np.abs(ctx.eval(mode=0)[some] - want) <= 2 * 2.0 ** -53 * M).all()
    for tol in (1e-5, 1e-10):
        got = ctx.eval(mode=1, tol=tol)
        assert (np.abs(got[some] - want) <= tol * np.abs(want) + 2.0 ** -42 * M + F).all()
        np.testing.assert_array_equal(ctx.eval_graph(mode=1, tol=tol), got)
        np.testing.assert_array_equal(ctx.eval_graph(mode=1, tol=tol), got)


def test_small_batch(ctx):  # noqa: F811
    """Two molecules of 150 points each in one batch, against each by itself."""
    from inca_parallel_gb300 import workloads as W
    scan = ([0.0], [1.0], [0.5], [50])
    mols = [(b, D) for _, b, D in W.batch_workload(24, max_prims=40)][:2]
    ctx.batch_clear()
    for b, D in mols:
        ctx.batch_add_closed_shell(b["alpha"], b["tmn"], b["xyz"], D, *scan, unique=True, nosym=True)
    ctx.batch_prepare(1e-12)
    got = ctx.batch_eval(mode=1, tol=1e-10)
    alone = []
    for b, D in mols:
        ctx.set_primitives(b["alpha"], b["tmn"], b["xyz"])
        ctx.gen_closed_shell_dm2(D, unique=True)
        ctx.prepare(1e-12)
        ctx.grid_scan(*scan, nosym=True)
        ctx.eval(mode=0)
        alone.append(ctx.radial_plot()[1])
    want = np.concatenate(alone)
    np.testing.assert_allclose(np.concatenate(got), want, rtol=1e-10)
