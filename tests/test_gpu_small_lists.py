"""Lists of up to 4 096 quartets are grouped, and their records sorted, by one block each. The same list followed by
quartets of value zero, which fail the first screening, goes through the general path and has to give the
same bits.
"""
import numpy as np
import pytest

from test_gpu_merged import BASES, ctx, system  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", sorted(BASES))
@pytest.mark.parametrize("n", [1, 2, 1023, 4095, 4096])
def test_small_list_as_the_general_path(ctx, name, n):  # noqa: F811
    s = system(name)
    q = np.arange(n) % len(s["v"])
    ijkl, v = s["ijkl"][q], s["v"][q] * (1 + q)
    pts = np.random.default_rng(n).normal(size=(150, 3))
    ctx.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    out = []
    for more in (0, 4097 - n):
        ctx.set_quartets(np.concatenate([ijkl, ijkl[:1].repeat(more, 0)]), np.concatenate([v, np.zeros(more)]))
        counts = ctx.prepare(1e-12)
        rec = ctx.records()
        ctx.grid_points(pts)
        out.append([np.array(counts[1:]), *(x[:n] for x in ctx.screening()), *rec.values(), ctx.eval(mode=0),
                    ctx.eval(mode=1, tol=1e-8)])
    assert out[0][0][1] > 0
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_small_lists_at_their_ends(ctx):  # noqa: F811
    """Nothing passes; an index beyond the basis; a batch of small molecules."""
    from inca_parallel_gb300 import workloads as W
    s = system("p")
    ctx.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    ctx.grid_points(np.zeros((3, 3)))
    ctx.set_quartets(s["ijkl"], np.zeros(len(s["v"])))
    assert ctx.prepare(1e-12) == (len(s["v"]), 0, 0)
    assert (ctx.eval(mode=0) == 0.0).all()
    ctx.set_quartets(np.concatenate([s["ijkl"], [[1, 1, 1, len(s["alpha"]) + 1]]]), np.append(s["v"], 1.0))
    with pytest.raises(RuntimeError, match="index"):
        ctx.prepare(1e-12)
    mols = []
    for k in range(5):
        b = W.random_molecule(np.random.default_rng(k), 2, 5, hi=20.0)
        mols.append((b, W.closed_shell_density(b, 2, k)[0]))
    scan = ([0.0], [2.0], [0.5], [50])
    ctx.batch_clear()
    for b, D in mols:
        ctx.batch_add_closed_shell(b["alpha"], b["tmn"], b["xyz"], D, *scan, unique=True)
    assert ctx.batch_prepare(1e-12)[0] <= 4096
    got = ctx.batch_eval(mode=0)
    for (b, D), one in zip(mols, got):
        ctx.set_primitives(b["alpha"], b["tmn"], b["xyz"])
        ctx.gen_closed_shell_dm2(D, unique=True)
        ctx.prepare(1e-12)
        ctx.grid_scan(*scan)
        ctx.eval(mode=0)
        np.testing.assert_allclose(ctx.radial_plot()[1], one, rtol=1e-12)
