"""What a context answers after a call that was refused or failed half way: never records or evaluations of
mixed inputs."""
import numpy as np
import pytest

from test_gpu_merged import ctx, system  # noqa: F401

pytestmark = pytest.mark.gpu


def prepared(c, name="p"):
    s = system(name)
    c.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    c.set_quartets(s["ijkl"], s["v"])
    c.prepare(1e-12)
    c.grid_points(np.array([[0.1, -0.2, 0.3], [1.0, 0.5, 0.2]]))
    return s


def same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


def test_refused_calls_leave_the_context_alone(ctx):  # noqa: F811
    s = prepared(ctx)
    rec, iv = ctx.records(), ctx.eval(mode=0)
    bad = np.zeros_like(s["tmn"][:2])
    with pytest.raises(RuntimeError):
        ctx.set_primitives([0.5, -1.0], bad, s["xyz"][:2])
    with pytest.raises(RuntimeError):
        ctx.prepare(0.0)
    ctx.batch_clear()
    with pytest.raises(RuntimeError):
        ctx.batch_prepare(1e-12)  # no molecules
    same(ctx.records(), rec)
    np.testing.assert_array_equal(ctx.eval(mode=0), iv)
    assert ctx.prepare(1e-12)[0] == len(s["v"])
    same(ctx.records(), rec)


def test_batch_without_a_grid_is_not_evaluated(ctx):  # noqa: F811
    """A batch whose grids are refused (no such angular rule), after a list of the context's own and after
    another batch: its molecules are in, so neither the old grid nor the old molecules may be used."""
    from inca_parallel_gb300 import workloads as W
    mols = [(b, D) for _, b, D in W.batch_workload(24, max_prims=40)][:3]

    def batch(k, nang):
        ctx.batch_clear()
        for b, D in mols[:k]:
            ctx.batch_add_closed_shell(b["alpha"], b["tmn"], b["xyz"], D, [0.0], [1.0], [0.5], [nang], unique=True)
        return ctx.batch_prepare(1e-12)

    prepared(ctx)
    for _ in range(2):
        with pytest.raises(RuntimeError):
            batch(3, 51)
        for call in (lambda: ctx.batch_eval(mode=1), lambda: ctx.eval(mode=0), lambda: ctx.eval(mode=1)):
            with pytest.raises(RuntimeError):
                call()
        batch(1, 50)
        one = ctx.batch_eval(mode=1)[0]
    batch(3, 50)
    np.testing.assert_allclose(ctx.batch_eval(mode=1)[0], one, rtol=1e-7)


def test_records_of_a_long_list():
    """inca_get_records over a list of more than one block of quartets (2^20), in input order: copies of a
    list one after the other give its own records again."""
    import torch
    from inca_parallel_gb300 import Context
    s = system("single")
    with Context(0) as c:
        c.set_primitives(s["alpha"], s["tmn"], s["xyz"])
        c.set_quartets(s["ijkl"], s["v"])
        c.prepare(1e-12)
        one = c.records()
        n = (1 << 20) // len(s["v"]) + 2
        c.set_quartets(np.tile(s["ijkl"], (n, 1)), np.tile(s["v"], n))
        c.prepare(1e-12)
        before = torch.cuda.mem_get_info()[0]
        got = c.records()
        assert torch.cuda.mem_get_info()[0] >= before
        for k in one:
            np.testing.assert_array_equal(got[k], np.concatenate([one[k]] * n), err_msg=k)


def test_after_running_out_of_memory(ctx):  # noqa: F811
    """A list no device holds (2e13 quartets: the allocation is refused at once): the context has no quartets
    then, and the next job finds no error pending."""
    n = 3000
    s = prepared(ctx)
    rec, iv = ctx.records(), ctx.eval(mode=0)
    ctx.set_primitives(np.linspace(0.1, 5.0, n), np.zeros((n, 3), dtype=np.int32), np.zeros((n, 3)))
    with pytest.raises(RuntimeError, match="records|memory"):
        ctx.gen_closed_shell_dm2(np.eye(n))
    for call in (ctx.records, ctx.screening, lambda: ctx.prepare(1e-12)):
        with pytest.raises(RuntimeError):
            call()
    ctx.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    ctx.set_quartets(s["ijkl"], s["v"])
    ctx.prepare(1e-12)
    ctx.grid_points(np.array([[0.1, -0.2, 0.3], [1.0, 0.5, 0.2]]))
    same(ctx.records(), rec)
    np.testing.assert_array_equal(ctx.eval(mode=0), iv)


def test_batch_grid_used_on(ctx):  # noqa: F811
    """A single molecule on the grid of the batch before it, and a lattice tuned after a batch: nothing is left of
    the batch's molecules."""
    from inca_parallel_gb300 import workloads as W
    ctx.batch_clear()
    for _, b, D in W.batch_workload(24, max_prims=40)[:3]:
        ctx.batch_add_closed_shell(b["alpha"], b["tmn"], b["xyz"], D, [0.0], [3.0], [0.1], [110], unique=True)
    ctx.batch_prepare(1e-12)
    ctx.batch_eval(mode=1)
    s = system("p")
    ctx.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    ctx.set_quartets(s["ijkl"], s["v"])
    ctx.prepare(1e-12)
    want = ctx.eval(mode=0)
    for _ in range(2):
        got = ctx.eval(mode=1, tol=1e-8)
        assert np.abs(got - want).max() <= 1e-8 * np.abs(want).max()
        got = ctx.eval_graph(mode=1, tol=1e-8)
        assert np.abs(got - want).max() <= 1e-8 * np.abs(want).max()
    ctx.batch_prepare(1e-12)
    ctx.batch_eval(mode=1)
    ctx.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    ctx.set_quartets(s["ijkl"], s["v"])
    ctx.prepare(1e-12)
    ctx.grid_cube([0.0, 0.0, 0.0], [0.3] * 3, [8, 8, 8])
    assert ctx.autotune(tol=1e-8, reps=1)["items_per_cta"] in (4, 8, 12, 24, 48)
    ctx.set_tuning(None)


def test_failed_grid_leaves_none(ctx):  # noqa: F811
    """A lattice that no device holds (refused at once): the grid before it is gone, and is not evaluated over the new
    one's arrays; refused arguments leave it."""
    prepared(ctx)
    want = ctx.eval(mode=0)
    with pytest.raises(RuntimeError):
        ctx.grid_cube([0.0, 0.0, 0.0], [0.1] * 3, [0, 4, 4])
    with pytest.raises(RuntimeError):
        ctx.grid_scan([0.0], [1.0], [0.5], [51])
    np.testing.assert_array_equal(ctx.eval(mode=0), want)
    with pytest.raises(RuntimeError):
        ctx.grid_cube([0.0, 0.0, 0.0], [0.1] * 3, [5000, 5000, 5000])
    for call in (lambda: ctx.eval(mode=0), lambda: ctx.eval(mode=1), lambda: ctx.autotune(reps=1), ctx.grid_copy):
        with pytest.raises(RuntimeError):
            call()
    ctx.grid_points(np.array([[0.1, -0.2, 0.3], [1.0, 0.5, 0.2]]))
    np.testing.assert_array_equal(ctx.eval(mode=0), want)
