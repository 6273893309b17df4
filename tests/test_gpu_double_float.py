"""The lattice form (double-float throughout) against the FP64 form on sums of positive terms: its rounding
errors have no preferred sign.

A term is three factors of the exponential times a polynomial. The steps of the exponential leave each factor
2.3e-14 rms off, and a lattice of at least 33 points an axis averages as many factors of a Gaussian an axis:
sqrt(3 / 33) 2.3e-14 = 7e-15 for the mean over the lattice, of which five times are allowed. (A low part that
is not below 2^-24 of its high part fails this: products of two low parts are dropped, and those of the
exponential's have one sign, 9e-14 of the sum where x^2/2 stays in them.)
"""
import numpy as np
import pytest

from test_gpu_merged import BASES, ctx  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["s", "p"])
@pytest.mark.parametrize("step", [0.05, 0.11, 0.17])
def test_lattice_errors_have_no_sign(ctx, name, step, monkeypatch):  # noqa: F811
    prims = BASES[name]
    n = len(prims)
    ctx.set_primitives([p[0] for p in prims], [p[1] for p in prims], [p[2] for p in prims])
    ijkl = np.stack([x.reshape(-1) for x in np.indices((n,) * 4)], 1) + 1
    ctx.set_quartets(ijkl.astype(np.int32), np.ones(len(ijkl)))
    ctx.prepare(1e-12)
    monkeypatch.setenv("INCA_DROP_FRACTION", "0")
    ctx.grid_cube([0.1, 0.0, -0.1], [step] * 3, [40, 33, 37])
    want = ctx.eval(mode=0)
    off = (ctx.eval(mode=1) - want) * np.sign(want)
    assert abs(off.sum()) <= 5 * 7e-15 * np.abs(want).sum()
