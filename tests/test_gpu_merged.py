"""Merged records (one per group of quartets that share their Gaussian) against the CPU oracle, which
evaluates every quartet by itself.

Bases at the edges of the merging rule: s shells (total degree 0), p (4), d (8), a whole g shell (16,
the largest merged degree), powers beyond it (products stay), shells with single components (few
quartets and high powers: products or merged by cost), the same shell listed twice and a centre at
-0, and more quartets in one group than a warp takes at a time.

Tolerances, from the oracle's own records, with the error model of a term (mixed_eval.cu):
M(r) = sum_q |A_q| E P (10 + 2 L + 3 |r'|^2), P = prod_d sum_k |C_dk| |r'_d|^k, L the sum of the degrees.
Both sides round every term within it, FP64 by 2^-53 M each and double-float by 2^-42 M. FP32 numbers
end at 2^-126: a Gaussian below it is zero and a record below 2^-120 is left out, which takes at most
F(r) = 2^-119 sum_q P / kappa (kappa: the scale of the normalised polynomials). The mixed form adds
its tolerance.
"""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

A0, A1, B0 = (0.0, 0.0, 0.0), (-0.0, 0.0, -0.0), (0.3, -0.8, 1.1)
FULL = {l: [(a, b, l - a - b) for a in range(l, -1, -1) for b in range(l - a, -1, -1)] for l in range(5)}


def shell(alpha, l, at):
    return [(alpha, t, at) for t in FULL[l]]


BASES = {
    "s": shell(0.7, 0, A0) + shell(2.1, 0, B0) + shell(0.4, 0, B0),
    "p": shell(0.9, 1, A0) + shell(0.5, 1, B0) + shell(1.7, 0, B0),
    "d": shell(1.1, 2, A0) + shell(0.6, 1, B0),
    "g": shell(0.8, 4, A0) + shell(0.5, 0, B0),
    "beyond": [(0.9, (4, 4, 4), A0), (0.6, (3, 0, 2), B0), (0.7, (0, 1, 0), A0)],
    "single": [(0.9, (1, 1, 1), A0), (0.6, (2, 0, 2), B0), (1.3, (0, 0, 4), A0), (0.5, (1, 0, 0), B0)],
    "twice": shell(0.9, 1, A0) + shell(0.9, 1, A1) + shell(0.5, 1, B0)[1:],
}


@pytest.fixture(scope="module")
def ctx():
    from inca_parallel_gb300 import build
    build.build()
    from inca_parallel_gb300 import Context
    c = Context(0)
    yield c
    c.close()


def system(name):
    prims = BASES[name]
    n = len(prims)
    rng = np.random.default_rng(sum(map(ord, name)))
    i, k = np.triu_indices(n)
    a, b = (x.reshape(-1) for x in np.meshgrid(np.arange(len(i)), np.arange(len(i)), indexing="ij"))
    ijkl = np.stack([i[a], i[b], k[a], k[b]], 1).astype(np.int32) + 1
    keep = rng.permutation(len(ijkl))[:3000]  # any order, and any part, of the list
    return {"alpha": np.array([p[0] for p in prims]), "tmn": np.array([p[1] for p in prims], dtype=np.int32),
            "xyz": np.array([p[2] for p in prims]), "ijkl": ijkl[keep], "v": rng.normal(size=len(keep))}


def majorant(rec, pts):
    """M and F at every point."""
    cu = np.log(2.0) ** -0.5  # u = cu r', E = 2^-|u|^2
    M, F = np.zeros(len(pts)), np.zeros(len(pts))
    n = 10 + 2 * rec["L"].sum(1)
    for g, r in enumerate(pts):
        u = np.abs(rec["sqe"][:, None] * (r + rec["d"]))
        y = (u * u).sum(1)
        P = kappa = 1.0
        for x in range(3):
            v, k = np.zeros(len(y)), np.zeros(len(y))
            for m in range(17):
                on = m <= rec["L"][:, x]
                c = np.abs(rec["C"][:, x, m])
                v = np.where(on, v * u[:, x] + c, v)
                k = np.where(on, np.maximum(k, c * cu ** (m - rec["L"][:, x])), k)
            P, kappa = P * v, kappa * np.where(k > 0, k, 1.0)
        M[g] = (np.abs(rec["A"]) * np.exp(-y) * P * (n + 3 * y)).sum()
        F[g] = 2.0 ** -119 * (P / kappa).sum()
    return M, F


@pytest.mark.parametrize("name", sorted(BASES))
def test_merged_records_match_oracle(ctx, name, monkeypatch):
    s = system(name)
    ctx.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    ctx.set_quartets(s["ijkl"], s["v"])
    counts = ctx.prepare(1e-12)
    ref = O.prepare(s, 1e-12, records=True)
    assert list(counts) == ref["counts"].tolist()
    rec = ctx.records()
    for k in ("A", "sqe", "d", "L", "C"):
        np.testing.assert_array_equal(rec[k], ref[k], err_msg=k)
    rng = np.random.default_rng(5)
    pts = np.concatenate([np.zeros((1, 3)), rng.normal(size=(60, 3)), 4.0 * rng.normal(size=(9, 3))])
    want, _ = O.intracule(s, 1e-12, pts)
    M, F = majorant(ref, pts)
    ctx.grid_points(pts)
    assert (np.abs(ctx.eval(mode=0) - want) <= 2 * 2.0 ** -53 * M).all()
    assert (np.abs(ctx.eval(mode=1, tol=1e-10) - want) <= 1e-10 * np.abs(want) + 2.0 ** -42 * M + F).all()
    # the lattice form, and the one-pass form on a grid of its size, against the FP64 form
    monkeypatch.setenv("INCA_DROP_FRACTION", "0")
    ctx.grid_cube([0.2, 0.0, -0.1], [0.3, 0.25, 0.2], [9, 10, 17])
    M, F = majorant(ref, ctx.grid_copy(weights=False)["r"])
    assert (np.abs(ctx.eval(mode=1) - ctx.eval(mode=0)) <= 2.0 ** -42 * M + F).all()
    monkeypatch.delenv("INCA_DROP_FRACTION")
    ctx.grid_scan([0.0], [3.0], [0.15], [302], nosym=True)
    g = ctx.grid_copy(cmap=True)
    M, F = (np.bincount(g["cmap"] - 1, g["w"] * x, minlength=ctx.nradi) for x in majorant(ref, g["r"]))
    ctx.eval(mode=0)
    I64 = ctx.radial_plot()[1]
    for tol in (1e-6, 1e-10):
        ctx.eval(mode=1, tol=tol)
        assert (np.abs(ctx.radial_plot()[1] - I64) <= tol * np.abs(I64) + 2.0 ** -42 * M + F).all()


def test_denormal_coefficients(ctx):
    """A centre 1e-40 off its neighbour leaves degree-0 coefficients below FP32's normal range: their
    majorant must stay finite, or the thresholds vanish and every term is corrected. Same work as with
    the two centres equal. (No term needs a correction at 1e-4 of a sum of positive amplitudes: FP32 terms
    err by less than 2^-24 (10 + 2 L + 3 |u|^2).)"""
    done = []
    for off in (0.0, 1e-40):
        prims = shell(0.9, 1, A0) + shell(0.5, 0, (off, off, off)) + shell(0.4, 0, B0)
        n = len(prims)
        ctx.set_primitives([p[0] for p in prims], [p[1] for p in prims], [p[2] for p in prims])
        ijkl = np.stack([x.reshape(-1) for x in np.indices((n,) * 4)], 1) + 1
        ctx.set_quartets(ijkl.astype(np.int32), np.ones(len(ijkl)))
        ctx.prepare(1e-12)
        ctx.grid_scan([0.0], [3.0], [0.15], [302], nosym=True)
        ctx.eval(mode=1, tol=1e-4)
        done.append(ctx.stats()["corrected_terms"])
    assert done[0] < n**4 * 302 * 10  # half of the terms
    assert abs(done[1] - done[0]) <= 0.01 * done[0] + 100


@pytest.mark.parametrize("name", ["s", "p", "d", "g", "single"])
def test_cube_with_a_budget(ctx, name):
    """The lattice form at a tolerance (left-out records and records in plain FP32 share a tenth of it),
    ragged tiles, against the FP64 form."""
    s = system(name)
    ctx.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    ctx.set_quartets(s["ijkl"], s["v"])
    ctx.prepare(1e-12)
    ref = O.prepare(s, 1e-12, records=True)
    ctx.grid_cube([0.2, 0.0, -0.1], [0.3, 0.25, 0.2], [17, 18, 35])
    M, F = majorant(ref, ctx.grid_copy(weights=False)["r"][::97])
    I64 = ctx.eval(mode=0)
    for tol in (1e-4, 1e-10):
        err = np.abs(ctx.eval(mode=1, tol=tol) - I64)[::97]
        assert (err <= 0.1 * tol * np.abs(I64).max() + 2.0 ** -42 * M + F).all()
