"""The performance cases of the framework: what its users run, over the sizes they run it at.

Each case is one whole job through the Python binding, as the `inca_gpu` driver or a script runs
it: molecule and DM2 in, screening, grid, evaluation, reduction, results on the host. Molecules are
CH4 (27 primitives, the benchmark's basis; its DM2 goes in from host memory, as a `.dm2p` file's
records do) or seeded random molecules of the benchmark's batch (s, p and d shells, exponents up to
200; their symmetry-unique DM2 is generated on the device from the 1-RDM). The tolerance of the
mixed form is 1e-10, the default of the driver and of `inca_eval`; thresh is 1e-12, the reference's.

  job       what a user does
  points    intracule_at_zero / intracule_two_points and short lists of explicit points
  integral  radial_integral on the automatic multicentre grid
  plot      radial_plot, I(s) shell by shell
  cube      cubeintra, the intracule on a lattice
  batch     radial_plot of several molecules at once
  records   inca_eval_records_noalloc on records and points that the caller keeps on the device
"""
import ctypes
import functools
import math

import numpy as np
import torch

from inca_parallel_gb300 import INCA_FP64, INCA_MIXED, Context, centercalc
from inca_parallel_gb300 import workloads as W

THRESH = 1e-12
TOL = 1e-10


def listed():
    return [
        # intracule_two_points of a small molecule: the smallest call, all latency
        {"name": "two_points_ch4", "job": "points", "system": "ch4", "npts": 2, "mode": "fp64"},
        # a profile along a line through the molecule, mixed precision
        {"name": "line_ch4", "job": "points", "system": "ch4", "npts": 501, "mode": "mixed"},
        # the reference's radial-integral input: one centre, 50 radial x 110 angular points
        {"name": "integral_ch4", "job": "integral", "system": "ch4", "nrad": 50, "nang": 110},
        # the reference's radial-plot input (s = 0 to 5 by 0.05, 110 angular points) in plain FP64
        {"name": "plot_ch4_fp64", "job": "plot", "system": "ch4", "mode": "fp64", "smax": 5.0, "step": 0.05, "nang": 110},
        # the benchmark's radial plot: s = 0 to 10 by 0.05, 590 angular points
        {"name": "plot_ch4_fine", "job": "plot", "system": "ch4", "mode": "mixed", "smax": 10.0, "step": 0.05,
         "nang": 590},
        # a molecule with d shells, ordinary grid
        {"name": "plot_mol41", "job": "plot", "system": "mol", "natoms": 4, "nprim": 41, "geometry": 11, "mode": "mixed",
         "smax": 10.0, "step": 0.1, "nang": 302},
        # a larger molecule's radial integral on its multicentre grid
        {"name": "integral_mol66", "job": "integral", "system": "mol", "natoms": 6, "nprim": 66, "geometry": 12,
         "nrad": 40, "nang": 110},
        # the largest: 13 million quartets, a production grid
        {"name": "integral_mol100", "job": "integral", "system": "mol", "natoms": 5, "nprim": 100, "geometry": 13,
         "nrad": 50, "nang": 194},
        # cubeintra: the benchmark's 48^3 lattice, and a ragged one around a molecule
        {"name": "cube_ch4_48", "job": "cube", "system": "ch4", "nx": 48, "ny": 48, "nz": 48, "step": 0.15},
        {"name": "cube_mol40", "job": "cube", "system": "mol", "natoms": 5, "nprim": 40, "geometry": 14, "nx": 41,
         "ny": 38, "nz": 35, "step": 0.2},
        # several small molecules in one batch
        {"name": "batch_6", "job": "batch", "nmol": 6, "natoms": 4, "nprim": 30, "geometry": 15, "smax": 10.0, "step": 0.1,
         "nang": 302},
        # a program with its own device memory: caller's records at caller's points, FP64
        {"name": "records_ch4", "job": "records", "system": "ch4", "npts": 1777},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: a job of the list with its sizes drawn from the ranges that users run."""
    job = rng.choice(["points", "integral", "plot", "plot", "cube", "batch", "records", "integral"])
    nang = rng.choice([50, 110, 194, 302, 434, 590])
    geometry = rng.randrange(100, 1 << 20)
    if rng.random() < 0.4:
        system = {"system": "ch4"}
    else:
        system = {"system": "mol", "natoms": rng.randint(2, 6), "nprim": round(_log(rng, 20, 70)), "geometry": geometry}
    if job == "points":
        return {"job": job, **system, "npts": round(_log(rng, 1, 1500)), "mode": rng.choice(["fp64", "mixed"])}
    if job == "integral":
        return {"job": job, **system, "nrad": rng.randint(20, 60), "nang": min(nang, 302)}
    if job == "plot":
        mode = rng.choice(["fp64", "mixed", "mixed"])
        fine = mode == "mixed"
        return {"job": job, **system, "mode": mode, "smax": round(rng.uniform(4.0, 10.0) if fine else 5.0, 2),
                "step": rng.choice([0.05, 0.1] if fine else [0.1, 0.25]), "nang": nang if fine else min(nang, 110)}
    if job == "cube":
        return {"job": job, **system, "nx": rng.randint(12, 48), "ny": rng.randint(12, 48), "nz": rng.randint(12, 48),
                "step": round(rng.uniform(0.1, 0.25), 3)}
    if job == "batch":
        return {"job": job, "nmol": rng.randint(2, 8), "natoms": rng.randint(2, 5), "nprim": round(_log(rng, 18, 40)),
                "geometry": geometry, "smax": 10.0, "step": rng.choice([0.1, 0.2]), "nang": min(nang, 302)}
    return {"job": job, **system, "npts": round(_log(rng, 64, 4096))}


# ---------------------------------------------------------------- inputs

@functools.lru_cache(maxsize=64)
def _molecule(natoms, nprim, geometry):
    b = W.random_molecule(np.random.default_rng(geometry), natoms, nprim, hi=200.0)
    return b, W.overlap(b)


@functools.lru_cache(maxsize=1)
def _ch4():
    b = W.ch4_basis()
    return b, W.overlap(b)


def _system(case):
    if case.get("system") == "ch4":
        return _ch4() + (5,)
    b, S = _molecule(case["natoms"], case["nprim"], case["geometry"])
    return b, S, max(1, min(W.electrons(b) // 2, len(b["alpha"]) // 3))


def _density(S, nocc, seed):
    """1-RDM of nocc random orbitals, orthonormal in the overlap metric."""
    C = np.random.default_rng(seed).normal(size=(len(S), nocc))
    w, U = np.linalg.eigh(C.T @ S @ C)
    C = C @ (U @ np.diag(w ** -0.5) @ U.T)
    return 2.0 * C @ C.T


def _pairs(n):
    i, k = np.triu_indices(n)
    return i.astype(np.int64), k.astype(np.int64)


def _records(D, unique):
    """Closed-shell DM2 records (i <= k, j <= l; unique: pair(ik) <= pair(jl)): 0-based ijkl and values."""
    pi, pk = _pairs(len(D))
    if unique:
        a, b = np.triu_indices(len(pi))
    else:
        a, b = (x.reshape(-1) for x in np.meshgrid(np.arange(len(pi)), np.arange(len(pi)), indexing="ij"))
    i, k, j, l = pi[a], pk[a], pi[b], pk[b]
    v = np.zeros(len(a))
    for p, q, on1 in ((i, k, True), (k, i, i != k)):
        for r, s, on2 in ((j, l, True), (l, j, j != l)):
            v += np.where(on1 & on2, D[p, q] * D[r, s] - 0.5 * D[p, s] * D[r, q], 0.0)
    if unique:
        v = np.where(a != b, 2.0 * v, v)
    return np.stack([i, j, k, l], 1), v


def _batch(case, seed):
    out = []
    for m in range(case["nmol"]):
        b, S, nocc = _system({"natoms": case["natoms"], "nprim": case["nprim"] - 2 * (m % 3), "geometry": case["geometry"] + m})
        out.append((b, _density(S, nocc, seed * 64 + m)))
    return out


def _line(n, seed):
    """n points along a line through the origin."""
    rng = np.random.default_rng(seed + 1)
    d = rng.normal(size=3)
    t = np.linspace(0.0, 5.0, n) if n > 2 else np.array([0.0, 1.0])[:n]
    return np.outer(t, d / np.linalg.norm(d))


def _cloud(n, seed):
    """n points of a caller's own choice around the origin, exponentially thinning."""
    rng = np.random.default_rng(seed + 1)
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1)[:, None] * rng.exponential(1.5, size=(n, 1))


def _radial_grid(ctx, case, basis):
    """CH4: the reference's single centre; molecules: the automatic multicentre grid."""
    full = case["system"] == "ch4"
    cent, Ps, alf = (np.zeros((1, 3)), np.ones(1), np.ones(1)) if full else centercalc(basis["an"], basis["cartes"])
    n = len(Ps)
    ctx.grid_radial([case["nrad"]] * n, [case["nang"]] * n, alf, cent, Ps, nosym=not full)


def _set_up(ctx, st):
    b = st["basis"]
    ctx.set_primitives(b["alpha"], b["tmn"], b["xyz"])
    if st["ijkl"] is not None:
        ctx.set_quartets(st["ijkl"], st["v"])
    else:
        ctx.gen_closed_shell_dm2(st["D"], unique=True)
    return ctx.prepare(THRESH)


def prepare(case, seed):
    if case["job"] == "batch":
        return {"case": case, "ctx": Context(0), "mols": _batch(case, seed)}
    basis, S, nocc = _system(case)
    D = _density(S, nocc, seed)
    st = {"case": case, "ctx": Context(0), "basis": basis, "D": D, "ijkl": None, "v": None}
    if case["system"] == "ch4":  # a .dm2p file's records, in host memory
        ijkl, st["v"] = _records(D, unique=False)
        st["ijkl"] = np.ascontiguousarray(ijkl + 1, dtype=np.int32)
    if case["job"] == "points":
        st["points"] = _line(case["npts"], seed)
    if case["job"] == "records":  # the survivors of the screening, kept on the device by the caller
        _set_up(st["ctx"], st)
        rec = st["ctx"].records()
        st["rec"] = {k: torch.from_numpy(np.ascontiguousarray(x)).cuda() for k, x in rec.items()}
        st["points"] = torch.from_numpy(_cloud(case["npts"], seed)).cuda()
    return st


# ---------------------------------------------------------------- the jobs

def run(state):
    case, ctx = state["case"], state["ctx"]
    job = case["job"]
    mode = INCA_FP64 if case.get("mode") == "fp64" else INCA_MIXED
    if job == "records":
        rec, pts = state["rec"], state["points"]
        out = torch.empty(len(pts), dtype=torch.float64, device="cuda")
        p = [ctypes.c_void_p(rec[k].data_ptr()) for k in ("A", "sqe", "d", "L", "C")]
        st = ctx.lib.inca_eval_records_noalloc(len(rec["A"]), *p, len(pts), ctypes.c_void_p(pts.data_ptr()),
                                               ctypes.c_void_p(out.data_ptr()),
                                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st:
            raise RuntimeError(f"inca_eval_records_noalloc: {st}")
        return {"ivec": out}
    if job == "batch":
        ctx.batch_clear()
        for b, D in state["mols"]:
            ctx.batch_add_closed_shell(b["alpha"], b["tmn"], b["xyz"], D, [0.0], [case["smax"]], [case["step"]],
                                       [case["nang"]], unique=True, nosym=True)
        counts = ctx.batch_prepare(THRESH)
        return {"counts": np.array(counts), "rintra": ctx.batch_eval(mode=INCA_MIXED, tol=TOL)}
    counts = np.array(_set_up(ctx, state))
    nosym = state["ijkl"] is None
    if job == "points":
        ctx.grid_points(state["points"])
        return {"counts": counts, "ivec": ctx.eval(mode=mode, tol=TOL)}
    if job == "cube":
        ctx.grid_cube([0.1, 0.0, -0.1], [case["step"]] * 3, [case["nx"], case["ny"], case["nz"]])
        return {"counts": counts, "ivec": ctx.eval(mode=mode, tol=TOL)}
    if job == "plot":
        ctx.grid_scan([0.0], [case["smax"]], [case["step"]], [case["nang"]], nosym=nosym)
        ctx.eval(mode=mode, tol=TOL, copy=False)
        radi, rintra = ctx.radial_plot()
        return {"counts": counts, "radi": radi, "rintra": rintra}
    _radial_grid(ctx, case, state["basis"])
    ctx.eval(mode=mode, tol=TOL, copy=False)
    total, vee, per_centre, vee_per_centre = ctx.radial_integral()
    return {"counts": counts, "total": total, "vee": vee, "per_centre": per_centre, "vee_per_centre": vee_per_centre}


# ---------------------------------------------------------------- the least work

def _ngrid(case, basis):
    job = case["job"]
    if job in ("points", "records"):
        return case["npts"]
    if job == "cube":
        return case["nx"] * case["ny"] * case["nz"]
    half = 2 if case.get("system") == "ch4" else 1  # r and -r are evaluated once where the DM2 is complete
    if job == "integral":
        nquad = 1 if half == 2 else len(centercalc(basis["an"], basis["cartes"])[1])
        return case["nrad"] * case["nang"] * nquad // half
    return (int(case["smax"] / case["step"]) + 1) * case["nang"] // half


def work(case):
    """Bytes: the DM2 values and indices, the density or the records in, the results out. Operations:
    one Gaussian (3 shifted coordinates, an exponential of about 10 operations) per point and pair of
    shell products (those that overlap by 1e-12 at least), the polynomial of a shell quartet (its
    monomials) on top."""
    if case["job"] == "batch":
        one = [work({"job": "plot", "system": "mol", "natoms": case["natoms"], "nprim": case["nprim"] - 2 * (m % 3),
                     "geometry": case["geometry"] + m, "smax": case["smax"], "step": case["step"], "nang": case["nang"]})
               for m in range(case["nmol"])]
        return {k: sum(w[k] for w in one) for k in ("bytes", "flops")}
    b = _system(case)[0]
    shells = {}
    for a, t, x in zip(b["alpha"], b["tmn"], b["xyz"]):
        shells[(a, tuple(x))] = max(shells.get((a, tuple(x)), 0), int(t.sum()))
    l = np.array(list(shells.values()))
    al, at = np.array([a for a, _ in shells]), np.array([x for _, x in shells])
    i, k = np.triu_indices(len(l))
    near = al[i] * al[k] / (al[i] + al[k]) * ((at[i] - at[k]) ** 2).sum(1) < -math.log(1e-12)
    by = np.bincount((l[i] + l[k])[near], minlength=9).astype(float)
    terms = 0.0
    for p in range(len(by)):
        for q in range(len(by)):
            terms += by[p] * by[q] * (32 + 2 * math.comb(p + q + 3, 3))
    n = len(b["alpha"])
    npair = n * (n + 1) // 2
    full = case["system"] == "ch4"
    if not full:
        terms /= 2
    npts = _ngrid(case, b)
    nin = (npair * npair * 24 if full else n * n * 8) if case["job"] != "records" else npair * npair * (
        1 if full else 0.5) * (5 * 8 + 12 + 6 * 8)
    return {"bytes": float(nin + 8 * npts), "flops": float(terms * npts)}


# ---------------------------------------------------------------- the same values in plain 64 bits

def _hermite_coefs(t, X, P, Q, a, b):
    """Coefficients (ascending powers of w = r + P - Q, one dimension) of
    int (x-Xi)^ti (x-Xk)^tk (x+r-Xj)^tj (x+r-Xl)^tl exp(-a(x-P)^2 - b(x+r-Q)^2) dx * sqrt(zeta) / exp(-ab/zeta w^2)."""
    deg = int(sum(int(x.max()) for x in t))
    nodes, wts = np.polynomial.hermite.hermgauss(deg // 2 + 1)
    z = a + b
    node = torch.tensor(nodes, device=P.device)[None, :] / z.sqrt()[:, None]
    poly = torch.zeros(len(P), len(nodes), deg + 1, dtype=torch.float64, device=P.device)
    poly[:, :, 0] = torch.tensor(wts, device=P.device)
    for m, (tt, xx) in enumerate(zip(t, X)):  # i, k on the first electron, j, l on the second
        c0 = node + ((P if m < 2 else Q) - xx)[:, None]
        c1 = -b / z if m < 2 else a / z
        for p in range(int(tt.max())):
            nxt = c0[:, :, None] * poly
            nxt[:, :, 1:] += c1[:, None, None] * poly[:, :, :-1]
            poly = torch.where((tt > p)[:, None, None], nxt, poly)
    return poly.sum(1)


def _intracule(basis, ijkl, v, pts):
    """Sum over DM2 records of v N_i N_j N_k N_l int g_i g_k (r1) g_j g_l (r1 + r) dr1, at pts (torch, 64 bits)."""
    dev = pts.device
    al = torch.tensor(basis["alpha"], device=dev)
    xyz = torch.tensor(basis["xyz"], device=dev)
    tmn = torch.tensor(basis["tmn"].astype(np.int64), device=dev)
    df = torch.tensor([1.0, 1.0, 3.0, 15.0, 105.0], device=dev, dtype=torch.float64)
    norm = (2 * al / math.pi) ** 0.75 * ((4 * al) ** tmn.sum(1) / df[tmn].prod(1)).sqrt()
    out = torch.zeros(len(pts), dtype=torch.float64, device=dev)
    at = torch.tensor(ijkl, device=dev)
    v = torch.tensor(v, device=dev)
    step = max(1, 50_000_000 // len(pts))
    for o in range(0, len(v), step):
        i, j, k, l = at[o:o + step].unbind(1)
        a, b = al[i] + al[k], al[j] + al[l]
        z = a + b
        P = (al[i, None] * xyz[i] + al[k, None] * xyz[k]) / a[:, None]
        Q = (al[j, None] * xyz[j] + al[l, None] * xyz[l]) / b[:, None]
        K = (al[i] * al[k] / a) * ((xyz[i] - xyz[k]) ** 2).sum(1) + (al[j] * al[l] / b) * ((xyz[j] - xyz[l]) ** 2).sum(1)
        amp = v[o:o + step] * norm[i] * norm[j] * norm[k] * norm[l] / z ** 1.5 * torch.exp(-K)
        term = amp[:, None]
        s2 = torch.zeros(1, dtype=torch.float64, device=dev)
        for d in range(3):
            w = pts[None, :, d] + (P[:, d] - Q[:, d])[:, None]
            c = _hermite_coefs([tmn[x, d] for x in (i, k, j, l)], [xyz[x, d] for x in (i, k, j, l)], P[:, d], Q[:, d], a, b)
            val = c[:, -1:].expand(-1, len(pts))
            for m in range(c.shape[1] - 2, -1, -1):
                val = torch.addcmul(c[:, m:m + 1], val, w)
            term = term * val
            s2 = s2 + w * w
        out += (term * torch.exp(-(a * b / z)[:, None] * s2)).sum(0)
    return out


def _eval_records(rec, pts):
    """The caller's records at the caller's points, in plain torch."""
    out = torch.zeros(len(pts), dtype=torch.float64, device="cuda")
    A, s, d, L, C = (rec[k] for k in ("A", "sqe", "d", "L", "C"))
    step = max(1, 50_000_000 // len(pts))
    for o in range(0, len(A), step):
        sl = slice(o, o + step)
        term, s2 = A[sl, None], 0.0
        for x in range(3):
            u = s[sl, None] * (pts[None, :, x] + d[sl, x:x + 1])
            val = C[sl, x, 0:1].expand(-1, len(pts))
            for m in range(1, int(L[sl, x].max()) + 1):
                val = torch.where((L[sl, x:x + 1] >= m), torch.addcmul(C[sl, x, m:m + 1], val, u), val)
            term = term * val
            s2 = s2 + u * u
        out += (term * torch.exp(-s2)).sum(0)
    return out


def exact(case, seed):
    """The intracule of the same density at the same points by Gauss-Hermite quadrature of its defining
    integral, summed with the grid's weights (read back: points and weights are this job's input). Cases
    of at most 3e10 quartet-points only."""
    job = case["job"]
    if job == "records":
        st = prepare(case, seed)
        return {"ivec": _eval_records(st["rec"], st["points"]).cpu().numpy()}
    if job == "batch":
        return None
    basis, S, nocc = _system(case)
    full = case["system"] == "ch4"
    npair = len(S) * (len(S) + 1) // 2
    if npair * npair * (1.0 if full else 0.5) * _ngrid(case, basis) > 3e10:
        return None
    ijkl, v = _records(_density(S, nocc, seed), unique=not full)
    g, ctx = {}, Context(0)
    if job == "points":
        pts = _line(case["npts"], seed)
    elif job == "cube":
        h = case["step"]
        ax = [c + (np.arange(n) - (n - 1) / 2) * h for c, n in zip((0.1, 0.0, -0.1), (case["nx"], case["ny"], case["nz"]))]
        pts = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    else:
        if job == "plot":
            ctx.grid_scan([0.0], [case["smax"]], [case["step"]], [case["nang"]], nosym=not full)
            g = ctx.grid_copy(cmap=True)
        else:
            _radial_grid(ctx, case, basis)
            g = ctx.grid_copy(vee=True, cmap=True)
        pts = g["r"]
    iv = _intracule(basis, ijkl, v, torch.tensor(pts, device="cuda")).cpu().numpy()
    if job == "plot":
        return {"counts": None, "radi": None, "rintra": np.bincount(g["cmap"] - 1, g["w"] * iv, minlength=ctx.nradi)}
    if job == "integral":
        per, vper = (np.bincount(g["cmap"] - 1, g[k] * iv, minlength=ctx.nquad) for k in ("w", "wvee"))
        return {"counts": None, "total": float(per.sum()), "vee": float(vper.sum()), "per_centre": per,
                "vee_per_centre": vper}
    return {"counts": None, "ivec": iv}
