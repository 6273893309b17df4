"""inca_eval_records_noalloc over its forms: one point to two tiles and a point more, lists below and above
the work at which the records are sorted (3.4e7 records x points), and one of more than a sort block.

Reference: the record formula in plain torch, 64 bits. Tolerance: a term is rounded (10 + 2 L + 3 y) times
on either side (y its exponent, L the sum of its degrees, P the polynomials of absolute values), and a sum
of n terms n times, 2^-53 each: 2 x 2^-53 sum |A| e^-y P (n + 10 + 2 L + 3 y).
"""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

COEF, BLOCK = 17, 1 << 19


def reference(rec, r, torch):
    A, s, d, L, C = (torch.from_numpy(rec[k]).cuda() for k in ("A", "sqe", "d", "L", "C"))
    out, tol = (torch.zeros(len(r), dtype=torch.float64, device="cuda") for _ in range(2))
    n = len(A)
    for g in range(0, n, 1 << 16):
        part = slice(g, min(n, g + (1 << 16)))
        for i, x in enumerate(torch.from_numpy(r).cuda()):
            u = s[part, None] * (x + d[part])
            v, a = C[part, :, 0], C[part, :, 0].abs()
            for m in range(1, int(L.max()) + 1):
                on = m <= L[part]
                v = torch.where(on, v * u + C[part, :, m], v)
                a = torch.where(on, a * u.abs() + C[part, :, m].abs(), a)
            y = (u * u).sum(1)
            e = A[part] * torch.exp(-y)
            out[i] += (e * v.prod(1)).sum()
            tol[i] += (e.abs() * a.prod(1) * (n + 10 + 2 * L[part].sum(1) + 3 * y)).sum()
    return out.cpu().numpy(), 2 * 2.0 ** -53 * tol.cpu().numpy()


@pytest.mark.parametrize("nrec,npts", [(1, 1), (31, 33), (5000, 128), (5000, 129), (5000, 257), (270000, 128),
                                       (140000, 257), (BLOCK + 5, 66)])
def test_records_against_torch(nrec, npts):
    import torch
    from inca_parallel_gb300 import _lib, build
    build.build()
    lib = _lib.load()
    rng = np.random.default_rng(nrec + npts)
    which = rng.integers(0, max(1, nrec // 40), size=nrec)  # records share their Gaussians, in no order
    m = which.max() + 1
    L = rng.integers(0, 3, size=(nrec, 3)).astype(np.int32)
    L[rng.random(nrec) < 0.001] = (16, 0, 5)
    rec = {"A": rng.normal(size=nrec), "sqe": rng.uniform(0.3, 3.0, size=m)[which],
           "d": np.ascontiguousarray(rng.normal(size=(m, 3))[which]), "L": L,
           "C": 0.5 * rng.normal(size=(nrec, 3, COEF))}
    r = rng.normal(size=(npts, 3))
    want, tol = reference(rec, r[:: max(1, npts // 16)], torch)
    dev = {k: torch.from_numpy(np.ascontiguousarray(rec[k])).cuda() for k in rec}
    pts = torch.from_numpy(r).cuda()
    got = []
    for _ in range(2):
        out = torch.full((npts,), float("nan"), dtype=torch.float64, device="cuda")
        st = lib.inca_eval_records_noalloc(nrec, *(ctypes.c_void_p(dev[k].data_ptr()) for k in ("A", "sqe", "d", "L", "C")),
                                           npts, ctypes.c_void_p(pts.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert st == 0
        got.append(out.cpu().numpy())
    np.testing.assert_array_equal(got[0], got[1])
    assert (np.abs(got[0][:: max(1, npts // 16)] - want) <= tol).all()
