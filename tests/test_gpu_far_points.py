"""Points so far out that a record's whole polynomial overflows, while each of its one-dimensional factors does
not: the term is zero, as in the reference's product with the exponential first."""
import ctypes
import itertools

import numpy as np
import pytest

import oracle_lib as O
from test_gpu_merged import ctx  # noqa: F401

pytestmark = pytest.mark.gpu
FAR = np.array([[1e105, 1e105, 1e105], [-1e105, 1e106, -2e105], [0.3, -0.2, 0.1]])


def test_merged_records(ctx):  # noqa: F811
    # quartets x y z s of p shells in every order: degree one in each dimension, three together, merged
    prims = [(0.9, t, (0.0, 0.0, 0.0)) for t in ((1, 0, 0), (0, 1, 0), (0, 0, 1))] + [(0.6, (0, 0, 0), (0.3, -0.8, 1.1))]
    s = {"alpha": np.array([p[0] for p in prims]), "tmn": np.array([p[1] for p in prims], dtype=np.int32),
         "xyz": np.array([p[2] for p in prims]),
         "ijkl": np.array(list(itertools.permutations((1, 2, 3))), dtype=np.int32)}
    s["ijkl"] = np.concatenate([s["ijkl"], np.full((6, 1), 4, dtype=np.int32)], 1)
    s["v"] = np.arange(1.0, 7.0)
    ctx.set_primitives(s["alpha"], s["tmn"], s["xyz"])
    ctx.set_quartets(s["ijkl"], s["v"])
    ctx.prepare(1e-12)
    want = O.intracule(s, 1e-12, FAR)[0]
    assert (want[:2] == 0.0).all()
    for n in (1, 2100):  # the few-point form and the general one
        ctx.grid_points(np.tile(FAR, (n, 1)))
        for mode in (0, 2):
            got = ctx.eval(mode=mode).reshape(n, 3)
            np.testing.assert_allclose(got, np.tile(want, (n, 1)), rtol=1e-12)


def test_callers_records(ctx):  # noqa: F811
    import torch
    n = 40
    rng = np.random.default_rng(1)
    rec = [rng.normal(size=n), np.full(n, 0.9), np.zeros((n, 3)), np.full((n, 3), 16, dtype=np.int32),
           rng.normal(size=(n, 3, 17))]
    dev = [torch.from_numpy(x).cuda() for x in rec]
    pts = torch.tensor([[1e8, 2e8, -1e8], [0.1, 0.2, 0.3]], dtype=torch.float64, device="cuda")
    out = torch.full((2,), float("nan"), dtype=torch.float64, device="cuda")
    assert ctx.lib.inca_eval_records_noalloc(
        n, *(ctypes.c_void_p(x.data_ptr()) for x in dev), 2, ctypes.c_void_p(pts.data_ptr()),
        ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    got = out.cpu().numpy()
    assert got[0] == 0.0 and np.isfinite(got[1])
