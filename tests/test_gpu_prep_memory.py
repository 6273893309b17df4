"""Device memory that inca_prepare holds, on shells with one component each (few quartets a group, high powers).

Per quartet: 56 bytes of sorting, 112 of groups, 20 of record keys, 17 of flags and screening values; a record
of its own, FP64 and FP32 (degrees up to 16 in each dimension: 57 doubles and 116 floats at most, 920 bytes), and
the numbers of a merged one, which has no more coefficients than the quartets' products cost (82 at most: 84
doubles). Under 2 000 together, and 1.3 GB for the polynomials of a slab.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_memory_of_sparse_shells():
    import torch
    from inca_parallel_gb300 import Context, build
    build.build()
    n = 55
    rng = np.random.default_rng(2)
    tmn = np.tile([[4, 0, 0], [0, 3, 1], [2, 1, 0], [1, 1, 1], [0, 0, 0]], (n // 5, 1)).astype(np.int32)
    D = rng.normal(size=(n, n))
    with Context(0) as c:
        c.set_primitives(np.linspace(0.3, 1.2, n), tmn, 0.5 * rng.normal(size=(n, 3)))
        q = c.gen_closed_shell_dm2(D + D.T, unique=True)
        before = torch.cuda.mem_get_info()[0]
        c.prepare(1e-12)
        assert before - torch.cuda.mem_get_info()[0] <= 2000 * q + 1.3e9


def test_scratch_above_4_gib_is_given_back():
    """s shells, every quartet a group of its own: 530 bytes of scratch a quartet, 5.5 GB for this list. Records,
    flags and screening values, 165 bytes a quartet, stay."""
    import torch
    from inca_parallel_gb300 import Context, build
    build.build()
    n = 95
    rng = np.random.default_rng(3)
    D = rng.normal(size=(n, n))
    with Context(0) as c:
        c.set_primitives(np.linspace(0.3, 1.2, n), np.zeros((n, 3), dtype=np.int32), 0.5 * rng.normal(size=(n, 3)))
        q = c.gen_closed_shell_dm2(D + D.T, unique=True)
        before = torch.cuda.mem_get_info()[0]
        counts = c.prepare(1e-12)
        assert counts[2] > 0.99 * q
        assert before - torch.cuda.mem_get_info()[0] <= 200 * q + (1 << 32)
        assert c.prepare(1e-12) == counts
