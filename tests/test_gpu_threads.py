"""Contexts of one device on several host threads: each prepares and reads back its own system, with its
own basis, threshold and normalisation, and has to get what it gets alone, bit by bit."""
import threading

import numpy as np
import pytest

from test_gpu_merged import system

pytestmark = pytest.mark.gpu

JOBS = (("p", 1e-12, True), ("single", 1e-3, False), ("d", 1e-6, True))


def job(c, thresh, normalize, repeats):
    out = []
    for _ in range(repeats):
        counts = c.prepare(thresh, normalize=normalize)
        rec = c.records()
        out.append([np.array(counts), *c.screening(), *(rec[k] for k in ("A", "sqe", "d", "L", "C"))])
    return out


def test_prepare_and_records_on_three_threads():
    from inca_parallel_gb300 import Context, build
    build.build()
    ctxs = []
    for name, _, _ in JOBS:
        s = system(name)
        c = Context(0)
        c.set_primitives(s["alpha"], s["tmn"], s["xyz"])
        c.set_quartets(s["ijkl"], s["v"])
        ctxs.append(c)
    alone = [job(c, thresh, norm, 1)[0] for c, (_, thresh, norm) in zip(ctxs, JOBS)]
    got = [None] * len(JOBS)
    start = threading.Barrier(len(JOBS))

    def run(k):
        start.wait()
        got[k] = job(ctxs[k], JOBS[k][1], JOBS[k][2], 40)

    threads = [threading.Thread(target=run, args=(k,)) for k in range(len(JOBS))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k, want in enumerate(alone):
        assert got[k] is not None
        for one in got[k]:
            for a, b in zip(one, want):
                np.testing.assert_array_equal(a, b)
    for c in ctxs:
        c.close()
