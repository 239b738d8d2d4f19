"""Many contexts of one process: runs that wait for their peers are in flight
together where they fit the device, and the others take the launch loops or the
cluster solver instead of standing in a row.  Every result has the bits of the
solve alone."""
import threading
import time

import numpy as np
import pytest

import mprgp_gb300 as M

pytestmark = pytest.mark.gpu

BODIES = {  # contexts, dims, precision, whether several fit together
    "425 vertices, FP64": (8, (4, 4, 16), M.PREC_FP64, True),
    "1,700 vertices, mixed": (8, (9, 9, 16), M.PREC_MIXED, True),
    "6,720 vertices, FP64": (4, (13, 15, 29), M.PREC_FP64, False),
    "17,856 vertices, mixed": (4, (23, 23, 30), M.PREC_MIXED, True),
}


@pytest.mark.parametrize("name", BODIES)
def test_contexts_together(name):
    n, dims, precision, fit = BODIES[name]
    qp = M.beam(*dims, extra_planes_max=2, extra_planes_min=2, plane_mode=2, v0_sigma=0.2, seed=3)
    o = M.default_options(tol=1e-8 * np.linalg.norm(qp.b), max_it=2000, kind=M.KIND_PLANES,
                          project_x0=1, precision=precision)
    ctxs = [M.Context(0) for _ in range(n)]
    probs = [M.load_beam(c, qp, 3) for c in ctxs]
    for p in probs:
        p.set_power_cache(False)

    def one(p):
        p.set_x(qp.x0)
        p.ctx.sync()
        t = time.perf_counter()
        assert p.solve(o).code == 0
        return time.perf_counter() - t

    alone = [one(probs[0]) for _ in range(4)]
    ref = probs[0].get_x()
    assert [one(p) > 0 for p in probs]
    together, bad = [], []
    for _ in range(5):
        gate = threading.Barrier(n)

        def work(p):
            p.set_x(qp.x0)
            p.ctx.sync()
            gate.wait()
            try:
                if p.solve(o).code != 0 or not np.array_equal(p.get_x(), ref):
                    bad.append("result")
            except M.MPRGPError as e:
                bad.append(repr(e))

        threads = [threading.Thread(target=work, args=(p,)) for p in probs]
        for t in threads:
            t.start()
        t0 = time.perf_counter()
        for t in threads:
            t.join(60)
        together.append(time.perf_counter() - t0)
    for p in probs:
        p.close()
    for c in ctxs:
        c.close()
    assert not bad
    if fit:  # in a row they would take n times one solve
        assert np.median(together) < 0.9 * n * np.median(alone), (together, alone)
