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


def test_solves_beside_a_server_of_another_context():
    """One thread serves a burst, two others solve bodies of both sizes meanwhile:
    every result has the bits of the solve alone."""
    def opts(q, precision):
        return M.default_options(tol=1e-8 * np.linalg.norm(q.b), max_it=2000, kind=M.KIND_PLANES,
                                 project_x0=1, precision=precision)

    def body(dims, seed):
        return M.beam(*dims, extra_planes_max=2, extra_planes_min=2, plane_mode=2, v0_sigma=0.2,
                      seed=seed)

    burst = [body(d, 20 + i) for i, d in enumerate([(4, 4, 9), (15, 17, 30), (6, 9, 14),
                                                    (23, 23, 30), (5, 5, 5), (12, 12, 30)] * 3)]
    mine = [(body((9, 9, 16), 1), M.PREC_MIXED), (body((23, 23, 30), 2), M.PREC_MIXED),
            (body((4, 4, 16), 3), M.PREC_FP64), (body((13, 15, 29), 4), M.PREC_FP64)]
    one = M.Context(0)
    ref = [one.solve_bsr(q, opts(q, pr), q.x0)[0] for q, pr in mine]
    served_ref = [one.solve_bsr(q, opts(q, M.PREC_MIXED), q.x0)[0] for q in burst]
    one.close()
    errors, done = [], threading.Event()

    def serve():
        try:
            c = M.Context(0)
            srv = M.Server(c, quantum_phases=128, power_launches=512, lanes=3)
            for _ in range(2):
                left = {srv.submit(i, q, opts(q, M.PREC_MIXED)): i for i, q in enumerate(burst)}
                for _ in range(1000000):
                    if not left:
                        break
                    srv.step()
                    for t in srv.poll():
                        state, x, face, st, _ = srv.result(t)
                        if st.code != 0 or not np.array_equal(x, served_ref[left.pop(t)]):
                            errors.append("served")
                if left:
                    errors.append("not served")
            srv.close()
            c.close()
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))
        finally:
            done.set()

    def solves(order):
        try:
            c = M.Context(0)
            while not done.is_set():
                for i in order:
                    q, pr = mine[i]
                    x, _, st = c.solve_bsr(q, opts(q, pr), q.x0)
                    if st.code != 0 or not np.array_equal(x, ref[i]):
                        errors.append(i)
            c.close()
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    threads = [threading.Thread(target=serve)] + [threading.Thread(target=solves, args=(o,))
                                                  for o in ([0, 1, 2, 3], [3, 1, 2, 0])]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors and not any(t.is_alive() for t in threads)
