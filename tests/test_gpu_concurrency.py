"""Solves of several contexts and threads at once: each kernel whose CTAs wait
for each other runs behind the one issued before it, so none waits for SMs the
other holds, and every result is the one the solve gives alone."""
import threading

import numpy as np
import pytest

import mprgp_gb300 as M

pytestmark = pytest.mark.gpu


def test_contexts_in_threads():
    dims = [(4, 4, 16), (14, 14, 17), (16, 18, 60), (24, 24, 70), (7, 9, 21)]
    qps = [M.beam(*d, extra_planes_max=2, extra_planes_min=2, plane_mode=2, v0_sigma=0.2, seed=i)
           for i, d in enumerate(dims)]

    def opt(i, q):
        return M.default_options(tol=1e-8 * np.linalg.norm(q.b), max_it=2000, kind=M.KIND_PLANES,
                                 project_x0=1, precision=i % 2)

    one = M.Context(0)
    alone = [one.solve_bsr(q, opt(i, q), q.x0)[0] for i, q in enumerate(qps)]
    one.close()
    errors = []

    def work(order):
        try:
            c = M.Context(0)
            for _ in range(4):
                for i in order:
                    x, _, st = c.solve_bsr(qps[i], opt(i, qps[i]), qps[i].x0)
                    if st.code != 0 or not np.array_equal(x, alone[i]):
                        errors.append((i, st.code))
            c.close()
        except Exception as e:  # noqa: BLE001
            errors.append(repr(e))

    threads = [threading.Thread(target=work, args=(o,))
               for o in ([0, 1, 2, 3, 4], [3, 2, 1, 0, 4], [4, 2, 3, 1, 0])]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert not errors and not any(t.is_alive() for t in threads)
