"""Synchronous runs beside a server's lanes, of their own and of another
context: the launch loops and the cluster solver, whose results are the bits of
the waiting kernels; the launch counts tell the two apart."""
import numpy as np
import pytest

import mprgp_gb300 as M

pytestmark = pytest.mark.gpu


def body(dims, seed):
    return M.beam(*dims, extra_planes_max=2, extra_planes_min=2, plane_mode=2, v0_sigma=0.2,
                  seed=seed)


def opts(qp, precision):
    return M.default_options(tol=1e-8 * np.linalg.norm(qp.b), max_it=2000, kind=M.KIND_PLANES,
                             project_x0=1, precision=precision)


def solve(ctx, qps, precision):
    """x of each, and the kernels the run launched."""
    probs = [M.load_beam(ctx, q, 3) for q in qps]
    for p in probs:
        p.set_power_cache(False)
    ctx.solve_batch(probs, [opts(q, precision) for q in qps])  # set-up kernels
    for p, q in zip(probs, qps):
        p.set_x(q.x0)
    before = ctx.counters()[0]
    st = ctx.solve_batch(probs, [opts(q, precision) for q in qps])
    launches = ctx.counters()[0] - before
    out = [p.get_x() for p in probs]
    for p in probs:
        p.close()
    assert all(s.code == 0 for s in st)
    return out, launches


@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_small_solves_beside_lanes(precision):
    qps = [body((4, 4, 16), 1), body((5, 4, 14), 2), body((4, 5, 15), 3)]  # 2 items each
    big = body((47, 47, 60), 4)
    own, other = M.Context(0), M.Context(0)
    ref, n = solve(own, qps, precision)
    # the power loop, the other phases (waiting engine or one cluster class), the
    # states in and out
    assert n == 4
    srv = M.Server(own, quantum_phases=64, power_launches=1003, lanes=3)
    for ctx in (own, other):
        # the request's power method is in flight, and stays so until the next step
        ticket = srv.submit(0 if ctx is own else 1, big, opts(big, M.PREC_FP64))
        srv.step()
        out, n = solve(ctx, qps, precision)
        if ctx is own:
            assert n == 3  # one cluster class, and no power loop that waits
        for a, b in zip(ref, out):
            assert np.array_equal(a, b)
        for _ in range(100000):
            if srv.result(ticket)[0] == 2:
                break
            srv.step()
    srv.close()
    out, n = solve(other, qps, precision)
    assert n == 4 and all(np.array_equal(a, b) for a, b in zip(ref, out))
    other.close()
    own.close()


@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_launch_loop_tuning_keeps_the_cluster_solver(precision):
    qps = [body((4, 4, 16), 1), body((5, 4, 14), 2)]
    ctx = M.Context(0)
    ref, n = solve(ctx, qps, precision)
    assert n == 4
    for bits in (2, 4, 64):
        ctx.set_tuning(bits, 0)
        out, n = solve(ctx, qps, precision)
        assert n == 3  # one cluster class, the states in and out
        assert all(np.array_equal(a, b) for a, b in zip(ref, out))
    ctx.close()
