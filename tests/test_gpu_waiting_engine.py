"""The waiting engine (resident CTAs, a counter per instance; one CTA an SM of
several groups, or an item split over two CTAs) against the persistent engine
with its grid barrier, which a cap on the CTAs per SM selects: the same bits,
step traces and counts, whatever the constraints, the algorithm and the layout."""
import numpy as np
import pytest

import mprgp_gb300 as M

pytestmark = pytest.mark.gpu

SEED = 0x5EED


@pytest.fixture(scope="module")
def context():
    c = M.Context(0)
    yield c
    c.close()


def beam(dims, walls, seed, mode=2, **kw):
    return M.beam(*dims, extra_planes_max=walls, extra_planes_min=walls, plane_mode=mode,
                  v0_sigma=0.2, seed=seed, **kw)


def solve_all(c, cap, qps, kind=M.KIND_PLANES, precision=M.PREC_FP64, algorithm=0, max_it=2000,
              trace=True):
    c.set_tuning(0, cap)
    probs, opts = [], []
    for qp in qps:
        p = M.Problem(c, qp.nv)
        if kind >= M.KIND_DECOUPLED:
            p.set_planes(qp.plane_ptr, qp.planes)
        else:
            x0 = qp.x0.reshape(-1, 3)
            L, U = x0 - 1e-3, x0 + 1.2e-3
            L[:, 1], U[:, 1] = np.maximum(L[:, 1], 0.0), np.maximum(U[:, 1], 5e-3)
            p.set_bounds(np.ascontiguousarray(L.reshape(-1)),
                         np.ascontiguousarray(U.reshape(-1)) if kind == M.KIND_BOX else None)
        p.set_matrix(qp.row_ptr, qp.cols, qp.vals, 3)
        p.set_rhs(qp.b)
        p.set_x(qp.x0)
        p.set_power_cache(False)
        if trace:
            p.set_trace(5000)
        probs.append(p)
        opts.append(M.default_options(tol=1e-8 * np.linalg.norm(qp.b), max_it=max_it, kind=kind,
                                      algorithm=algorithm, project_x0=1, seed=SEED,
                                      precision=precision))
    stats = c.solve_batch(probs, opts)
    c.set_tuning(0, 0)
    out = []
    for p, st in zip(probs, stats):
        out.append((p.get_x(), p.get_face(), p.get_trace() if trace else np.zeros(1),
                    (st.code, st.iterations, st.num_cg, st.num_exp, st.num_prop, st.active,
                     st.phases, st.spmv_fp64, st.spmv_fp32, st.residual)))
        p.close()
    return out


def check(c, qps, **kw):
    for (xa, fa, ta, sa), (xb, fb, tb, sb) in zip(solve_all(c, 3, qps, **kw),
                                                  solve_all(c, 0, qps, **kw)):
        assert sa == sb
        assert np.array_equal(xa, xb) and np.array_equal(fa, fb) and np.array_equal(ta, tb)


# vertices on both sides of: one and two items, the cluster solver's 16 items,
# two CTAs an item (76 items), one item an SM (152), 256 items (the longer sum),
# one and two rounds of four groups (608), and a partial last warp throughout
@pytest.mark.parametrize("dims", [(2, 2, 2), (4, 4, 16), (14, 15, 17), (15, 17, 61), (16, 18, 60),
                                  (24, 24, 70), (30, 30, 72), (40, 41, 98)])
@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_sizes(context, dims, precision):
    check(context, [beam(dims, 2, 7)], precision=precision, max_it=60)


@pytest.mark.parametrize("dims", [(4, 4, 16), (15, 17, 30), (20, 21, 40)])
@pytest.mark.parametrize("kind,algorithm", [
    (M.KIND_DECOUPLED, 0), (M.KIND_PLANES, 0), (M.KIND_PLANES, M.ALG_PLAIN), (M.KIND_BOX, 0),
    (M.KIND_LOWER, 0)])
def test_kinds(context, dims, kind, algorithm):
    check(context, [beam(dims, 0 if kind == M.KIND_DECOUPLED else 2, 8)], kind=kind,
          algorithm=algorithm)


@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_tilted_planes(context, precision):
    """General normals: candidates leave the feasible set, delta^T A delta
    phases with and without rows to work on."""
    check(context, [beam((15, 17, 30), 2, 5, mode=1, active_frac=0.3, max_tilt=0.6)],
          precision=precision, max_it=300)


def test_batches(context):
    small = [beam(d, 2, 20 + i) for i, d in enumerate([(2, 2, 2), (7, 9, 21), (14, 14, 17)])]
    mid = [beam(d, 2, 40 + i) for i, d in enumerate([(15, 17, 30), (16, 16, 64), (20, 20, 60)])]
    check(context, mid, precision=M.PREC_MIXED)
    check(context, small + mid, precision=M.PREC_MIXED)
    check(context, small * 3, precision=M.PREC_FP64)
    check(context, mid * 5, precision=M.PREC_FP64, trace=False)
    check(context, small + mid * 9, precision=M.PREC_MIXED, trace=False)


@pytest.mark.parametrize("dims", [(15, 17, 30), (24, 24, 70)])
@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_resumed_after_short_runs(context, dims, precision):
    """A server whose runs end after 3 phases: any phase may be the first."""
    qp = beam(dims, 2, 9)
    opt = M.default_options(tol=1e-8 * np.linalg.norm(qp.b), max_it=2000, kind=M.KIND_PLANES,
                            project_x0=1, seed=SEED, precision=precision)
    x, face, _, stats = solve_all(context, 3, [qp], precision=precision)[0]
    srv = M.Server(context, quantum_phases=3, power_launches=1003)
    try:
        t = srv.submit(0, qp, opt)
        for _ in range(100000):
            srv.step()
            if srv.poll():
                break
        state, xs, fs, st, _ = srv.result(t)
        assert state == 2 and (st.code, st.iterations, st.phases) == (stats[0], stats[1], stats[6])
        assert np.array_equal(xs, x) and np.array_equal(fs, face)
    finally:
        srv.close()
