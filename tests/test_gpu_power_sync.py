"""The power loops whose CTAs wait for each other -- matrix slices in shared
memory with one or several CTAs an item, the persistent loop with one or two
items a CTA, one cluster an instance -- against the loop of one launch a phase:
the same bits, from a cold start, a stored vector and a resumed run, whether
the loop stops early or at its limit."""
import numpy as np
import pytest

import mprgp_gb300 as M

pytestmark = pytest.mark.gpu

SEED = 0x5EED
LAUNCH_LOOP = 64  # tuning bit: a launch per phase; small instances in the cluster solver


@pytest.fixture(scope="module")
def context():
    c = M.Context(0)
    yield c
    c.close()


def corner(dims, seed):
    return M.beam(*dims, extra_planes_max=2, extra_planes_min=2, plane_mode=2, v0_sigma=0.2,
                  seed=seed)


def wide(nv, blocks, seed):
    """A diagonally dominant problem with `blocks` blocks a row, some of them
    longer: rows whose slices need several CTAs an item."""
    qp = M.beam(1, 1, nv // 4 - 1, seed=seed)
    rng = np.random.default_rng(seed)
    n = qp.nv
    pairs = {(i, i) for i in range(n)}
    for i in range(n):
        k = blocks // 2 + (3 if i % 50 == 0 else 0)
        for j in rng.choice(n, size=min(k, n), replace=False):
            pairs |= {(i, int(j)), (int(j), i)}
    rows, cols = np.array(sorted(pairs)).T
    val = {}
    blocks_v = np.zeros((len(rows), 9))
    for e, (i, j) in enumerate(zip(rows, cols)):
        if i == j:
            blocks_v[e] = (4.0 * np.eye(3)).reshape(-1)
        else:
            key = (min(i, j), max(i, j))
            if key not in val:
                val[key] = rng.uniform(-0.01, 0.01, (3, 3))
            blocks_v[e] = (val[key] if i <= j else val[key].T).reshape(-1)
    qp.row_ptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    qp.cols, qp.vals = cols.astype(np.int32), blocks_v
    return qp


def solve_all(c, bits, qps, precision, rel_tol=1e-8, warm=False):
    c.set_tuning(bits, 0)
    probs, opts = [], []
    for qp in qps:
        probs.append(M.load_beam(c, qp, 3))
        probs[-1].set_power_cache(False)
        opts.append(M.default_options(tol=rel_tol * np.linalg.norm(qp.b), max_it=2000,
                                      kind=M.KIND_PLANES, project_x0=1, seed=SEED,
                                      precision=precision, use_ev=int(warm)))
        if warm:
            probs[-1].set_ev(np.cos(np.arange(qp.n) * 0.7) * 0.01)
    stats = c.solve_batch(probs, opts)
    out = []
    for p, st in zip(probs, stats):
        ev = p.get_ev()
        out.append((p.get_x(), p.get_face(), np.zeros(1) if ev is None else ev,
                    (st.code, st.iterations, st.power_iters, st.power_passes, st.phases,
                     st.spec_rad, st.alpha_bar, st.residual)))
        p.close()
    c.set_tuning(0, 0)
    return out


def check(c, qps, precision, **kw):
    ref = solve_all(c, LAUNCH_LOOP, qps, precision, **kw)
    got = solve_all(c, 0, qps, precision, **kw)
    for (xa, fa, ea, sa), (xb, fb, eb, sb) in zip(ref, got):
        assert sa == sb
        assert np.array_equal(xa, xb) and np.array_equal(fa, fb) and np.array_equal(ea, eb)


# 27 vertices (a partial warp), 256 (one full item), 257-ish, several items,
# and sizes on both sides of each form's capacity
SIZES = [(2, 2, 2), (3, 3, 15), (4, 4, 16), (7, 9, 21), (15, 15, 17), (15, 17, 61), (20, 20, 60),
         (24, 24, 70)]


@pytest.mark.parametrize("dims", SIZES)
@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_one_instance(context, dims, precision):
    check(context, [corner(dims, 5)], precision)


@pytest.mark.parametrize("dims", [(4, 4, 16), (15, 17, 30), (24, 24, 70)])
@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_early_stop_and_stored_start(context, dims, precision):
    """A tolerance the power method meets in a few iterations (its vector is
    then stored), and a start from a stored vector."""
    qp = corner(dims, 6)
    check(context, [qp], precision, rel_tol=0.02)
    check(context, [qp], precision, warm=True)
    check(context, [qp], precision, warm=True, rel_tol=0.02)


@pytest.mark.parametrize("blocks", [24, 44, 90])
@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_wide_rows(context, blocks, precision):
    check(context, [wide(400, blocks, 3)], precision)


@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_batches(context, precision):
    """Small and large instances together: all in one launch where they fit,
    else one cluster an instance beside the persistent loop (two items a CTA
    in the last batch)."""
    small = [corner(d, 20 + i) for i, d in
             enumerate([(2, 2, 2), (3, 3, 15), (4, 5, 11), (7, 9, 21), (9, 9, 30), (14, 14, 17)])]
    check(context, small, precision)
    check(context, small * 8, precision)
    mid = [corner(d, 40 + i) for i, d in enumerate([(15, 17, 30), (16, 16, 64)])]
    check(context, small * 3 + mid * 2, precision)
    check(context, small + mid * 8, precision)


def test_precisions_mixed_in_one_run(context):
    qps = [corner((4, 4, 16), 3), corner((15, 17, 30), 4), corner((5, 5, 9), 5)]
    ref = [solve_all(context, LAUNCH_LOOP, [q], p)[0] for q, p in
           zip(qps, (M.PREC_FP64, M.PREC_MIXED, M.PREC_MIXED))]
    probs, opts = [], []
    for q, p in zip(qps, (M.PREC_FP64, M.PREC_MIXED, M.PREC_MIXED)):
        probs.append(M.load_beam(context, q, 3))
        probs[-1].set_power_cache(False)
        opts.append(M.default_options(tol=1e-8 * np.linalg.norm(q.b), max_it=2000,
                                      kind=M.KIND_PLANES, project_x0=1, seed=SEED, precision=p))
    context.solve_batch(probs, opts)
    for p, (x, face, _, _) in zip(probs, ref):
        assert np.array_equal(p.get_x(), x) and np.array_equal(p.get_face(), face)
        p.close()


@pytest.mark.parametrize("lanes", [0, 2, 3])
@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_served_in_short_power_runs(context, lanes, precision):
    """A server whose runs end after 5 power phases: the loops resume."""
    qps = [corner((4, 4, 16), 3), corner((15, 17, 30), 4)]
    opts = [M.default_options(tol=0.02 * np.linalg.norm(q.b), max_it=2000, kind=M.KIND_PLANES,
                              project_x0=1, seed=SEED, precision=precision) for q in qps]
    ref = [solve_all(context, LAUNCH_LOOP, [q], precision, rel_tol=0.02)[0] for q in qps]
    srv = M.Server(context, quantum_phases=16, power_launches=5, lanes=lanes)
    try:
        tickets = [srv.submit(i, q, o) for i, (q, o) in enumerate(zip(qps, opts))]
        todo = set(tickets)
        for _ in range(100000):
            srv.step()
            todo -= set(srv.poll())
            if not todo:
                break
        assert not todo
        for t, (x, face, _, stats) in zip(tickets, ref):
            state, xs, fs, st, _ = srv.result(t)
            assert state == 2 and st.code == stats[0]
            assert np.array_equal(xs, x) and np.array_equal(fs, face)
            assert (st.spec_rad, st.power_iters) == (stats[5], stats[2])
    finally:
        srv.close()
