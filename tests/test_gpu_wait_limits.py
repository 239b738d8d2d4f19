"""Waits that run out, form by form: a limit far shorter than any phase ends
the launch with MPRGP_TIMEOUT, for the instances of that launch alone, and the
context then solves with the bits of a context that never gave up."""
import ctypes as C

import numpy as np
import pytest

import mprgp_gb300 as M

pytestmark = pytest.mark.gpu


def body(dims, seed=1):
    return M.beam(*dims, extra_planes_max=2, extra_planes_min=2, plane_mode=2, v0_sigma=0.2,
                  seed=seed)


def opts(qp, precision, **kw):
    return M.default_options(tol=1e-8 * np.linalg.norm(qp.b), max_it=2000, kind=M.KIND_PLANES,
                             project_x0=1, precision=precision, **kw)


def solve(ctx, probs, qps, precisions, **kw):
    """(rc, codes, x) of one run over the problems."""
    n = len(probs)
    for p, q in zip(probs, qps):
        p.set_x(q.x0)
    handles = (C.c_void_p * n)(*[p.h for p in probs])
    o = (M.Options * n)(*[opts(q, pr, **kw) for q, pr in zip(qps, precisions)])
    st = (M.Stats * n)()
    rc = M.lib().mprgp_solve_batch(ctx.h, n, handles, o, st)
    return rc, [s.code for s in st], [p.get_x() for p in probs]


F, X = M.PREC_FP64, M.PREC_MIXED
FORMS = {
    # name: (bodies, precisions, instances past their power method, CTAs an SM)
    "power sync, whole items": ([(9, 9, 16)], [X], [], 0),
    "power sync, 8 CTAs an item": ([(4, 4, 16)], [F], [], 0),
    "power sync, 4 CTAs an item": ([(12, 12, 30)], [F], [], 0),
    "power sync, 2 CTAs an item": ([(23, 23, 30)], [F], [], 0),
    "persistent power loop": ([(29, 29, 55)], [X], [], 0),
    "waiting engine, whole items": ([(29, 29, 55)], [X], [0], 0),
    "waiting engine, 8 CTAs an item": ([(4, 4, 16)], [F], [0], 0),
    "waiting engine, 4 CTAs an item": ([(12, 12, 30)], [F], [0], 0),
    "waiting engine, 2 CTAs an item": ([(23, 23, 30)], [F], [0], 0),
    "engine with a grid barrier": ([(12, 12, 30)], [F], [0], 2),
    "clusters beside the persistent loop": ([(29, 29, 55), (9, 9, 16), (4, 4, 16)], [X, X, X], [], 0),
}


@pytest.mark.parametrize("form", FORMS)
def test_limit_then_normal_solve(form):
    dims, precisions, past, ctas = FORMS[form]
    qps = [body(d, i + 1) for i, d in enumerate(dims)]
    ctx = M.Context(0)
    probs = [M.load_beam(ctx, q, 3) for q in qps]
    rc, codes, ref = solve(ctx, probs, qps, precisions)
    assert rc == 0 and codes == [0] * len(qps)
    ctx.set_tuning(0, ctas)
    for i, p in enumerate(probs):
        p.set_power_cache(i in past)
    if past:  # the cache starts empty again with the matrix: fill it
        rc, codes, x = solve(ctx, probs, qps, precisions)
        assert rc == 0 and all(np.array_equal(a, b) for a, b in zip(ref, x))
    for _ in range(2):
        rc, codes, _ = solve(ctx, probs, qps, precisions, wait_limit_s=1e-9)
        assert rc == M.TIMEOUT and codes[0] == M.TIMEOUT
        rc, codes, x = solve(ctx, probs, qps, precisions)
        assert rc == 0 and codes == [0] * len(qps)
        for a, b in zip(ref, x):
            assert np.array_equal(a, b)
    for p in probs:
        p.close()
    ctx.close()


@pytest.mark.parametrize("precision", [F, X])
def test_small_instance_keeps_its_result(precision):
    """Only the large instance's waits run out; the small one, past its power
    method, has no launch that can give up."""
    qps = [body((9, 9, 16)), body((29, 29, 55), 2)]
    ctx = M.Context(0)
    probs = [M.load_beam(ctx, q, 3) for q in qps]
    rc, codes, ref = solve(ctx, probs, qps, [precision] * 2)
    assert rc == 0 and codes == [0, 0]
    probs[1].set_power_cache(False)
    rc, codes, x = solve(ctx, probs, qps, [precision] * 2, wait_limit_s=1e-9)
    assert rc == M.TIMEOUT
    assert codes == [0, M.TIMEOUT]
    assert np.array_equal(x[0], ref[0])
    rc, codes, x = solve(ctx, probs, qps, [precision] * 2)
    assert rc == 0 and all(np.array_equal(a, b) for a, b in zip(ref, x))
    for p in probs:
        p.close()
    ctx.close()
