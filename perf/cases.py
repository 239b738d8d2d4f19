"""The solver's measured cases: what a contact simulation asks of the library.

Every case is a seeded implicit-Euler FEM beam (a x b x c cubes, six
tetrahedra each; the generator of the tests and the benchmark) taken through
the public Python binding.  The beams keep their material, timestep and
contact depth; a seed sets the velocities (and with them b), the sizes set
everything else.

  solve     one cold QP solve of a resident problem: set x, run the power
            method and MPRGP, read x and the active set back
  bounds    the one-call solve of host arrays (matrix upload included) with
            box bounds and plain MPRGP
  step      one timestep of a running simulation on the device: b from the
            state, contact planes from the positions, warm-started solve
  batch     many uneven problems in one call
  serve     a burst of requests, some of them follow-up timesteps, through
            the continuous-batching server
  product   the sparse matrix-vector product alone
  assemble  A and b from the tetrahedra into a problem, and the residual's
            product with the new A
  ica       the comparison contact solver

The power method's result is reused between solves of one matrix only where a
simulation reuses it (step); the other solves are cold on every pass.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import mprgp_gb300 as M

REL_TOL = 1e-8      # the solver's stopping test: ||g_P|| <= 1e-8 ||b||
POWER_SEED = 0x5EED
DT, GRAVITY = 0.01, (0.0, -9.8, 0.0)
# floor and two walls of the timestep loop, and its proximity distance
STEP_PLANES = np.array([[0.0, 1.0, 0.0, 0.0], [1.0, 0.0, 0.0, -0.01], [0.0, 0.0, 1.0, -0.01]])
STEP_DELTA = 0.025
SOFT, STIFF = (1e5, 0.45), (1e6, 0.49)
_CTX = {}


def listed():
    return [
        # the smallest call: the 425-vertex beam on a floor, full precision;
        # a thousand dependent phases of two work items, all latency
        {"name": "solve_425_fp64", "what": "solve", "a": 4, "b": 4, "c": 16, "walls": 0,
         "kind": "decoupled", "mixed": False},
        # a ragged small body in a corner (up to three planes a vertex), mixed
        {"name": "solve_1760_mixed", "what": "solve", "a": 7, "b": 9, "c": 21, "walls": 2,
         "kind": "planes", "mixed": True},
        # a medium body in full precision, too large for one cluster
        {"name": "solve_17856_fp64", "what": "solve", "a": 15, "b": 17, "c": 61, "walls": 1,
         "kind": "planes", "mixed": False},
        # one large body, mixed: its FP32 matrix just fits L2
        {"name": "solve_140481_mixed", "what": "solve", "a": 32, "b": 32, "c": 128, "walls": 2,
         "kind": "planes", "mixed": True},
        # the call the reference's users make: host arrays in, solution out,
        # here with box bounds and the plain algorithm
        {"name": "bounds_6720_fp64", "what": "bounds", "a": 13, "b": 14, "c": 31},
        # a frame of the largest, stiff, nearly incompressible body
        {"name": "step_348145_mixed", "what": "step", "a": 48, "b": 48, "c": 144, "mixed": True},
        # many uneven bodies at once
        {"name": "batch_48_mixed", "what": "batch", "count": 48, "hi": 24, "hi_c": 48,
         "mix": 1, "mixed": True},
        # a burst of requests from several clients, three in ten follow-ups
        {"name": "serve_48_mixed", "what": "serve", "count": 48, "hi": 32, "hi_c": 64,
         "mix": 2, "mixed": True},
        # the product alone, the largest matrix (streams from memory) and an
        # odd-sized one in single precision
        {"name": "product_348145_fp64", "what": "product", "a": 48, "b": 48, "c": 144,
         "mixed": False},
        {"name": "product_71808_fp32", "what": "product", "a": 33, "b": 31, "c": 65,
         "mixed": True},
        # a change of material or mesh: A and b anew, two million tetrahedra
        {"name": "assemble_348145", "what": "assemble", "a": 48, "b": 48, "c": 144, "mixed": True},
        # the comparison solver on a small body
        {"name": "ica_1377", "what": "ica", "a": 8, "b": 8, "c": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["solve", "solve", "solve", "bounds", "step", "batch", "serve", "product",
                       "product", "assemble", "ica"])
    mixed = rng.random() < 0.5
    if what in ("batch", "serve"):
        hi = _log_int(rng, 8, 24 if what == "batch" else 32)
        return {"what": what, "count": _log_int(rng, 4, 48), "hi": hi, "hi_c": 2 * hi,
                "mix": rng.randrange(1 << 20), "mixed": mixed}
    # vertices spread over the logarithm of the range, and a ragged shape
    top = {"solve": 140000, "bounds": 20000, "step": 340000, "product": 340000,
           "assemble": 340000, "ica": 2700}[what]
    if what == "step" and not mixed:
        top //= 3  # a frame in full precision costs about twice as much
    nv = math.exp(rng.uniform(math.log(200), math.log(top)))
    long = rng.uniform(1.0, 4.0)
    flat = rng.uniform(0.7, 1.4)
    side = max(2.0, (nv / long) ** (1.0 / 3.0) - 1.0)
    case = {"what": what, "a": max(2, round(side)), "b": max(2, round(side * flat)),
            "c": max(2, round(side * long / flat))}
    if what == "solve":
        case.update(walls=rng.randrange(3), kind=rng.choice(["planes", "decoupled"]), mixed=mixed)
    elif what in ("step", "product", "assemble"):
        case["mixed"] = mixed
    return case


# ------------------------------------------------------------------ inputs --
def _context():
    if "ctx" not in _CTX:
        _CTX["ctx"] = M.Context(0)
    return _CTX["ctx"]


def _beam(case, seed, walls, sigma=0.2, **kw):
    return M.beam(case["a"], case["b"], case["c"], extra_planes_min=walls,
                  extra_planes_max=walls, plane_mode=2, v0_sigma=sigma, seed=seed + 1, **kw)


def _planes_of(case):
    return 0 if case.get("kind") == "decoupled" else case.get("walls", 0)


def _kind(case):
    return M.KIND_DECOUPLED if case.get("kind") == "decoupled" else M.KIND_PLANES


def _options(case, b, **kw):
    prec = M.PREC_MIXED if case.get("mixed") else M.PREC_FP64
    args = dict(tol=REL_TOL * float(np.linalg.norm(b)), max_it=20000, kind=_kind(case),
                project_x0=1, seed=POWER_SEED, precision=prec)
    args.update(kw)
    return M.default_options(**args)


def _bounds(qp):
    """Each coordinate within a millimetre of its start, and above the floor."""
    x0 = qp.x0.reshape(-1, 3)
    L, U = x0 - 1e-3, x0 + 1.2e-3
    L[:, 1] = np.maximum(L[:, 1], 0.0)
    U[:, 1] = np.maximum(U[:, 1], 5e-3)
    return np.ascontiguousarray(L.reshape(-1)), np.ascontiguousarray(U.reshape(-1))


def _burst(case, seed):
    """(dims, walls, seed, follow-ups) of each scene of a batch or a burst:
    the case's `mix` sets the bodies, the seed their velocities."""
    rng, push = np.random.default_rng(case["mix"]), np.random.default_rng(seed)
    scenes, left = [], case["count"]
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    while left > 0:
        dims = (log(4, case["hi"]), log(4, case["hi"]), log(4, case["hi_c"]))
        more = int(rng.random() < 0.43) if case["what"] == "serve" else 0
        more = min(more, left - 1)
        scenes.append((dims, int(rng.integers(0, 3)), int(push.integers(1, 2**31)), more))
        left -= 1 + more
    return scenes


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    ctx = _context()
    what = case["what"]
    state = {"what": what, "case": case}
    if what == "solve":
        qp = _beam(case, seed, _planes_of(case))
        prob = M.load_beam(ctx, qp, 3 if case["mixed"] else 1)
        prob.set_power_cache(False)
        state.update(prob=prob, x0=qp.x0, opt=_options(case, qp.b))
    elif what == "bounds":
        qp = _beam(case, seed, 0)
        L, U = _bounds(qp)
        state.update(ctx=ctx, qp=qp, L=L, U=U, x0=np.minimum(np.maximum(qp.x0, L), U),
                     opt=_options(case, qp.b, kind=M.KIND_BOX, project_x0=0))
    elif what == "step":
        E, nu = STIFF
        tets, X, x0, v0 = M.beam_mesh(case["a"], case["b"], case["c"], young=E, poisson=nu,
                                      v0_sigma=0.1, seed=seed + 1)
        fem = M.FemMesh(ctx, tets, X, E, nu, 1000.0)
        prob = M.Problem(ctx, X.size // 3)
        prob.set_x(x0)
        fem.assemble(DT, GRAVITY, x0, v0, prob=prob, precisions=3 if case["mixed"] else 1)
        # the frame before: it also runs the matrix's power method
        prob.collide_planes(STEP_PLANES, STEP_DELTA)
        prob.solve(_options(case, fem.get_b()))
        x = prob.get_x()
        state.update(fem=fem, prob=prob, x=x, v=(x - x0) / DT)
    elif what == "batch":
        qps = [M.beam(*dims, extra_planes_min=w, extra_planes_max=w, plane_mode=2, v0_sigma=0.2,
                      seed=s) for dims, w, s, _ in _burst(case, seed)]
        probs = [M.load_beam(ctx, q, 3 if case["mixed"] else 1) for q in qps]
        for p in probs:
            p.set_power_cache(False)
        state.update(ctx=ctx, probs=probs, x0=[_cuda(q.x0) for q in qps],
                     opts=[_options(case, q.b) for q in qps])
    elif what == "serve":
        scenes = []
        for dims, w, s, more in _burst(case, seed):
            q = M.beam(*dims, extra_planes_min=w, extra_planes_max=w, plane_mode=2, v0_sigma=0.2,
                       seed=s)
            arrays = {k: _cuda(getattr(q, k))
                      for k in ("row_ptr", "cols", "vals", "b", "plane_ptr", "planes", "x0")}
            # a follow-up: the body is pushed a little further down
            push = q.b.copy()
            push[1::3] *= 1.0 - 1e-3
            scenes.append({"nv": q.nv, "nnzb": q.nnzb, "m": len(q.planes), "arrays": arrays,
                           "opt": _options(case, q.b, use_ev=1), "more": more,
                           "b2": _cuda(push),
                           "opt2": _options(case, push, use_ev=1, project_x0=0)})
        server = M.Server(ctx, max_slots=512, quantum_phases=512, power_launches=1003, lanes=3)
        state.update(server=server, scenes=scenes)
    elif what == "product":
        qp = _beam(case, seed, 0)
        prob = M.load_beam(ctx, qp, 2 if case["mixed"] else 1)
        x = torch.from_numpy(_vector(qp.n, seed)).cuda()
        state.update(prob=prob, x=x, y=torch.empty_like(x),
                     prec=M.PREC_MIXED if case["mixed"] else M.PREC_FP64)
    elif what == "assemble":
        E, nu = STIFF
        tets, X, x0, v0 = M.beam_mesh(case["a"], case["b"], case["c"], young=E, poisson=nu,
                                      v0_sigma=0.1, seed=seed + 1)
        fem = M.FemMesh(ctx, tets, X, E, nu, 1000.0)
        state.update(fem=fem, prob=M.Problem(ctx, X.size // 3), x=x0, v=v0, xd=_cuda(x0),
                     y=torch.empty(X.size, dtype=torch.float64, device="cuda"),
                     precisions=3 if case["mixed"] else 1)
    elif what == "ica":
        qp = _beam(case, seed, 1)
        state.update(ctx=ctx, qp=qp, x0=qp.x0)
    else:
        raise ValueError(what)
    ctx.sync()
    return state


def _vector(n, seed):
    return np.random.default_rng(seed + 17).standard_normal(n)


# --------------------------------------------------------------------- run --
def _serve(state):
    server, scenes = state["server"], state["scenes"]
    owner, got = {}, {}
    for i, s in enumerate(scenes):
        a = {k: t.data_ptr() for k, t in s["arrays"].items()}
        t = server.submit_ref(i, s["nv"], s["nnzb"], s["m"], s["opt"], a["b"], a["row_ptr"],
                              a["cols"], a["vals"], a["plane_ptr"], a["planes"], a["x0"])
        owner[t] = (i, 0)
    while owner:
        server.step()
        for t in server.poll():
            i, k = owner.pop(t)
            _, x, face, _, _ = server.result(t)
            got[i, k] = (x, face)
            s = scenes[i]
            if k < s["more"]:
                n = server.submit_ref(i, s["nv"], 0, s["m"], s["opt2"], s["b2"].data_ptr())
                owner[n] = (i, k + 1)
    order = sorted(got)
    return {"x": np.concatenate([got[k][0] for k in order]),
            "face": np.concatenate([got[k][1] for k in order])}


def run(state):
    what = state["what"]
    if what == "solve":
        prob = state["prob"]
        prob.set_x(state["x0"])
        prob.solve(state["opt"])
        return {"x": prob.get_x(), "face": prob.get_face()}
    if what == "bounds":
        x, face, _ = state["ctx"].solve_bsr(state["qp"], state["opt"], state["x0"], state["L"],
                                            state["U"])
        return {"x": x, "face": face}
    if what == "step":
        fem, prob = state["fem"], state["prob"]
        prob.set_x(state["x"])
        fem.rhs(DT, GRAVITY, state["x"], state["v"], prob=prob)
        prob.collide_planes(STEP_PLANES, STEP_DELTA)
        b = fem.get_b()
        prob.solve(_options(state["case"], b, project_x0=0))
        return {"x": prob.get_x(), "face": prob.get_face(), "b": b}
    if what == "batch":
        probs = state["probs"]
        for p, x in zip(probs, state["x0"]):
            p.set_x(x.data_ptr(), on_device=True)
        state["ctx"].solve_batch(probs, state["opts"])
        return {"x": np.concatenate([p.get_x() for p in probs]),
                "face": np.concatenate([p.get_face() for p in probs])}
    if what == "serve":
        return _serve(state)
    if what == "product":
        state["prob"].spmv(state["x"].data_ptr(), state["y"].data_ptr(), state["prec"])
        return {"y": state["y"]}
    if what == "assemble":
        fem, prob = state["fem"], state["prob"]
        fem.assemble(DT, GRAVITY, state["x"], state["v"], prob=prob,
                     precisions=state["precisions"])
        prob.spmv(state["xd"].data_ptr(), state["y"].data_ptr())
        return {"y": state["y"], "b": fem.get_b()}
    x, lam, _ = state["ctx"].ica_solve(state["qp"], state["x0"], max_it=1000, tol=1e-6)
    return {"x": x, "lambda": lam}


# -------------------------------------------------------------------- work --
def _sizes(a, b, c):
    """(vertices, 3x3 blocks) of a beam: the blocks are the vertices and both
    ends of the grid, face-diagonal and body-diagonal edges."""
    nv = (a + 1) * (b + 1) * (c + 1)
    edges = (a * (b + 1) * (c + 1) + (a + 1) * b * (c + 1) + (a + 1) * (b + 1) * c +
             a * b * (c + 1) + a * (b + 1) * c + (a + 1) * b * c + a * b * c)
    return nv, nv + 2 * edges


def _one(a, b, c, mixed, passes):
    """Bytes and operations of one call on a beam: A, b, x and a plane a
    vertex in, x and the active set out; `passes` products with A."""
    nv, nnzb = _sizes(a, b, c)
    value = 4 if mixed else 8
    return (nnzb * (9 * value + 4) + nv * (4 + 3 * 8 * 3 + 32 + 1), 18.0 * nnzb * passes)


def work(case):
    what = case["what"]
    mixed = case.get("mixed", False)
    if what in ("batch", "serve"):
        # the sizes' mean over their log-uniform range
        mean = lambda lo, hi: (hi - lo) / math.log(hi / lo) if hi > lo else lo  # noqa: E731
        side, length = mean(4, case["hi"]), mean(4, case["hi_c"])
        by, fl = _one(round(side), round(side), round(length), mixed, 1060)
        return {"bytes": by * case["count"], "flops": fl * case["count"]}
    dims = (case["a"], case["b"], case["c"])
    nv, nnzb = _sizes(*dims)
    if what == "product":
        value = 4 if mixed else 8
        return {"bytes": nnzb * (9 * value + 4) + nv * (4 + 48), "flops": 18.0 * nnzb}
    if what == "assemble":
        tets = 6 * dims[0] * dims[1] * dims[2]
        # connectivity and positions in; A in each precision, b and y out
        by = tets * 16 + nnzb * (9 * (12 if mixed else 8) + 4) + nv * 5 * 24
        return {"bytes": by, "flops": tets * 16 * 45.0 + 18.0 * nnzb}
    passes = {"solve": 1060, "bounds": 1200, "step": 400, "ica": 1000}[what]
    by, fl = _one(*dims, mixed, passes)
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------------------- exact --
def _element_terms(case, seed):
    """Rest-shape gradients (T, 4, 3), volumes, tets and the state of a beam."""
    E, nu = STIFF
    tets, X, x0, v0 = M.beam_mesh(case["a"], case["b"], case["c"], young=E, poisson=nu,
                                  v0_sigma=0.1, seed=seed + 1)
    P = X.reshape(-1, 3)
    p0 = P[tets[:, 0]]
    D = np.stack([P[tets[:, k]] - p0 for k in (1, 2, 3)], axis=2)
    G = np.linalg.inv(D)  # row k: the gradient of corner k + 1
    grads = np.concatenate([-G.sum(axis=1, keepdims=True), G], axis=1)
    return tets, grads, np.abs(np.linalg.det(D)) / 6.0, P, x0.reshape(-1, 3), v0.reshape(-1, 3)


def _stiffness_times(tets, grads, vol, u):
    """K u element by element: stress of the displacement gradient."""
    E, nu = STIFF
    lam, mu = nu * E / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    H = np.einsum("tai,taj->tij", u[tets], grads)  # du_i / dX_j
    S = mu * (H + H.transpose(0, 2, 1))
    S[:, [0, 1, 2], [0, 1, 2]] += lam * np.trace(H, axis1=1, axis2=2)[:, None]
    F = vol[:, None, None] * np.einsum("tij,taj->tai", S, grads)
    out = np.zeros_like(u)
    for k in range(3):
        out[:, k] = np.bincount(tets.reshape(-1), F[:, :, k].reshape(-1), len(u))
    return out


def _dense(qp):
    A = np.zeros((qp.n, qp.n))
    rows = np.repeat(np.arange(qp.nv), np.diff(qp.row_ptr))
    blocks = qp.vals.reshape(-1, 3, 3)
    for i in range(3):
        for j in range(3):
            A[3 * rows + i, 3 * qp.cols + j] = blocks[:, i, j]
    return A


def _box_qp(A, b, L, U):
    """min 1/2 x'Ax - b'x with L <= x <= U by the primal-dual active set
    method; None if it does not settle."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    At, bt = torch.from_numpy(A).to(dev), torch.from_numpy(b).to(dev)
    low, up = torch.from_numpy(L).to(dev), torch.from_numpy(U).to(dev)
    at_low, at_up = torch.zeros_like(bt, dtype=torch.bool), torch.zeros_like(bt, dtype=torch.bool)
    x = torch.empty_like(bt)
    scale = float(torch.diagonal(At).mean())
    for _ in range(60):
        fixed = at_low | at_up
        free = ~fixed
        x[at_low], x[at_up] = low[at_low], up[at_up]
        sub = At[free][:, free]
        r = bt[free] - At[free][:, fixed] @ x[fixed]
        f = torch.linalg.cholesky(sub)
        y = torch.cholesky_solve(r[:, None], f)
        y += torch.cholesky_solve(r[:, None] - sub @ y, f)
        x[free] = y[:, 0]
        force = (At @ x - bt) / scale
        force[free] = 0.0
        new_low, new_up = force + (low - x) > 0, -force + (x - up) > 0
        if bool((new_low == at_low).all()) and bool((new_up == at_up).all()):
            return x.cpu().numpy()
        at_low, at_up = new_low, new_up
    return None


def _axis_bounds(qp):
    """The axis-aligned planes n.x + p >= 0 as lower bounds of coordinates."""
    L = np.full(qp.n, -np.inf)
    vert = np.repeat(np.arange(qp.nv), np.diff(qp.plane_ptr))
    axis = np.argmax(qp.planes[:, :3], axis=1)
    np.maximum.at(L, 3 * vert + axis, -qp.planes[:, 3])
    return L, 3 * vert + axis


def exact(case, seed):
    what = case["what"]
    if what == "product":
        qp = _beam(case, seed, 0)
        x = _vector(qp.n, seed).reshape(-1, 3)
        rows = np.repeat(np.arange(qp.nv), np.diff(qp.row_ptr))
        t = np.einsum("kij,kj->ki", qp.vals.reshape(-1, 3, 3), x[qp.cols])
        y = np.stack([np.bincount(rows, t[:, i], qp.nv) for i in range(3)], axis=1)
        return {"y": y.reshape(-1)}
    if what == "assemble":
        tets, grads, vol, X, x0, v0 = _element_terms(case, seed)
        mass = np.bincount(tets.reshape(-1), np.repeat(1000.0 * vol / 4.0, 4), len(X))[:, None]
        g = np.array(GRAVITY)
        y = mass * x0 + DT * DT * _stiffness_times(tets, grads, vol, x0)
        b = (mass * (x0 + DT * v0) + DT * DT * mass * g +
             DT * DT * _stiffness_times(tets, grads, vol, X))
        return {"y": y.reshape(-1), "b": b.reshape(-1)}
    if what not in ("solve", "bounds", "ica"):
        return None  # many or very large QPs
    if _sizes(case["a"], case["b"], case["c"])[0] > 3000:
        return None  # a dense factorisation no longer fits the time
    qp = _beam(case, seed, {"solve": _planes_of(case), "bounds": 0, "ica": 1}[what])
    if what == "bounds":
        L, U = _bounds(qp)
    else:
        L, at = _axis_bounds(qp)
        U = np.full(qp.n, np.inf)
    A = _dense(qp)
    x = _box_qp(A, qp.b, L, U)
    if x is None:
        return None
    if what == "ica":
        force = A @ x - qp.b
        return {"x": x, "lambda": np.where(x[at] <= L[at] + 1e-12, force[at], 0.0)}
    return {"x": x, "face": None}
