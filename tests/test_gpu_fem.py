"""GPU FEM assembly (mprgp_fem_*): A = M + h^2 K and b = M(x + h v) + h^2 M g
+ h^2 K X of a tetrahedral mesh, against the host assembly of the same beam
(mprgp_beam_build), and solves from the GPU-assembled system."""
import numpy as np
import pytest

import mprgp_gb300 as M

pytestmark = pytest.mark.gpu

KW = dict(extra_planes_max=2, extra_planes_min=2, plane_mode=2, seed=41)


def _sorted_rows(row_ptr, cols, vals):
    """Per row, blocks sorted by column (the host generator's order may differ)."""
    out_c, out_v = [], []
    for r in range(len(row_ptr) - 1):
        s, e = row_ptr[r], row_ptr[r + 1]
        o = np.argsort(cols[s:e], kind="stable")
        out_c.append(cols[s:e][o])
        out_v.append(vals[s:e][o])
    return np.concatenate(out_c), np.concatenate(out_v)


@pytest.mark.parametrize("dims", [(3, 2, 5), (6, 5, 12)])
def test_gpu_assembly_matches_host(ctx, dims):
    qp = M.beam(*dims, **KW)
    p = qp.params
    tets, X, x0, v0 = M.beam_mesh(*dims, **KW)
    assert np.array_equal(x0, qp.x0)
    fem = M.FemMesh(ctx, tets, X, p["young"], p["poisson"], p["rho"])
    fem.assemble(p["dt"], (0.0, p["gravity"], 0.0), x0, v0)
    rp, cols, vals, b, mass = fem.get()
    fem.close()
    assert np.array_equal(rp, qp.row_ptr)
    hc, hv = _sorted_rows(qp.row_ptr, np.asarray(qp.cols), np.asarray(qp.vals).reshape(-1, 9))
    assert np.array_equal(cols, hc)
    assert np.abs(vals - hv).max() <= 1e-13 * np.abs(hv).max()
    assert np.linalg.norm(b - qp.b) <= 1e-13 * np.linalg.norm(qp.b)
    assert np.all(mass > 0)


def test_solve_from_gpu_assembly(ctx):
    dims = (6, 5, 12)
    qp = M.beam(*dims, **KW)
    p = qp.params
    grav = (0.0, p["gravity"], 0.0)
    tets, X, x0, v0 = M.beam_mesh(*dims, **KW)
    fem = M.FemMesh(ctx, tets, X, p["young"], p["poisson"], p["rho"])
    pr = M.Problem(ctx, qp.nv)
    fem.assemble(p["dt"], grav, x0, v0, prob=pr, precisions=3)
    pr.set_planes(qp.plane_ptr, qp.planes)
    pr.set_x(x0)
    opt = M.default_options(tol=1e-10 * np.linalg.norm(qp.b), max_it=20000, kind=M.KIND_PLANES,
                            project_x0=1, seed=0x5EED)
    st = pr.solve(opt)
    xg = pr.get_x()
    xh, _, sh = ctx.solve_bsr(qp, opt, qp.x0)
    assert st.code == 0 and sh.code == 0
    assert np.linalg.norm(xg - xh) <= 1e-8 * np.linalg.norm(xh)
    # the next timestep: only b is recomputed on the device
    v1 = (xg - x0) / p["dt"]
    fem.rhs(p["dt"], grav, xg, v1, prob=pr)
    _, _, _, b1, mass = fem.get()
    m3 = np.repeat(mass, 3)
    g3 = np.tile(grav, qp.nv)
    kx = (qp.b - m3 * (x0 + p["dt"] * v0) - p["dt"] ** 2 * m3 * g3) / p["dt"] ** 2
    b1_ref = m3 * (xg + p["dt"] * v1) + p["dt"] ** 2 * m3 * g3 + p["dt"] ** 2 * kx
    assert np.linalg.norm(b1 - b1_ref) <= 1e-10 * np.linalg.norm(b1_ref)
    opt.project_x0 = 0
    st2 = pr.solve(opt)
    assert st2.code == 0
    fem.close()
    pr.close()


def _assembled(tets, X, E, nu, rho, h):
    """A of the mesh by element blocks in numpy, dense."""
    lam, mu = nu * E / ((1 + nu) * (1 - 2 * nu)), E / (2 * (1 + nu))
    P = X.reshape(-1, 3)
    A = np.zeros((X.size, X.size))
    for t in tets:
        D = (P[t[1:]] - P[t[0]]).T
        G = np.linalg.inv(D)
        g = np.vstack([-G.sum(axis=0), G])
        V = abs(np.linalg.det(D)) / 6
        for i in range(4):
            A[3 * t[i]:3 * t[i] + 3, 3 * t[i]:3 * t[i] + 3] += rho * V / 4 * np.eye(3)
            for j in range(4):
                K = V * (lam * np.outer(g[i], g[j]) + mu * np.outer(g[j], g[i]) +
                         mu * (g[i] @ g[j]) * np.eye(3))
                A[3 * t[i]:3 * t[i] + 3, 3 * t[j]:3 * t[j] + 3] += h * h * K
    return A


def _hub(points, rng):
    """Points on a spiral and one vertex (the first) joined to all of them."""
    ang = np.arange(points - 1) * 0.37
    ring = np.stack([np.cos(ang), np.sin(ang), 0.1 * np.arange(points - 1)], axis=1)
    ring += 0.05 * rng.standard_normal(ring.shape)
    i = np.arange(1, points - 2)
    return (np.vstack([[0.1, 0.2, -1.0], ring]),
            np.stack([np.zeros_like(i), i, i + 1, i + 2], axis=1))


@pytest.mark.parametrize("points,hub", [
    (4, "first"),     # a single tet: one partial warp
    (33, "last"),     # one row past a warp
    (89, "first"),    # the widest row that fits shared memory
    (90, "first"),    # one that does not: the form in global memory
    (150, "first"),
    (150, "last"),
])
def test_assembly_of_a_hub(ctx, points, hub):
    """A vertex joined to every other one, on both sides of the width that
    shared memory holds.  Bound: a block sums at most 200 element blocks, so
    200 eps times the largest entry, and ten times that for the gradients'
    own rounding on random tets."""
    rng = np.random.default_rng(points)
    P, tets = _hub(points, rng)
    if hub == "last":
        P = np.vstack([P[1:], P[:1]])
        tets = (tets - 1) % points
    E, nu, rho, h = 1e5, 0.4, 1000.0, 0.01
    X = P.reshape(-1).copy()
    fem = M.FemMesh(ctx, tets.astype(np.int32), X, E, nu, rho)
    fem.assemble(h, (0.0, -9.8, 0.0), X)
    rp, cols, vals, b, mass = fem.get()
    A = _assembled(tets, X, E, nu, rho, h)
    got = np.zeros_like(A)
    for r in range(points):
        for k in range(rp[r], rp[r + 1]):
            got[3 * r:3 * r + 3, 3 * cols[k]:3 * cols[k] + 3] = vals[k].reshape(3, 3)
    assert np.abs(got - A).max() <= 2000 * 2.2e-16 * np.abs(A).max()
    K = (A - np.kron(np.diag(mass), np.eye(3)))
    m3 = np.repeat(mass, 3)
    g = np.tile([0.0, -9.8, 0.0], points)
    want = m3 * X + h * h * m3 * g + K @ X
    scale = np.abs(K).sum(axis=1).max() * np.abs(X).max() + np.abs(want).max()
    assert np.abs(b - want).max() <= 2000 * 2.2e-16 * scale
    fem.close()


@pytest.mark.parametrize("dims", [(1, 1, 1), (3, 4, 7), (9, 9, 9)])
def test_assembly_forms_agree(ctx, dims):
    """A body beside a hub too wide for shared memory is assembled in global
    memory; alone, in shared memory: the same operations in the same order, so
    the same bits."""
    rng = np.random.default_rng(5)
    tets, X, x0, v0 = M.beam_mesh(*dims, young=1e5, poisson=0.4, v0_sigma=0.1, seed=3)
    tets = np.asarray(tets).reshape(-1, 4)
    X = X + 0.003 * rng.standard_normal(X.size)
    P, hub = _hub(120, rng)
    both = []
    for t, x in ((tets, X), (np.vstack([tets, hub + X.size // 3]), np.hstack([X, P.ravel() + 9]))):
        fem = M.FemMesh(ctx, t.astype(np.int32), x, 1e5, 0.4, 1000.0)
        fem.assemble(0.01, (0.0, -9.8, 0.0), x)
        both.append(fem.get())
    nv = X.size // 3
    nb = both[0][0][nv]
    for one, two, n in zip(both[0], both[1], (nv + 1, nb, nb, X.size, nv)):
        assert np.array_equal(np.asarray(one).reshape(n, -1), np.asarray(two)[:n].reshape(n, -1))
