"""The separable per-vertex form (every plane of a vertex on a coordinate axis
of its own) against the general form and the oracle."""
import numpy as np
import pytest

import helpers as H
import mprgp_gb300 as M

pytestmark = pytest.mark.gpu

SEED = 0x5EED


def _options(qp, rel_tol, **kw):
    return M.default_options(tol=rel_tol * np.linalg.norm(qp.b), max_it=20000, project_x0=1,
                             seed=SEED, **kw)


@pytest.mark.parametrize("dims", [(2, 2, 2), (4, 4, 16), (6, 5, 7), (17, 15, 16)])
@pytest.mark.parametrize("kind", [M.KIND_DECOUPLED, M.KIND_PLANES])
@pytest.mark.parametrize("precision", [M.PREC_FP64, M.PREC_MIXED])
def test_separable_equals_general(ctx, dims, kind, precision):
    """mprgp_solve_noalloc keeps no axis codes, so every vertex takes the
    general form there; on a floor alone both entry points lay the rows out
    alike and the solutions are equal bit for bit."""
    torch = pytest.importorskip("torch")
    qp = M.beam(*dims, v0_sigma=0.2, seed=11)
    opt = _options(qp, 1e-8, kind=kind, precision=precision)
    x, face, st = ctx.solve_bsr(qp, opt, qp.x0)
    d = {k: torch.from_numpy(np.ascontiguousarray(getattr(qp, k))).cuda()
         for k in ("row_ptr", "cols", "vals", "b", "plane_ptr", "planes", "x0")}
    f = torch.zeros(len(qp.planes), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    code, sg = M.solve_noalloc(torch.cuda.current_stream().cuda_stream, qp.nv, qp.nnzb,
                               d["row_ptr"].data_ptr(), d["cols"].data_ptr(),
                               d["vals"].data_ptr(), d["b"].data_ptr(),
                               d["plane_ptr"].data_ptr(), d["planes"].data_ptr(), opt,
                               d["x0"].data_ptr(), f.data_ptr())
    torch.cuda.synchronize()
    assert code == 0 and st.code == 0
    assert (st.iterations, st.num_cg, st.num_exp, st.num_prop) == \
        (sg.iterations, sg.num_cg, sg.num_exp, sg.num_prop)
    assert np.array_equal(x, d["x0"].cpu().numpy()) and np.array_equal(face, f.cpu().numpy())


def test_mixed_vertices_match_oracle(ctx):
    """Separable vertices beside ones that are not -- two planes on one axis,
    a tilted plane -- in one problem: the oracle's solution and active set."""
    qp = M.beam(5, 4, 9, extra_planes_max=2, extra_planes_min=2, plane_mode=2, seed=3)
    lists = [[tuple(p) for p in qp.planes[qp.plane_ptr[v]:qp.plane_ptr[v + 1]]]
             for v in range(qp.nv)]
    # an inactive second floor, or a tilted plane well below the body
    n = np.array([0.6, 0.8, 0.0])
    for v in range(0, qp.nv, 3):
        if len(lists[v]) < 3:
            lists[v].append((0.0, 1.0, 0.0, 0.05) if v % 2 else (*n, 1.0))
    qp.plane_ptr = np.concatenate([[0], np.cumsum([len(p) for p in lists])]).astype(np.int32)
    qp.planes = np.array([p for q in lists for p in q])
    A, b, J, c = H.qp_from_beam(qp)
    opt = _options(qp, 1e-10, kind=M.KIND_PLANES)
    xo, _, so, _ = H.oracle_solve("general", A, b, qp.x0, J, c, tol=opt.tol, max_it=20000, seed=SEED)
    x, face, st = ctx.solve_bsr(qp, opt, qp.x0)
    assert st.code == 0 and int(so["code"]) == 0
    assert np.linalg.norm(x - xo) <= 1e-8 * np.linalg.norm(xo)
    assert np.array_equal(face != 0, np.asarray(H.decide_face_planes(J, c, xo)) != 0)
