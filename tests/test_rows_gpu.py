"""Structured and general rows at the sizes where their split can go wrong: grids with no structured
node, a single one, odd row starts (runs that begin on an odd CSR value), runs longer and shorter than
a chunk, hx != hy, ply boundaries (nodes between two materials are general), periodic images, and each
element type, against the element-by-element sums of perf.cases in 64-bit torch.  Bounds: K and P are
sums of at most 24 element terms per entry, so 1e-13 of the block's norm is far above their rounding;
FP32-mixed K 1e-5, the stated accuracy of that option."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TRI3, QUAD4, TET4 = 0, 1, 2


def _desc(elem, n, incl, law, periodic, ply=0.0):
    from pigfem_b200 import capi, rve
    dim = 3 if elem == TET4 else 2
    coh, par = (capi.COH_BL, rve.BL_PARAMS) if law else (capi.COH_NONE, (0.0,) * 4)
    return capi.ProblemDesc(elem_type=elem, n=n, lo=(0.0,) * dim, hi=(1.0, 0.7, 1.3)[:dim],
                            inclusions=np.array(incl, dtype=np.float64).reshape(-1, dim + 1), coh_law=coh, coh=par,
                            subscale=periodic, eps_macro=(0.01, -0.004, 0.002, 0.001, -0.002, 0.003) if periodic else (0.0,) * 6,
                            ply_frac=ply, ply=(36.2e3, 7.11e3, 2.32e3, 2.17e3, 0.335) if ply else (0.0,) * 5)


CIRCLE, SPHERE = [[0.41, 0.37, 0.183]], [[0.52, 0.37, 0.31, 0.213]]
GRIDS = [(TRI3, (2, 2), [], False, False), (TRI3, (3, 2), [], False, False), (TRI3, (4, 4), [], False, True),
         (TRI3, (131, 9), CIRCLE, False, False), (TRI3, (67, 70), CIRCLE, True, False), (TRI3, (33, 41), CIRCLE, False, True),
         (QUAD4, (2, 2), [], False, False), (QUAD4, (97, 13), CIRCLE, True, False), (QUAD4, (23, 31), CIRCLE, False, True),
         (TET4, (2, 3, 2), [], False, False), (TET4, (4, 3, 5), [], False, True), (TET4, (9, 17, 11), SPHERE, True, False),
         (TET4, (13, 8, 10), SPHERE, False, True)]


def _rel(a, b):
    n = np.linalg.norm(b)
    return np.linalg.norm(a - b) / n if n else float(np.abs(a).max(initial=0.0))


@pytest.mark.parametrize("elem,n,incl,law,periodic", GRIDS)
def test_rows_against_element_sums(elem, n, incl, law, periodic):
    from perf import cases
    from pigfem_b200 import capi, rve
    P = capi.Problem(_desc(elem, n, incl, law, periodic))
    if law:
        U = rve.interface_state(P, seed=3)
    else:
        U = np.random.default_rng(4).uniform(-1e-3, 1e-3, P.n_free + P.n_const)[P.nodes()[1].reshape(-1)]
    E = cases._Exact(P, {"law": "bilinear" if law else "none"})
    vals, F = E.assemble(U, [np.array(P.desc.eps_macro)[:E.nv]])
    ref = {k: v.cpu().numpy() for k, v in cases._named(P, vals, F).items()}
    for flags, tol in ((capi.FUNC | capi.JAC, 1e-13), (capi.FUNC | capi.JAC | capi.FP32, 1e-5)):
        out = P.assemble(U, 1.0, flags=flags)
        for k, v in ref.items():
            assert _rel(out[k], v) <= (tol if k == "K_ff" else 1e-13), (k, flags, _rel(out[k], v))
    full = P.assemble(U, 1.0)
    only = P.assemble(U, 1.0, flags=capi.FUNC)
    assert np.array_equal(only["P_f"], full["P_f"]) and np.array_equal(only["P_p"], full["P_p"])
    P.close()


@pytest.mark.parametrize("elem,n", [(TRI3, (40, 30)), (QUAD4, (40, 30)), (TET4, (8, 15, 7))])
def test_ply_boundaries_are_general_rows(elem, n):
    """Structured nodes have one material around them; K's rows of the others come from the image:
    K is symmetric and annihilates translations to rounding (the largest entry times 1e-12)."""
    import scipy.sparse as sp
    from pigfem_b200 import capi
    P = capi.Problem(_desc(elem, n, [], False, True, ply=0.2))
    out = P.assemble(np.zeros(P.n_nodes * P.dim), 1.0)
    blocks = [P.pattern(b) for b in range(4)]
    K = sp.bmat([[sp.csr_matrix((out["K_" + k].copy(), blocks[b][1], blocks[b][0]), shape=blocks[b][2])
                  for b, k in row] for row in (((0, "ff"), (1, "fp")), ((2, "pf"), (3, "pp")))]).tocsr()
    top = np.abs(K.data).max()
    assert np.abs((K - K.T).data).max(initial=0.0) <= 1e-12 * top
    dofs = P.nodes()[1]
    for d in range(P.dim):
        t = np.zeros(K.shape[0])
        t[dofs[:, d]] = 1.0
        assert np.abs(K @ t).max() <= 1e-11 * top
    P.close()


@pytest.mark.parametrize("n", [(2, 2), (40, 50), (45, 45), (46, 45), (120, 97)])
def test_residual_norm_over_block_counts(n):
    """One block, exactly one and a few more values than a block, several blocks, repeated calls: the
    norm of the host copy to the rounding of a sum of n squares (1e-13 relative), the same bits twice."""
    from pigfem_b200 import capi
    P = capi.Problem(_desc(TRI3, n, [], False, False))
    U = np.random.default_rng(1).uniform(-1e-3, 1e-3, P.n_nodes * 2)
    ref = np.linalg.norm(P.assemble(U, 1.0)["P_f"])
    got = [P.residual_norm() for _ in range(3)]
    assert abs(got[0] - ref) <= 1e-13 * ref and got[0] == got[1] == got[2]
    P.close()
