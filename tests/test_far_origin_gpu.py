"""Structured rows of a box far from the origin.  The shapes of a uniform grid depend on the cell size
alone, so K's structured rows, and the residual they give for the same displacements, are those of the
same box at the origin bit for bit (the corners are powers of two and sums of few, so the box has the
same size in both places).  The other rows are formed from the nodes' coordinates, which are rounded
at the box's distance: relative to K, 16 of those roundings (eps |lo| / h) bound them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TRI3, QUAD4, TET4 = 0, 1, 2
LO = (1024.0, -512.0, 2048.0)


def _problem(elem, n, lo):
    from pigfem_b200 import capi
    dim = 3 if elem == TET4 else 2
    return capi.Problem(capi.ProblemDesc(elem_type=elem, n=n, lo=lo[:dim],
                                         hi=[a + b for a, b in zip(lo, (1.0, 0.75, 1.25))][:dim]))


@pytest.mark.parametrize("elem,n", [(TRI3, (49, 37)), (QUAD4, (49, 37)), (TET4, (11, 13, 9))])
def test_structured_rows_depend_on_the_cell_size_alone(elem, n):
    from pigfem_b200 import capi
    far, near = _problem(elem, n, LO), _problem(elem, n, (0.0, 0.0, 0.0))
    dim, U = far.dim, np.random.default_rng(2).uniform(-1e-3, 1e-3, far.n_nodes * far.dim)
    nodes = far.debug("dn_node")[far.debug("fast_dn")]
    dofs = far.nodes()[1][nodes].reshape(-1)
    assert len(dofs) and dofs.max() < far.n_free
    rp, _, _ = far.pattern(0)
    vals = np.concatenate([np.arange(rp[d], rp[d + 1]) for d in dofs])
    steps = 16 * np.finfo(np.float64).eps * max(abs(a) * k for a, k in zip(LO[:dim], n)) / 0.75
    for flags in (capi.FUNC | capi.JAC, capi.FUNC | capi.JAC | capi.FP32):
        a, b = far.assemble(U, 1.0, flags=flags), near.assemble(U, 1.0, flags=flags)
        assert np.array_equal(a["K_ff"][vals], b["K_ff"][vals])
        assert np.array_equal(a["P_f"][dofs], b["P_f"][dofs])
        assert np.abs(a["K_ff"] - b["K_ff"]).max() <= steps * np.abs(b["K_ff"]).max()
    far.close()
    near.close()
