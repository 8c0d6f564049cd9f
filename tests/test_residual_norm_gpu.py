"""The residual norm at systems of one value less than a block takes, of exactly a block, of one block
and a few values, and of several (periodic grids, whose DOF count can be even); and after a launch that
failed, which is reported instead of the value the call before left."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, periodic=True):
    from pigfem_b200 import capi
    return capi.Problem(capi.ProblemDesc(elem_type=0, n=n, lo=(0.0, 0.0), hi=(1.0, 0.7), subscale=periodic,
                                         eps_macro=(0.01, -0.004, 0.002, 0.0, 0.0, 0.0) if periodic else (0.0,) * 6))


# (bound: the rounding of a sum of n squares in a tree, far below 1e-13 relative)
@pytest.mark.parametrize("n,periodic,n_free", [((32, 64), True, 4094), ((3, 683), True, 4096), ((40, 51), False, 4159),
                                               ((6, 683), True, 8194), ((4, 1024 * 4 + 1), True, 32774)])
def test_norm_at_block_boundaries(n, periodic, n_free):
    P = _problem(n, periodic)
    assert P.n_free == n_free
    U = np.random.default_rng(1).uniform(-1e-3, 1e-3, P.n_nodes * 2)
    ref = np.linalg.norm(P.assemble(U, 1.0)["P_f"])
    got = [P.residual_norm() for _ in range(3)]
    assert abs(got[0] - ref) <= 1e-13 * ref and got[0] == got[1] == got[2]
    P.close()


def test_a_launch_that_failed_is_reported():
    from pigfem_b200 import capi
    P = _problem((10, 12))
    rng = np.random.default_rng(1)
    P.assemble(rng.uniform(-1e-3, 1e-3, P.n_nodes * 2), 1.0)
    first = P.residual_norm()
    ref = np.linalg.norm(P.assemble(rng.uniform(-1e-2, 1e-2, P.n_nodes * 2), 1.0)["P_f"])
    P.debug_set("fail_launch", 1)
    with pytest.raises(capi.PigfemError) as e:
        P.residual_norm()
    assert e.value.code == 10
    again = P.residual_norm()
    assert again != first and abs(again - ref) <= 1e-13 * ref
    P.close()
