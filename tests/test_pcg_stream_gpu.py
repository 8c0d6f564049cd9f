"""The device PCG on systems whose matrix does not stay in shared memory: a warp's ring of stages is
refilled chunk after chunk, through several launches of one solve, and row groups longer than a stage
are read from global memory.  Ordinary meshes have none of the latter, and many chunks a warp only in
systems of benchmark size, so some cases lower a chunk's capacity ("pcg_stage_values").

Each right-hand side's solution is bitwise the one it has alone and the one of every repeat, and meets
its tolerance on a host product with the same CSR.  Bound: the residual the iteration carries differs
from b - A x by the rounding of its updates, at most eps per iteration of |A| |x| (twice, for r and x)."""
import numpy as np
import pytest

from tests.test_pcg_shapes_gpu import _system
from tests.golden.cases import CASES, spec_kwargs

pytestmark = pytest.mark.gpu

RTOL = 1e-7


def _solve(P, b, x0):
    import torch
    db, dx = torch.from_numpy(b.copy()).cuda(), torch.from_numpy(x0.copy()).cuda()
    it, _ = P.pcg_solve(db.data_ptr(), dx.data_ptr(), b.shape[0], RTOL, 100000)
    return it, dx.cpu().numpy()


# name, grid, chunk capacity (0: a stage's), chunks read directly: none, some or all
@pytest.mark.parametrize("name,n,values,direct", [
    ("lin_tri3_subscale", (420, 410), 0, "none"), ("lin_tet4_subscale", (34, 33, 35), 0, "none"),
    ("lin_tri3_subscale", (160, 150), 36, "some"), ("lin_tet4_subscale", (19, 14, 23), 136, "some"),
    ("lin_tri3_subscale", (160, 150), 4, "all"), ("lin_tet4_subscale", (19, 14, 23), 16, "all")])
@pytest.mark.parametrize("nrhs", [1, 6])
def test_streamed_matrix(name, n, values, direct, nrhs):
    P, K = _system(name, n)
    P.debug_set("pcg_stage_values", values)
    rng = np.random.default_rng(7 + nrhs)
    B = rng.standard_normal((nrhs, P.n_free))
    X0 = rng.standard_normal((nrhs, P.n_free)) * 1e-6
    it, X = _solve(P, B, X0)
    blocks, chunks, per_warp, stages, n_direct = P.debug("pcg_shape")
    assert per_warp > stages                                   # the ring is refilled
    assert {"none": n_direct == 0, "some": 0 < n_direct < chunks, "all": n_direct == chunks}[direct]
    norm = abs(K).sum(axis=1).max()
    for s in range(nrhs):
        drift = 2 * np.finfo(np.float64).eps * (it[s] + 1) * norm * np.linalg.norm(X[s])
        assert np.linalg.norm(K @ X[s] - B[s]) <= RTOL * np.linalg.norm(B[s]) + drift
    if not values:
        assert max(it) > 128                                   # and over launches of the solve
    for s in {0, nrhs - 1}:
        it1, x1 = _solve(P, B[s:s + 1], X0[s:s + 1])
        assert it1[0] == it[s] and np.array_equal(x1[0], X[s])
    for _ in range(20 if not values else 3):
        again, x2 = _solve(P, B, X0)
        assert list(again) == list(it) and np.array_equal(x2, X)
    P.close()


def test_chunk_capacity_is_set_before_the_first_solve():
    from pigfem_b200 import capi
    P, _ = _system("lin_tri3_subscale")
    _solve(P, np.ones((1, P.n_free)), np.zeros((1, P.n_free)))
    with pytest.raises(capi.PigfemError):
        P.debug_set("pcg_stage_values", 8)
    with pytest.raises(capi.PigfemError):
        P.debug_set("no_such_setting", 1)
    P.close()
