"""The device PCG over right-hand-side counts, row lengths and system sizes: every count is split into
passes of at most six, rows of cut elements exceed the usual length (some a whole stage), and small
systems leave blocks and warps without work.  Each right-hand side's solution is bitwise the one it
has alone, and meets its tolerance on a host product with the same CSR.  (The 3D cases are periodic:
prescribed u_x alone leaves the rotation about x free, so K_ff is singular.)"""
import os

import numpy as np
import pytest

from tests.conftest import ROOT
from tests.golden.cases import CASES, spec_kwargs

pytestmark = pytest.mark.gpu


def _system(name, n=None):
    import scipy.sparse as sp
    from pigfem_b200 import capi
    c = dict(CASES[name])
    if n is not None:
        c["n"] = n
        if c["elem_type"] == 2:   # a sphere the set-up takes on any grid: its centre at z <= y
            c["incl"] = [[0.52, 0.49, 0.47, 0.31]]
    P = capi.Problem(capi.ProblemDesc(**spec_kwargs(c)))
    out = P.assemble(np.zeros(P.n_nodes * P.dim), 1.0)
    rp, ci, _ = P.pattern(0)
    return P, sp.csr_matrix((out["K_ff"].copy(), ci, rp), shape=(P.n_free, P.n_free))


@pytest.mark.parametrize("name,n", [("lin_tri3_one_fiber", None),
                                    ("lin_tri3_polygon", None), ("lin_quad4_two_fibers_one_element", None),
                                    ("lin_tri3_subscale", (97, 61)), ("lin_tet4_subscale", None),
                                    ("lin_tet4_subscale", (19, 14, 23))])
@pytest.mark.parametrize("nrhs", [1, 2, 4, 5, 6, 7, 16])
def test_any_count_equals_alone_and_solves(name, n, nrhs):
    import torch
    P, K = _system(name, n)
    rng = np.random.default_rng(nrhs)
    B = rng.standard_normal((nrhs, P.n_free))
    X0 = rng.standard_normal((nrhs, P.n_free)) * 1e-6      # a nonzero initial guess
    db = torch.from_numpy(B.copy()).cuda()
    dx = torch.from_numpy(X0.copy()).cuda()
    it, rr = P.pcg_solve(db.data_ptr(), dx.data_ptr(), nrhs, 1e-9, 100000)
    X = dx.cpu().numpy()
    for s in range(nrhs):
        # the tolerance, on the host's own product: the recursive residual drifts by rounding only
        assert np.linalg.norm(K @ X[s] - B[s]) <= 1.01e-9 * np.linalg.norm(B[s])
    for s in {0, nrhs // 2, nrhs - 1}:
        x1 = torch.from_numpy(X0[s].copy()).cuda()
        it1, _ = P.pcg_solve(db[s].contiguous().data_ptr(), x1.data_ptr(), 1, 1e-9, 100000)
        assert it1[0] == it[s] and np.array_equal(x1.cpu().numpy(), X[s])
    P.close()


def test_iteration_limit_and_zero_right_hand_side():
    import torch
    from pigfem_b200 import capi
    P, _ = _system("lin_tet4_subscale")
    b = torch.zeros(2, P.n_free, dtype=torch.float64, device="cuda")
    x = torch.ones_like(b)
    it, rr = P.pcg_solve(b.data_ptr(), x.data_ptr(), 2, 1e-10, 100)     # b = 0: the guess stays
    assert list(it) == [0, 0] and bool((x == 1).all())
    b[0].uniform_(-1, 1)
    x.zero_()
    with pytest.raises(capi.PigfemError):                               # at most one round of 16
        P.pcg_solve(b.data_ptr(), x.data_ptr(), 2, 1e-14, 1)
    it, _ = P.pcg_solve(b.data_ptr(), x.data_ptr(), 2, 1e-10, 100000)   # and the context still solves
    assert it[0] > 0 and it[1] == 0
    P.close()
