"""A solve whose working memory cannot be had, at each of its allocations in turn, reports it and leaves
the context as it was: the next solve allocates what is missing, gives the bits of an undisturbed
context's and holds the same memory.  (The allocations fail on the host; nothing is launched.)"""
import numpy as np
import pytest

from tests.test_pcg_shapes_gpu import _system

pytestmark = pytest.mark.gpu


def _solve(P, nrhs):
    import torch
    b = torch.from_numpy(np.random.default_rng(5).standard_normal((6, P.n_free))[:nrhs].copy()).cuda()
    x = torch.zeros_like(b)
    P.pcg_solve(b.data_ptr(), x.data_ptr(), nrhs, 1e-9, 100000)
    return x.cpu().numpy()


@pytest.mark.parametrize("name", ["lin_tri3_subscale", "lin_tet4_subscale"])
def test_solve_after_a_failed_allocation(name):
    from pigfem_b200 import capi
    P, _ = _system(name)
    want6, held = _solve(P, 6), P.device_bytes()[0]
    P.close()
    failed = 0
    for k in range(1, 40):
        P, _ = _system(name)
        P.debug_set("fail_alloc", k)
        try:
            got = _solve(P, 6)
        except capi.PigfemError as e:
            assert e.code == 10          # PG_ERR_DEVICE
            failed += 1
            u = np.zeros(P.n_nodes * P.dim)
            P.assemble(u, 1.0)           # the rest of the context is unharmed
            assert np.array_equal(_solve(P, 6), want6)
            assert P.device_bytes()[0] == held
            P.close()
            continue
        assert np.array_equal(got, want6)   # k is past the solve's allocations
        P.close()
        break
    assert failed == 13                     # six tables, seven vectors: all were reached


def test_failed_growth_keeps_the_context_usable():
    from pigfem_b200 import capi
    P, _ = _system("lin_tet4_subscale")
    want1 = _solve(P, 1)
    for k in range(1, 8):
        P.debug_set("fail_alloc", k)
        with pytest.raises(capi.PigfemError):
            _solve(P, 6)
        assert np.array_equal(_solve(P, 1), want1)
    want6 = _solve(P, 6)
    assert np.array_equal(want6[0], want1[0])
    P.close()
