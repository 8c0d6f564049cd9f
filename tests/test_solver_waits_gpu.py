"""Waits inside the solver's kernel are bounded in time: when a grid barrier of a solve's second launch
waits for an arrival that never comes, it gives up after its limit, the call reports PG_ERR_DEVICE and
the context solves afterwards."""
import time

import numpy as np
import pytest

from tests.test_pcg_shapes_gpu import _system

pytestmark = pytest.mark.gpu

LIMIT_MS = 400
SYSTEMS = [("lin_tri3_subscale", (97, 61)), ("lin_tet4_subscale", (19, 14, 23))]


def _solve_in_vain(name, n):
    """A solve whose second launch waits in vain: its x, and the milliseconds the call took."""
    import torch
    from pigfem_b200 import capi
    P, _ = _system(name, n)
    b = torch.from_numpy(np.random.default_rng(3).standard_normal((3, P.n_free))).cuda()

    def solve(x):
        it, _ = P.pcg_solve(b.data_ptr(), x.data_ptr(), 3, 1e-9, 100000)
        return it, x.cpu().numpy()

    it, want = solve(torch.zeros_like(b))
    assert min(it) > 2 * 128          # three launches at least: one is queued behind the second
    P.debug_set("pcg_wait_ms", LIMIT_MS)
    P.debug_set("pcg_missing", 1)
    x = torch.full_like(b, 0.25)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    with pytest.raises(capi.PigfemError) as e:
        solve(x)
    ms = 1e3 * (time.perf_counter() - t0)
    assert e.value.code == 10 and "ran out" in str(e.value)
    P.debug_set("pcg_missing", 0)
    assert np.array_equal(solve(torch.zeros_like(b))[1], want)
    P.close()
    return x.cpu().numpy(), ms


@pytest.mark.parametrize("name,n", SYSTEMS)
def test_a_barrier_that_waits_in_vain_gives_up_at_its_limit(name, n):
    _, ms = _solve_in_vain(name, n)
    assert LIMIT_MS <= ms <= 5 * LIMIT_MS


@pytest.mark.parametrize("name,n", SYSTEMS)
def test_a_solve_that_ran_out_waits_once_and_keeps_its_guess(name, n):
    """The launch queued behind the one that gave up returns at once (two waits would take twice the
    limit), and x is the caller's guess still."""
    x, ms = _solve_in_vain(name, n)
    assert ms < 1.5 * LIMIT_MS
    assert np.all(x == 0.25)
