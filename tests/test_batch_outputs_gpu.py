"""Batched calls for the residual alone, or the matrices alone: the outputs asked for are bitwise those of
each context assembled alone, the others keep what the call before left, whichever graph ran last."""
import numpy as np
import pytest

from tests.test_batch_gpu import _outputs, _problems

pytestmark = pytest.mark.gpu

NAMES = {2: ["coh_bl", "coh_xn", "lin_tri3_three_fibers", "coh_bl_polygon", "lin_tri3_subscale"],
         3: ["coh_tet4_bl", "coh_tet4_opaug_two_spheres", "lin_tet4_subscale", "lin_tet4_uncut"]}


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("fp32", [False, True], ids=["fp64", "fp32_mixed"])
def test_outputs_asked_for_alone(dim, fp32):
    from pigfem_b200 import capi
    mixed = capi.FP32 if fp32 else 0
    probs, us = _problems(NAMES[dim], extra_2d=2 if dim == 2 else 0)
    others = [0.75 * u for u in us]
    B = capi.Batch(probs)

    def batch(u, flags):
        B.assemble([x.data_ptr() for x in u], flags)
        B.wait()
        return [_outputs(P) for P in probs]

    def alone(u, flags):
        out = []
        for P, x in zip(probs, u):
            P.assemble_device(x.data_ptr(), 1.0, flags)
            out.append(_outputs(P))
        return out

    both = capi.FUNC | capi.JAC | mixed
    want = {"us": alone(us, both), "others": alone(others, both)}
    state = batch(us, both)
    for flags, u, name in ((capi.FUNC | mixed, others, "others"), (capi.JAC | mixed, others, "others"),
                           (capi.JAC | mixed, us, "us"), (capi.FUNC | mixed, us, "us")):
        got = batch(u, flags)
        for i, g in enumerate(got):
            for k in g:
                # (internal variables and zones come from the law, whatever is asked for)
                asked = k not in ("K_ff", "K_fp", "K_pf", "K_pp", "P_f", "P_p") or bool(flags & (capi.JAC if k[0] == "K" else capi.FUNC))
                assert np.array_equal(g[k], (want[name] if asked else state)[i][k]), (flags, i, k)
        state = got
    B.close()
    for P in probs:
        P.close()
