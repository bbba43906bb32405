"""What the FP64 column solve's refinement pass leaves to block LU, against the oracle.

* ``max_iter`` below 1 allows no solve: every column whose first residual is above ``tol`` is reported as failed and
  keeps var0, as the oracle's Newton loop does.  No solve takes part, so the step agrees to the 1e-11 of the other
  single-step comparisons."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

import oracle as orc  # noqa: E402
from fedg import cases  # noqa: E402
from fedg import lib as fl  # noqa: E402
from test_gpu_parity import perturbed, relerr, to_np  # noqa: E402


def pair_of(case, b):
    o = orc.Oracle(case.porder, case.NeX, case.NeY, case.NeZ, case.dom)
    o.set_base_state(b["dens_hyd"], b["pres_hyd"])
    ctx = fl.Context(case)
    ctx.set_base_state(b["dens_hyd"], b["pres_hyd"], b["therm_hyd"])
    return o, ctx


@pytest.mark.parametrize("max_iter", [0, -1])
@pytest.mark.parametrize("p", [2, 3, 7])
def test_no_solve_allowed(p, max_iter):
    case = cases.replace(cases.C1().scaled(2, 1, 3, porder=p), eqs="HEVI")
    q, b = perturbed(case, 8, amp=0.3)
    o, ctx = pair_of(case, b)
    ref, rfail, _ = o.step_hevi(q, 1e-3, 1, max_iter=max_iter, tol=1e-13)
    qd = [ctx.tensor(a) for a in q]
    nfail, its = ctx.update(qd, 1, eqs=fl.HEVI, dt=1e-3, max_iter=max_iter, tol=1e-13)
    assert nfail == rfail == 2 * case.NeX * case.NeY * (p + 1) ** 2 and its == 0.0
    assert max(relerr(g, r) for g, r in zip(to_np(qd), ref)) < 1e-11
