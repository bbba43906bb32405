"""What the FP64 column solve's refinement pass leaves to block LU, against the oracle.

* ``max_iter`` below 1 allows no solve: every column whose first residual is above ``tol`` is reported as failed and
  keeps var0, as the oracle's Newton loop does.  No solve takes part, so the step agrees to the 1e-11 of the other
  single-step comparisons.
* A right-hand side of S = 1e37 (in MOMZ) overflows the FP32 sweeps, not the FP64 problem: the one linearised solve
  of ``max_iter = 1``, which no later residual checks, is finite and equals the oracle's.  The tendency is a difference
  from q* over dt, so it is compared as in test_gpu_fp64_paths.py, times dt against the size of the right-hand side:
  S, S / 340 m/s of density and 300 K of that in RHOT, 8e-13 of it."""
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


@pytest.mark.parametrize("p", [2, 3, 7])
def test_overflowing_sweeps(p):
    case = cases.replace(cases.C1().scaled({2: 141, 3: 79}.get(p, 2), 1, 3, porder=p), eqs="HEVI")
    q0, b = perturbed(case, 9, amp=0.1)
    q = [a.copy() for a in q0]
    q[3] = q0[3] + 1e37 * np.sin(np.pi * b["z"] / case.dom[5])
    o, ctx = pair_of(case, b)
    dt = 1e-3
    ref, rfail, _ = o.cal_vi(q, q0, dt, dt, 1, 0.0, want_iters=True)
    got, nfail, _ = ctx.cal_vi([ctx.tensor(a) for a in q], [ctx.tensor(a) for a in q0], dt, dt, 1, 0.0, want_status=True)
    assert nfail == rfail == 0
    for v, scale in ((0, 1e37 / 340.0), (3, 1e37), (4, 1e37 * 300.0 / 340.0)):
        assert np.max(np.abs(got[v].cpu().numpy() - ref[v])) * dt / scale < 8e-13, v
