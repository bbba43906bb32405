"""The FP64 kernels at the edges of their branches.

* DPRES at the ends of the ranges of the pressure's binomial series (|DRHOT/THERM_hyd| = 2^-8 and 2^-4),
  against an extended-precision pow.  Both branches round a handful of times (THERM_hyd**kap, its
  argument, the sum, the product), each below one unit of PRES: 8 * 2^-53 PRES.
* The fused SSP-RK3 stage against the separate tendency, Runge-Kutta and filter kernels, which run when
  tracer-flux outputs are registered: every node takes the same roundings in both, so they agree bit for bit.
* The column solve by iterative refinement over element orders and column shapes (odd column counts, one
  element, the tallest column), at a step its sweeps solve and at one that goes to block LU, against the
  oracle.  Both accept a residual of 1e-13 of DENS_hyd, 340 m/s DENS_hyd and RHOT_hyd, so with ||J^-1|| below 4 the
  solutions differ by less than 8e-13 of those scales."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

import oracle as orc  # noqa: E402
from fedg import cases  # noqa: E402
from fedg import lib as fl  # noqa: E402
from test_gpu_parity import perturbed, to_np  # noqa: E402


def context(case, b):
    ctx = fl.Context(case)
    ctx.set_base_state(b["dens_hyd"], b["pres_hyd"], b["therm_hyd"])
    return ctx


@pytest.mark.skipif(np.finfo(np.longdouble).eps > 1e-18, reason="needs an extended-precision long double")
@pytest.mark.parametrize("p", [1, 3])
def test_dpres_series_edges(p):
    case = cases.C1().scaled(2, 1, 3, porder=p)
    _, b = cases.initial_state(case)
    e = 2.0 ** -52
    x = [0.0, 1e-18, 1e-5, 2.0 ** -8 * (1 - e), 2.0 ** -8, 2.0 ** -8 * (1 + e), 0.03, 2.0 ** -4 * (1 - e), 2.0 ** -4,
         2.0 ** -4 * (1 + e), 0.3]
    x = np.array(x + [-v for v in x])
    th, ph = b["therm_hyd"], b["pres_hyd"]
    dr = th * np.resize(x, th.shape)
    ctx = context(case, b)
    pres, dpres = to_np(ctx.drhot2pres(ctx.tensor(dr)))
    ld = np.longdouble
    p00, rd, kap = ld(cases.PRES00), ld(cases.RDRY), ld(cases.CPDRY / cases.CVDRY)
    ref = p00 * (rd / p00 * (ld(1) * th + dr)) ** kap
    bound = 8 * 2.0 ** -53 * np.asarray(ref, float)
    assert np.all(np.abs(pres - ref) <= bound)
    assert np.all(np.abs(dpres - (ref - ph)) <= bound)


@pytest.mark.parametrize("p", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("mesh", [(1, 1, 1), (3, 1, 3)])
def test_fused_stage_bitwise(p, mesh):
    case = cases.C1().scaled(*mesh, porder=p)
    q, b = perturbed(case, 5, amp=0.3)
    got = []
    for flux in (False, True):
        ctx = context(case, b)
        if flux:
            ctx.set_tracer_flux([ctx.empty() for _ in range(3)] + [ctx.empty_face() for _ in range(2)] +
                                [ctx.empty() for _ in range(2)])
        qd = [ctx.tensor(a) for a in q]
        ctx.update(qd, 2, eqs=fl.HEVE, dt=1e-3)
        got.append(to_np(qd))
        ctx.set_tracer_flux(None)
    for a, r in zip(*got):
        assert np.all(np.isfinite(r)) and np.array_equal(a, r)


@pytest.mark.parametrize("dt", [0.004, 0.1])
@pytest.mark.parametrize("p,mesh", [(1, (1, 1, 1)), (2, (3, 1, 64)), (4, (1, 3, 2)), (5, (1, 1, 7)), (6, (1, 1, 64)),
                                    (7, (1, 1, 1)), (7, (1, 1, 64))])
def test_refinement_column_solve(p, mesh, dt):
    case = cases.C1().scaled(*mesh, porder=p)
    q0, b = perturbed(case, 6, amp=0.1)
    rng = np.random.default_rng(7)
    sc = [1e-4 * b["dens_hyd"], 0.1, 0.1, 0.1, 0.03]
    q = [a + s * rng.standard_normal(a.shape) for a, s in zip(q0, sc)]
    o = orc.Oracle(p, *mesh, case.dom)
    o.set_base_state(b["dens_hyd"], b["pres_hyd"])
    ref, rfail, _ = o.cal_vi(q, q0, dt, dt, 30, 1e-13, want_iters=True)
    ctx = context(case, b)
    got, nfail, _ = ctx.cal_vi([ctx.tensor(a) for a in q], [ctx.tensor(a) for a in q0], dt, dt, 30, 1e-13, want_status=True)
    assert rfail == nfail == 0
    scale = [b["dens_hyd"]] + [340.0 * b["dens_hyd"]] * 3 + [b["therm_hyd"]]
    for g, r, s in zip(to_np(got), ref, scale):
        assert np.max(np.abs(g - r) * dt / s) < 8e-13
