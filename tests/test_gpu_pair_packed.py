"""Kernels that carry two consecutive elements per thread, on meshes where a pair of elements straddles
rows, lids and layers or the last element has no partner; all element orders.

Numerical diffusion in float pairs against the FP64 oracle, with the bound of the other float-pair tests: the
change of each field, relative to the largest change, within 1e-10."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

from fedg import cases  # noqa: E402
from fedg import lib as fl  # noqa: E402
from test_gpu_nd import VARS, setup  # noqa: E402
from test_gpu_trc import setup as setup_trc, t1  # noqa: E402


@pytest.mark.parametrize("porder", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("ne,nlap", [((1, 1, 1), 1), ((3, 1, 3), 2), ((1, 3, 5), 1)])
def test_numdiff_pair(porder, ne, nlap):
    case = cases.C1().scaled(*ne, porder=porder)
    o, ctx, q, b = setup(case, seed=50 + porder)
    coef = {1: 2.0e2, 2: 5.0e5}[nlap]
    ref = o.numdiff_apply(q, nlap, coef, 0.5 * coef, 0.01)
    qd = [ctx.tensor(a) for a in q]
    ctx.numdiff_apply(qd, nlap, coef, 0.5 * coef, 0.01, prec=fl.PREC_PAIR)
    for v in range(5):
        dref = ref[v] - q[v]
        err = np.max(np.abs((qd[v].cpu().numpy() - q[v]) - dref)) / max(np.max(np.abs(dref)), 1e-300)
        assert err < 1e-10, (VARS[v], err)


@pytest.mark.parametrize("porder", [1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("ne", [(1, 1, 1), (3, 1, 3), (1, 3, 5)])
@pytest.mark.parametrize("limiter", [True, False])
def test_tracer_pair(porder, ne, limiter):
    """Two tracer steps with a source, distinct densities and (limiter) the filter, against the FP64 oracle, with
    the float-pair tests' 1e-11 relative L2."""
    case = t1(ne, porder)
    o, ctx, q, b, _ = setup_trc(case, seed=60 + porder, wobble=0.3)
    rng = np.random.default_rng(61)
    Q = 1.0 + rng.random(o.shape)
    mf = [q[1], q[2], q[3]]
    aM, aP = o.trc_alphdens_advtest(q[0], q[1], q[2], q[3])
    dd = [q[0] + s * b["dens_hyd"] * rng.standard_normal(o.shape) for s in (1e-4, 2e-4)]
    rhoq = 1e-5 * rng.random(o.shape)
    filt = dict(etac_h=2.0 / 3.0, alpha_h=36.0, ord_h=16, etac_v=0.5, alpha_v=30.0, ord_v=12) if limiter else None
    dt = 0.05 * case.dt
    ref = o.trc_step(Q, mf, aM, aP, dd[0], q[0], dt, nsteps=2, ddens=dd[1], rhoq_tp=rhoq, limiter=limiter, tmar=True,
                     filter=filt)
    Qd = ctx.tensor(Q)
    ctx.trc_update(Qd, [ctx.tensor(m) for m in mf], ctx.tensor(aM), ctx.tensor(aP), ctx.tensor(dd[0]), ctx.tensor(q[0]), dt,
                   nsteps=2, ddens=ctx.tensor(dd[1]), rhoq_tp=ctx.tensor(rhoq), limiter=limiter, tmar=True, filter=filt,
                   prec=fl.PREC_PAIR)
    got = Qd.cpu().numpy()
    assert np.linalg.norm(got - ref) < 1e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("ne", [(16, 38, 4), (17, 13, 11)])
def test_tracer_fp64_block_rule(ne):
    """p = 3 at the largest mesh of the two-elements-per-block rule (2432 elements, a whole wave) and at the one
    below it (2431, the last block half empty): one limited step against the oracle, FP64 on both sides."""
    case = t1(ne, 3)
    o, ctx, q, b, _ = setup_trc(case, seed=70, wobble=0.3)
    Q = 1.0 + np.random.default_rng(71).random(o.shape)
    aM, aP = o.trc_alphdens_advtest(q[0], q[1], q[2], q[3])
    dt = 0.05 * case.dt
    ref = o.trc_step(Q, q[1:4], aM, aP, q[0], q[0], dt, nsteps=1, limiter=True, tmar=True)
    qd = [ctx.tensor(a) for a in q]
    Qd = ctx.tensor(Q)
    ctx.trc_update(Qd, qd[1:4], ctx.tensor(aM), ctx.tensor(aP), qd[0], qd[0], dt, nsteps=1, limiter=True, tmar=True)
    got = Qd.cpu().numpy()
    assert np.linalg.norm(got - ref) < 1e-12 * np.linalg.norm(ref)
