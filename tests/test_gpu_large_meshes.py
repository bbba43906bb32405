"""The kernels that only larger meshes take: the far side of each size at which the tracer's and the numerical diffusion's
launches change (elements per block, nodes per thread, registers), each with an odd element count or a ragged last block.

Against the FP64 oracle with the tolerances of the same comparisons on small meshes (FP64 tracer 1e-12 and float pairs
1e-11 relative L2, diffusion 1e-10 of the largest change).  Above 8192 elements at p = 7 a periodic mesh of three tiles
holds the same flow in each, and is compared with the tile, which the other cases compare with the oracle; the sums of an
element are taken in another order there, so the bound is twice the float pairs'."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

from fedg import cases  # noqa: E402
from fedg import lib as fl  # noqa: E402
from test_gpu_nd import VARS, setup as setup_nd  # noqa: E402
from test_gpu_trc import setup as setup_trc, t1  # noqa: E402


def tracer_step(ctx, Q, q, aM, aP, dt, limiter, prec):
    qd = [ctx.tensor(a) for a in q]
    Qd = ctx.tensor(Q)
    ctx.trc_update(Qd, qd[1:4], ctx.tensor(aM), ctx.tensor(aP), qd[0], qd[0], dt, nsteps=1, limiter=limiter, tmar=limiter,
                   prec=prec)
    return Qd.cpu().numpy()


@pytest.mark.parametrize("p,ne,prec,tol", [
    (3, (19, 13, 10), fl.PREC_FP64, 1e-12),  # four elements per block (2470, the last one half empty)
    (3, (9, 7, 11), fl.PREC_PAIR, 1e-11),    # more than a block per SM (693)
    (7, (7, 5, 3), fl.PREC_PAIR, 1e-11),     # two elements per block, at most a block per SM (105)
    (7, (7, 9, 5), fl.PREC_PAIR, 1e-11),     # two nodes per thread in the stage (315)
])
@pytest.mark.parametrize("limiter", [True, False])
def test_tracer(p, ne, prec, tol, limiter):
    case = t1(ne, p)
    o, ctx, q, b, _ = setup_trc(case, seed=80, wobble=0.3)
    Q = 1.0 + np.random.default_rng(81).random(o.shape)
    aM, aP = o.trc_alphdens_advtest(q[0], q[1], q[2], q[3])
    dt = 0.05 * case.dt
    ref = o.trc_step(Q, q[1:4], aM, aP, q[0], q[0], dt, nsteps=1, limiter=limiter, tmar=limiter)
    got = tracer_step(ctx, Q, q, aM, aP, dt, limiter, prec)
    assert np.linalg.norm(got - ref) < tol * np.linalg.norm(ref)


def test_tracer_pair_two_nodes_everywhere():
    """8379 elements at p = 7: two nodes per thread in the coefficient kernel as well."""
    small, big = t1((7, 19, 21), 7), t1((21, 19, 21), 7)
    q, b = cases.initial_state(small)
    rng = np.random.default_rng(82)
    for v, s in ((0, 3e-4 * b["dens_hyd"]), (1, 0.9), (2, 0.9), (3, 0.3)):
        q[v] = q[v] + s * rng.standard_normal(q[v].shape)
    Q = 1.0 + rng.random(q[0].shape)
    tile = lambda a: np.tile(a.reshape(21, 19, 7, -1), (1, 1, 3, 1)).reshape(big.Ne, -1)  # noqa: E731
    got = []
    for case, f in ((small, lambda a: a), (big, tile)):
        ctx = fl.Context(case)
        ctx.set_base_state(*[f(b[k]) for k in ("dens_hyd", "pres_hyd", "therm_hyd")])
        qs = [f(a) for a in q[:4]]
        aM, aP = (t.cpu().numpy() for t in ctx.trc_alphdens_advtest(*[ctx.tensor(a) for a in qs]))
        got.append(tracer_step(ctx, f(Q), qs, aM, aP, 0.05 * small.dt, True, fl.PREC_PAIR))
        ctx.close()
    ref = tile(got[0])
    assert np.linalg.norm(got[1] - ref) < 2e-11 * np.linalg.norm(ref)


@pytest.mark.parametrize("nlap", [1, 2])
def test_numdiff_pair_two_nodes(nlap):
    """1001 elements at p = 7: two nodes per thread."""
    case = cases.C2().scaled(7, 11, 13)
    o, ctx, q, b = setup_nd(case, 83)
    coef = {1: 2.0e2, 2: 5.0e5}[nlap]
    ref = o.numdiff_apply(q, nlap, coef, 0.5 * coef, 0.01)
    qd = [ctx.tensor(a) for a in q]
    ctx.numdiff_apply(qd, nlap, coef, 0.5 * coef, 0.01, prec=fl.PREC_PAIR)
    for v in range(5):
        dref = ref[v] - q[v]
        err = np.max(np.abs((qd[v].cpu().numpy() - q[v]) - dref)) / np.max(np.abs(dref))
        assert err < 1e-10, (VARS[v], err)
