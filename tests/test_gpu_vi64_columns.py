"""FP64 column solve: a column's result is its own.

* A strong change of one column's input leaves every other column's tendency bit for bit as it was.
* The convergence test is an FP64 one: first residuals within 1e-9 of the tolerance, on either side of it, are told apart.
  From var0 = 0, a state of rest, the first residual is q* itself.
* The parts of a decomposed domain equal the whole domain bit for bit at the orders whose elements do not fill whole
  warps of columns (test_gpu_slabs.py holds p = 7).

At p <= 3 the meshes have more than 4 x 152 pairs of columns: smaller ones are left to block LU as a whole.  The size of
the first and the last such mesh is held to the oracle, with the tolerance of test_gpu_fp64_paths.py."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

import oracle as orc  # noqa: E402
from fedg import cases  # noqa: E402
from fedg import lib as fl  # noqa: E402
from test_gpu_parity import perturbed, to_np  # noqa: E402
from test_gpu_slabs import _full, _slabs  # noqa: E402


@pytest.mark.parametrize("max_iter,tol", [(1, 0.0), (30, 1e-12)])
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5, 6, 7])
def test_column_independent_of_the_others(p, max_iter, tol):
    nx = {1: 309, 2: 141, 3: 79}.get(p, 3)
    case = cases.replace(cases.C1().scaled(nx, 1, 3, porder=p), eqs="HEVI")
    q0, b = perturbed(case, 11, amp=0.1)
    rng = np.random.default_rng(12)
    q = [a + s * rng.standard_normal(a.shape) for a, s in zip(q0, (1e-5, 0.01, 0.01, 0.01, 0.003))]
    ctx = fl.Context(case)
    ctx.set_base_state(b["dens_hyd"], b["pres_hyd"], b["therm_hyd"])
    NF, ij = (p + 1) ** 2, (p + 1) ** 2 - 1
    big = [a.copy() for a in q]
    for v in (0, 3, 4):
        big[v].reshape(3, nx, p + 1, NF)[:, 1, :, ij] += 300.0 * (q[v] - q0[v]).reshape(3, nx, p + 1, NF)[:, 1, :, ij]
    got = []
    for x in (q, big):
        t, nfail, _ = ctx.cal_vi([ctx.tensor(a) for a in x], [ctx.tensor(a) for a in q0], 1e-3, 1e-3, max_iter, tol, want_status=True)
        assert nfail == 0
        got.append([a.reshape(3, nx, p + 1, NF) for a in to_np(t)])
    for a, r in zip(*got):
        same = a == r
        if a is not got[0][1] and a is not got[0][2]:  # MOMX and MOMY do not see the change
            assert not same[:, 1, :, ij].all()
        same[:, 1, :, ij] = True
        assert same.all()


@pytest.mark.parametrize("p", [2, 3, 7])
def test_tolerance_in_fp64(p):
    tol = 1e-6
    ne = {2: 144, 3: 81, 7: 9}[p]
    case = cases.replace(cases.C1().scaled(ne // 9, 9, 2, porder=p), eqs="HEVI")
    _, b = cases.initial_state(case)
    NF, rng = (p + 1) ** 2, np.random.default_rng(13)
    ctx = fl.Context(case)
    ctx.set_base_state(b["dens_hyd"], b["pres_hyd"], b["therm_hyd"])
    zero = np.zeros_like(b["dens_hyd"])
    q = [zero.copy() for _ in range(5)]
    below = rng.random((ne, NF)) < 0.5
    dens, lev = (a.reshape(2, ne, p + 1, NF) for a in (b["dens_hyd"], q[0]))
    for e in range(ne):
        for c in range(NF):
            l, f = rng.integers(0, 2 * (p + 1)), 1.0 + 1e-9 * rng.uniform(0.5, 1.0)
            lev[l // (p + 1), e, l % (p + 1), c] = tol * dens[l // (p + 1), e, l % (p + 1), c] * (1.0 / f if below[e, c] else f)
    _, nfail, st = ctx.cal_vi([ctx.tensor(a) for a in q], [ctx.tensor(zero)] * 5, 1e-3, 1e-3, 30, tol, want_status=True)
    assert nfail == 0 and np.array_equal(st.cpu().numpy().reshape(ne, NF) == 0, below)


@pytest.mark.parametrize("p", [1, 2, 4, 5, 6])
def test_parts_equal_one_domain(p):
    case = cases.C2().scaled(*{1: (20, 16, 3), 2: (12, 12, 3)}.get(p, (4, 2, 3)), porder=p)
    q, b = cases.initial_state(case)
    opts = dict(eqs=fl.HEVI, prec=fl.PREC_FP64, dt=0.04, max_iter=30, tol=1e-10)
    want = _full(fl, case, b, q, opts, 3)
    got = _slabs(fl, case, b, q, opts, 3, (2, 2))
    for v in range(5):
        assert np.array_equal(got[v], want[v]), (v, np.abs(got[v] - want[v]).max())


@pytest.mark.parametrize("p,nx", [(1, 304), (1, 305), (2, 135), (2, 136), (3, 76), (3, 77)])
def test_block_lu_rule(p, nx):
    """The largest meshes of the rule (304, 135 and 76 elements: 608 pairs of columns or just below) and the next."""
    case = cases.replace(cases.C1().scaled(nx, 1, 2, porder=p), eqs="HEVI")
    q0, b = perturbed(case, 14, amp=0.1)
    rng = np.random.default_rng(15)
    q = [a + s * rng.standard_normal(a.shape) for a, s in zip(q0, (1e-4 * b["dens_hyd"], 0.1, 0.1, 0.1, 0.03))]
    o = orc.Oracle(p, nx, 1, 2, case.dom)
    o.set_base_state(b["dens_hyd"], b["pres_hyd"])
    ref, rfail, _ = o.cal_vi(q, q0, 1e-3, 1e-3, 30, 1e-13, want_iters=True)
    ctx = fl.Context(case)
    ctx.set_base_state(b["dens_hyd"], b["pres_hyd"], b["therm_hyd"])
    got, nfail, _ = ctx.cal_vi([ctx.tensor(a) for a in q], [ctx.tensor(a) for a in q0], 1e-3, 1e-3, 30, 1e-13, want_status=True)
    assert rfail == nfail == 0
    scale = [b["dens_hyd"]] + [340.0 * b["dens_hyd"]] * 3 + [b["therm_hyd"]]
    for g, r, s in zip(to_np(got), ref, scale):
        assert np.max(np.abs(g - r) * 1e-3 / s) < 8e-13
