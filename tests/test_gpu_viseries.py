"""The float-pair column solve's series kernel against the same solve with LU corrections only
(``set_vi_neumann(0)``), and both against the FP64 oracle, over the shapes of its layout: one element per
column, odd counts, columns of 1 to 64 elements, p = 3 and 7, at vertical Courant numbers where the series solves every
column (test_gpu_physics.py runs the float-pair path at Courant numbers of 2 to 4, where the columns go to
the LU kernel).

Tolerance: both solves accept a residual of at most 1e-13 of DENS_hyd, 340 m/s DENS_hyd and RHOT_hyd, so two
implicit stages differ by a few 1e-13 of those scales times ||J^-1|| (below 4 here); momentum is measured
against 1 m/s of hydrostatic momentum, which takes MOMZ to 340 x 1e-12 < 1e-9."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

import oracle as orc  # noqa: E402
from fedg import cases  # noqa: E402
from fedg import lib as fl  # noqa: E402
from test_gpu_mixed import report  # noqa: E402
from test_gpu_parity import to_np  # noqa: E402


def smooth_state(p, mesh):
    case = cases.replace((cases.C1() if p == 3 else cases.C5()).scaled(*mesh), eqs="HEVI")
    q, b = cases.initial_state(case)
    xmin, xmax, ymin, ymax, zmin, zmax = case.dom
    h = np.sin(2 * np.pi * (b["x"] - xmin) / (xmax - xmin)) + 0.5 * np.cos(2 * np.pi * (b["y"] - ymin) / (ymax - ymin))
    s = np.pi * (b["z"] - zmin) / (zmax - zmin)
    q[4] = q[4] + 1e-3 * b["therm_hyd"] * h * np.cos(s)
    q[3] = q[3] + 0.5 * b["dens_hyd"] * np.sin(s) * h
    q[1] = q[1] + b["dens_hyd"] * np.cos(s) * h
    return case, q, b


def solve(case, q, b, nterm, dt, tol, max_iter=30):
    ctx = fl.Context(case)
    ctx.set_base_state(b["dens_hyd"], b["pres_hyd"], b["therm_hyd"])
    ctx.set_ref_wind(0.0, 0.0)
    ctx.set_vi_neumann(nterm)
    qd = [ctx.tensor(a) for a in q]
    nfail, its = ctx.update(qd, 1, eqs=fl.HEVI, prec=fl.PREC_PAIR, dt=dt, max_iter=max_iter, tol=tol)
    return to_np(qd), nfail, its


@pytest.mark.parametrize("p,mesh,dt", [
    (3, (1, 1, 1), 0.01), (3, (3, 1, 5), 0.01), (3, (2, 3, 64), 0.01),
    (7, (1, 1, 1), 0.002), (7, (1, 3, 2), 0.002), (7, (1, 1, 13), 0.002), (7, (1, 1, 14), 0.002), (7, (3, 1, 17), 0.002), (7, (1, 1, 33), 0.002),
])
def test_series_equals_lu(p, mesh, dt):
    case, q, b = smooth_state(p, mesh)
    o = orc.Oracle(case.porder, case.NeX, case.NeY, case.NeZ, case.dom)
    o.set_base_state(b["dens_hyd"], b["pres_hyd"])
    ref = o.step_hevi(q, dt, 1, max_iter=30, tol=1e-13)[0]
    got = []
    for nterm in (2, 0):
        x, nfail, its = solve(case, q, b, nterm, dt, 1e-13)
        assert nfail == 0 and its >= 1.0
        got.append(x)
    fe, _ = report("series - LU", got[0], got[1], b)
    assert max(fe) < 1e-9, fe
    fe, _ = report("series - oracle", got[0], ref, b)
    assert max(fe) < 1e-9, fe


@pytest.mark.parametrize("p", [3, 7])
def test_iteration_limit_reports_the_columns(p):
    """max_iter = 1 leaves every column of a perturbed state unconverged at tol 1e-13, as LU alone does."""
    case = cases.replace((cases.C1() if p == 3 else cases.C5()).scaled(2, 1, 3), eqs="HEVI")
    q, b = cases.initial_state(case)
    q[4] = q[4] + 1e-3 * b["therm_hyd"] * np.cos(np.pi * b["z"] / case.dom[5])
    fails = []
    for nterm in (2, 0):
        ctx = fl.Context(case)
        ctx.set_base_state(b["dens_hyd"], b["pres_hyd"], b["therm_hyd"])
        ctx.set_vi_neumann(nterm)
        qd = [ctx.tensor(a) for a in q]
        fails.append(ctx.update(qd, 1, eqs=fl.HEVI, prec=fl.PREC_PAIR, dt=0.005, max_iter=1, tol=1e-13)[0])
    assert fails[0] == fails[1] > 0


@pytest.mark.parametrize("p", [3, 7])
def test_mixed_warps_count_each_column_once(p):
    """Warps of the LU kernel with columns that the series accepted beside columns that it left: a NaN at one node
    reaches the nodes on its lines in the first stage, so in its element and the four beside it some pairs of columns
    are not finite and the others are.  Each implicit stage counts each column once, either as failed or with its
    solves, so the mean times the columns that did not fail is a whole number.  Away from those elements (the mesh is
    wide enough for two stages) the step is bit-equal to the one without the NaN."""
    case, q, b = smooth_state(p, (7, 7, 2))
    dt = 0.01 if p == 3 else 0.002
    tol = 1e-10  # some columns take one solve, others two
    want, nfail, _ = solve(case, q, b, 2, dt, tol)
    assert nfail == 0
    q = [a.copy() for a in q]
    q[0][24, 0] = np.nan  # element (3, 3), layer 0, node (0, 0, 0)
    x, nfail, its = solve(case, q, b, 2, dt, tol)
    solved = 2 * 49 * (p + 1) ** 2 - nfail
    assert 0 < nfail < solved
    assert 1.0 < its < 2.0 and abs(its * solved - round(its * solved)) < 1e-6, (its, nfail)
    for g, r in zip(x, want):
        for e in (0, 6, 42, 48):
            assert np.array_equal(g[e], r[e])
