"""Both column solves on either side of the vertical Courant number up to which their first pass is tried: flat elements
(dz = dx / 8), the face dissipation's diagonal entry d = (impl_fac/2) Lift Fscale_z c at 0.6, 0.97 and 1.03 of the limit
(0.40 to 0.90 for p = 1 to 7).

Float pairs against block LU alone (``set_vi_neumann(0)``) with the tolerance of test_gpu_viseries.py; FP64 against the
oracle with that of test_gpu_fp64_paths.py."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

import oracle as orc  # noqa: E402
from fedg import cases  # noqa: E402
from fedg import lib as fl  # noqa: E402
from test_gpu_mixed import report  # noqa: E402
from test_gpu_parity import perturbed, to_np  # noqa: E402

LIMIT = {1: 0.40, 2: 0.53, 3: 0.65, 4: 0.72, 5: 0.78, 6: 0.83, 7: 0.90}


def flat_case(p, mesh, h=100.0):
    nx, ny, nz = mesh
    return cases.replace(cases.C5().scaled(*mesh, porder=p), eqs="HEVI",
                         dom=(0.0, nx * h, 0.0, ny * h, 0.0, nz * h / 8.0))


def impl_for(case, b, d):
    dz = (case.dom[5] - case.dom[4]) / case.NeZ
    cs = np.sqrt(cases.CPDRY / cases.CVDRY * b["pres_hyd"] / b["dens_hyd"]).max()
    return d / (0.5 * (case.porder + 1) ** 2 / 2.0 * (2.0 / dz) * cs)


@pytest.mark.parametrize("frac", [0.6, 0.97, 1.03])
@pytest.mark.parametrize("p,mesh", [(3, (3, 1, 5)), (3, (2, 2, 16)), (7, (2, 1, 4)), (7, (1, 1, 16))])
def test_pair(p, mesh, frac):
    case = flat_case(p, mesh)
    q, b = cases.initial_state(case)
    s = np.pi * b["z"] / case.dom[5]
    h = np.sin(2 * np.pi * b["x"] / case.dom[1])
    q[4] = q[4] + 1e-3 * b["therm_hyd"] * h * np.cos(s)
    q[3] = q[3] + 0.5 * b["dens_hyd"] * np.sin(s) * h
    dt = impl_for(case, b, frac * LIMIT[p]) / (1.0 - 1.0 / np.sqrt(2.0))
    got = []
    for nterm in (2, 0):
        ctx = fl.Context(case)
        ctx.set_base_state(b["dens_hyd"], b["pres_hyd"], b["therm_hyd"])
        ctx.set_ref_wind(0.0, 0.0)
        ctx.set_vi_neumann(nterm)
        qd = [ctx.tensor(a) for a in q]
        nfail, its = ctx.update(qd, 1, eqs=fl.HEVI, prec=fl.PREC_PAIR, dt=dt, max_iter=30, tol=1e-13)
        assert nfail == 0 and its >= 1.0
        got.append(to_np(qd))
    fe, _ = report("series - LU", got[0], got[1], b)
    assert max(fe) < 1e-9, fe


@pytest.mark.parametrize("frac", [0.6, 0.97, 1.03])
@pytest.mark.parametrize("p", [1, 2, 3, 4, 5, 6, 7])
def test_fp64(p, frac):
    case = flat_case(p, ({1: 309, 2: 141, 3: 79}.get(p, 2), 1, 5))  # smaller meshes of p <= 3 go to block LU
    q0, b = perturbed(case, 6, amp=0.1)
    rng = np.random.default_rng(7)
    sc = [1e-4 * b["dens_hyd"], 0.1, 0.1, 0.1, 0.03]
    q = [a + s * rng.standard_normal(a.shape) for a, s in zip(q0, sc)]
    impl = impl_for(case, b, frac * LIMIT[p])
    o = orc.Oracle(p, case.NeX, case.NeY, case.NeZ, case.dom)
    o.set_base_state(b["dens_hyd"], b["pres_hyd"])
    ref, rfail, _ = o.cal_vi(q, q0, impl, impl, 30, 1e-13, want_iters=True)
    ctx = fl.Context(case)
    ctx.set_base_state(b["dens_hyd"], b["pres_hyd"], b["therm_hyd"])
    got, nfail, _ = ctx.cal_vi([ctx.tensor(a) for a in q], [ctx.tensor(a) for a in q0], impl, impl, 30, 1e-13, want_status=True)
    assert rfail == nfail == 0
    scale = [b["dens_hyd"]] + [340.0 * b["dens_hyd"]] * 3 + [b["therm_hyd"]]
    for g, r, s in zip(to_np(got), ref, scale):
        assert np.max(np.abs(g - r) * impl / s) < 8e-13
