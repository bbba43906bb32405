"""The float-pair stage kernel at the edges of its layout.

* A periodic mesh tiled two or three times in x and y holds the same flow in every tile, and every node's
  arithmetic is independent of where its element lies: the tiles equal the small mesh bit for bit.  The
  small meshes are one element (its own neighbour), odd element counts (the last block of two p = 3
  elements half empty) and one element layer (both vertical faces are lids).
* A smooth state whose DRHOT / RHOT_hyd crosses the range of the pressure's binomial series (3 %) inside
  the elements, where one node of a packed pair takes pow() and the other does not, against the FP64
  oracle.  The fields are continuous across the elements, so the FP32 wave speed multiplies roundoff-size
  jumps in the first stage and O(dt) ones later: the 1e-9 of the other float-pair tests holds."""
import numpy as np
import pytest

from conftest import have_gpu

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_gpu(), reason="needs a CUDA GPU")]

import oracle as orc  # noqa: E402
from fedg import cases  # noqa: E402
from fedg import lib as fl  # noqa: E402
from test_gpu_mixed import report  # noqa: E402
from test_gpu_parity import to_np  # noqa: E402


def run(case, q, b, dt, steps):
    ctx = fl.Context(case)
    ctx.set_base_state(b["dens_hyd"], b["pres_hyd"], b["therm_hyd"])
    ctx.set_ref_wind(0.0, 0.0)
    qd = [ctx.tensor(a) for a in q]
    nfail, _ = ctx.update(qd, steps, eqs=fl.HEVE, prec=fl.PREC_PAIR, dt=dt)
    assert nfail == 0
    return to_np(qd)


@pytest.mark.parametrize("mesh", [(1, 1, 1), (1, 3, 2), (3, 1, 3), (5, 3, 1)])
@pytest.mark.parametrize("p,dt", [(3, 2e-3), (7, 1e-3)])
def test_tiles_equal_bitwise(p, dt, mesh):
    base = cases.C1() if p == 3 else cases.C5()
    nx, ny, nz = mesh
    small = cases.replace(base.scaled(nx, ny, nz), eqs="HEVE")
    q, b = cases.initial_state(small)
    rng = np.random.default_rng(3)
    q = [a + s * b["dens_hyd"] * rng.uniform(-1, 1, size=a.shape) for a, s in zip(q, (1e-3, 1.0, 1.0, 0.3, 0.3))]
    ref = run(small, q, b, dt, 2)
    tx, ty = 3, 2
    big = cases.replace(base.scaled(nx * tx, ny * ty, nz), eqs="HEVE")
    _, bb = cases.initial_state(big)
    shape = (nz, ny, nx, small.Np)
    tile = lambda a: np.tile(a.reshape(shape), (1, ty, tx, 1)).reshape(big.Ne, big.Np)  # noqa: E731
    for k in ("dens_hyd", "pres_hyd", "therm_hyd"):
        bb[k] = tile(b[k])
    got = run(big, [tile(a) for a in q], bb, dt, 2)
    for g, r in zip(got, ref):
        assert np.array_equal(g, tile(r))


@pytest.mark.parametrize("p,dt", [(3, 2e-3), (7, 1e-3)])
def test_pressure_series_and_pow_in_one_element(p, dt):
    case = cases.replace((cases.C1() if p == 3 else cases.C5()).scaled(2, 2, 2), eqs="HEVE", noise={}, bubble={})
    q, b = cases.initial_state(case)
    xmin, xmax, ymin, ymax, zmin, zmax = case.dom
    w = np.sin(2 * np.pi * (b["x"] - xmin) / (xmax - xmin)) * np.cos(2 * np.pi * (b["y"] - ymin) / (ymax - ymin)) * np.cos(
        np.pi * (b["z"] - zmin) / (zmax - zmin))
    q[4] = q[4] + 0.06 * b["therm_hyd"] * w
    q[0] = q[0] + 0.02 * b["dens_hyd"] * w
    o = orc.Oracle(case.porder, case.NeX, case.NeY, case.NeZ, case.dom)
    o.set_base_state(b["dens_hyd"], b["pres_hyd"])
    ref = o.step_heve(q, dt, 1)
    fe, _ = report(f"pair pow p={p}", run(case, q, b, dt, 1), ref, b)
    assert max(fe) < 1e-9, fe
