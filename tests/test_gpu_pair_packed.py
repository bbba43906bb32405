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
