"""Cell means of the FP32-bulk state on hexahedra are summed in FP64.

A step of length 0 with the Everywhere indicator and the FinDiff limiter returns
every element's mean as a float pair.  Against the FP64 mean of the float pair
it was formed from: one rounding of the low word (2^-49) and those of a sum of
27 terms of one sign with weights that are FP64 roundings (28 x 2^-53), 5e-15."""
import numpy as np
import pytest
import torch

from rkdg3d_gb300 import cases
from rkdg3d_gb300 import mesh as M
from rkdg3d_gb300.solver import (BC_SLIP, FP32_BULK, FUN_BJ, IND_EVERYWHERE, LIM_FINDIFF, RS_HLLC, AVG_EINFELDT,
                                 TUNE_HEX_KERNEL, Context)
from tests.helpers import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 2, 5])
@pytest.mark.parametrize("order,n", [(1, (13, 7, 5)), (2, (7, 6, 5))])
def test_fp32_hexahedral_means(cuda, order, n, variant):
    mesh = M.hex_grid(*n, periodic=(False,) * 3)
    case = cases.Case("means", mesh, order, RS_HLLC, AVG_EINFELDT, bcs=[(a, BC_SLIP, None) for a in range(1, 7)])
    case.limiter = (LIM_FINDIFF, IND_EVERYWHERE, FUN_BJ, 1, 0)
    ctx = Context(mesh, order, device=0, precision=FP32_BULK)
    cases.configure_context(case, ctx)
    ctx.set_tableau(1, [0.0], [1.0], [0.0])
    ctx.set_tuning(TUNE_HEX_KERNEL, variant)
    x = random_state(ctx.node_coords(), seed=51, amp=0.1, vel=0.2)
    hi = x.astype(np.float32).astype(np.float64)
    pair = (hi + (x - hi).astype(np.float32)).reshape(5, -1, (order + 1) ** 3)
    w = np.polynomial.legendre.leggauss(order + 1)[1] / 2
    w3 = (w[:, None, None] * w[:, None] * w).ravel()
    ref = (pair.astype(np.longdouble) * w3).sum(2)
    size = (np.abs(pair) * w3).sum(2)
    xd = torch.tensor(x, device="cuda")
    ctx.step(xd, 0.0)
    got = xd.cpu().numpy().reshape(pair.shape)
    assert np.array_equal(got.min(2), got.max(2))
    assert (np.abs(got[..., 0] - ref) / size).max() < 5e-15
