"""The limiter's last hope (StateIsPhysical at the vertices) judges states of any
magnitude, also where density times energy underflows.

A step of length 0 with the Multi limiter.  Variations below the indicator's
+-1e-3 switch leave a physical element as it is; what stays has to be the float
pair (or the double) that went in."""
import pytest
import torch

from rkdg3d_gb300 import cases
from rkdg3d_gb300 import mesh as M
from rkdg3d_gb300.solver import (AVG_EINFELDT, BC_SLIP, FP32_BULK, FP64, FUN_BJ, IND_BJ, LIM_MULTI, RS_RUSANOV, Context)
from tests.helpers import random_state, rel_l1

pytestmark = pytest.mark.gpu


def box(geom, order):
    mesh = M.hex_grid(3, 3, 2, periodic=(False,) * 3) if geom == M.GEOM_CUBE else M.quad_grid(5, 3, 0, 1, 0, 0.7)
    case = cases.Case("hope", mesh, order, RS_RUSANOV, AVG_EINFELDT, bcs=[(a, BC_SLIP, None) for a in range(1, 7)])
    case.limiter = (LIM_MULTI, IND_BJ, FUN_BJ, 1, 0)
    return case


@pytest.mark.parametrize("prec,scale", [(FP32_BULK, 1e-20), (FP64, 1e-160)])
@pytest.mark.parametrize("geom,order", [(M.GEOM_SQUARE, 1), (M.GEOM_SQUARE, 2), (M.GEOM_CUBE, 1), (M.GEOM_CUBE, 2)])
def test_tiny_states_stay(cuda, geom, order, prec, scale):
    case = box(geom, order)
    ctx = Context(case.mesh, order, device=0, precision=prec)
    cases.configure_context(case, ctx)
    ctx.set_tableau(1, [0.0], [1.0], [0.0])
    x = random_state(ctx.node_coords(), seed=81, amp=0.1, vel=0.2) * scale
    xd = torch.tensor(x, device="cuda")
    ctx.step(xd, 0.0)
    assert rel_l1(xd.cpu().numpy(), x) < (1e-13 if prec == FP64 else 1e-6)
