"""RKDG_TUNE_GENERIC_BLOCK sets the CTA of the planar face pass (and element pass):
every size gives the same bits, right-hand side and wave speeds, in a batch too."""
import numpy as np
import pytest
import torch

from rkdg3d_gb300 import cases
from rkdg3d_gb300 import mesh as M
from rkdg3d_gb300.solver import (AVG_TRRS, BC_SLIP, FP32_BULK, FP64, RS_HLLC, TUNE_GENERIC_BLOCK, Context)
from tests.helpers import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [FP64, FP32_BULK])
@pytest.mark.parametrize("geom,order", [(M.GEOM_SQUARE, 1), (M.GEOM_SQUARE, 2), (M.GEOM_SQUARE, 3),
                                        (M.GEOM_TRIANGLE, 1), (M.GEOM_TRIANGLE, 2)])
def test_face_pass_blocks(cuda, geom, order, prec):
    mesh = M.quad_grid(37, 23, 0, 1, 0, 0.7) if geom == M.GEOM_SQUARE else M.tri_grid(37, 23, 0, 1, 0, 1, jitter=0.2)
    case = cases.Case("tune", mesh, order, RS_HLLC, AVG_TRRS, bcs=[(a, BC_SLIP, None) for a in range(1, 5)])
    seen = None
    for block in (0, 32, 96, 256):
        ctx = Context(mesh, order, device=0, precision=prec)
        cases.configure_context(case, ctx)
        ctx.set_tuning(TUNE_GENERIC_BLOCK, block)
        x = torch.tensor(random_state(ctx.node_coords(), seed=95), device="cuda")
        y = torch.empty_like(x)
        out = [ctx.face_speed(x), ctx.rhs(x, y)]
        ctx.step(x, 1e-4)
        out += [y.cpu().numpy(), x.cpu().numpy()]
        ctx.batch_setup([0, mesh.num_elements], [1.4], [0.0])
        ctx.batch_run(x, 1.0, 0.3, max_steps=2, limit_initial=False)
        out.append(x.cpu().numpy())
        if seen is not None:
            assert out[:2] == seen[:2]
            assert all(np.array_equal(a, b) for a, b in zip(out[2:], seen[2:]))
        seen = out
