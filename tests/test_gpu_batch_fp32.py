"""FP32-bulk batches take the arithmetic of the same problem run alone: it
follows from the element, the order and the precision, not from the batch.

What differs is the Runge-Kutta coefficients: alone the host rounds
coefficient x dt to a float pair, in a batch the device multiplies two float
pairs, equal but for the low word's last bits (2^-46 of the increment).  After
some steps without hard switches the two states agree to 1e-12; FP32 fluxes
rounded in another way part by 1e-9 and more."""
import numpy as np
import pytest
import torch

from rkdg3d_gb300 import cases
from rkdg3d_gb300 import mesh as M
from rkdg3d_gb300.solver import (AVG_EINFELDT, AVG_TRRS, BC_SLIP, FP32_BULK, FUN_VENKATAKRISHNAN, IND_BJ, LIM_MULTI,
                                 RS_HLLC, RS_RUSANOV, Context)
from tests.helpers import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limited", [False, True])
@pytest.mark.parametrize("rs,avg", [(RS_RUSANOV, AVG_TRRS), (RS_HLLC, AVG_EINFELDT)])
@pytest.mark.parametrize("geom,order", [(M.GEOM_SQUARE, 1), (M.GEOM_SQUARE, 2), (M.GEOM_SQUARE, 3),
                                        (M.GEOM_TRIANGLE, 1), (M.GEOM_TRIANGLE, 2)])
def test_batch_equals_alone(cuda, geom, order, rs, avg, limited):
    def grid(n, i):
        if geom == M.GEOM_SQUARE:
            return M.quad_grid(n, 5, 2 * i, 2 * i + 1, 0, 0.7)
        return M.tri_grid(n, 5, 2 * i, 2 * i + 1, 0, 0.7, jitter=0.2, seed=3)

    meshes = [grid(n, i) for i, n in enumerate((23, 40))]
    off = np.concatenate([[0], np.cumsum([m.num_elements for m in meshes])])

    def case_of(mesh):
        c = cases.Case("b", mesh, order, rs, avg, covolume=0.005, bcs=[(a, BC_SLIP, None) for a in range(1, 5)])
        if limited:
            c.limiter = (LIM_MULTI, IND_BJ, FUN_VENKATAKRISHNAN, 1, 0)
        return c

    case = case_of(cases.union_mesh(meshes))
    ctx = Context(case.mesh, order, device=0, precision=FP32_BULK)
    cases.configure_context(case, ctx)
    ctx.batch_setup(off, [1.4, 1.4], [0.005, 0.005])
    x = random_state(ctx.node_coords(), b=0.005, seed=61, amp=0.1, vel=0.2).reshape(4, -1)
    nd = x.shape[1] // case.mesh.num_elements
    xd = torch.tensor(x.ravel(), device="cuda")
    ctx.batch_run(xd, 1e19, dt0=2.0 ** -12, dt_mode=2, max_steps=3, limit_initial=False)
    got = xd.cpu().numpy().reshape(4, -1)
    for p in range(2):
        c = case_of(meshes[p])
        one = Context(c.mesh, order, device=0, precision=FP32_BULK)
        cases.configure_context(c, one)
        cut = slice(nd * off[p], nd * off[p + 1])
        xs = torch.tensor(np.ascontiguousarray(x[:, cut]).ravel(), device="cuda")
        one.run(xs, 1e19, dt0=2.0 ** -12, dt_mode=2, max_steps=3, limit_initial=False)
        ref = xs.cpu().numpy().reshape(4, -1)
        assert np.abs(got[:, cut] - ref).max() <= 1e-12 * np.abs(ref).max()
