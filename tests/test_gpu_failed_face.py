"""A face point whose state is non-physical carries no flux: the call reports the
error, and the neighbour's right-hand side is that of an element whose face
has no integrator, to the rounding of its sums (FP64 1e-12, FP32 1e-5 of the
largest value, the contracts of one right-hand side)."""
import numpy as np
import pytest
import torch

from rkdg3d_gb300 import cases
from rkdg3d_gb300 import mesh as M
from rkdg3d_gb300.solver import (AVG_EINFELDT, AVG_TRRS, BC_SLIP, FP32_BULK, FP64, RS_HLLC, RS_RUSANOV,
                                 TUNE_HEX_KERNEL, Context, UnphysicalStateError)
from tests.helpers import random_state

pytestmark = pytest.mark.gpu


def context(mesh, order, rs, avg, prec, attrs):
    case = cases.Case("fail", mesh, order, rs, avg, bcs=[(a, BC_SLIP, None) for a in attrs])
    ctx = Context(mesh, order, device=0, precision=prec)
    cases.configure_context(case, ctx)
    return ctx


@pytest.mark.parametrize("prec", [FP64, FP32_BULK])
@pytest.mark.parametrize("rs,avg", [(RS_RUSANOV, AVG_TRRS), (RS_HLLC, AVG_EINFELDT)])
@pytest.mark.parametrize("order,variant", [(1, 0), (2, 0), (1, 1), (2, 1), (1, 2), (2, 2), (1, 4), (2, 4), (1, 5), (2, 5)])
def test_failed_face_has_no_flux(cuda, order, variant, rs, avg, prec):
    """Two elements side by side along x, the second one non-physical."""
    two = context(M.hex_grid(2, 1, 1, box=((0, 2), (0, 1), (0, 1)), periodic=(False,) * 3), order, rs, avg, prec,
                  range(1, 7))
    two.set_tuning(TUNE_HEX_KERNEL, variant)
    x = random_state(two.node_coords(), seed=71, amp=0.1, vel=0.2).reshape(5, 2, -1)
    x[0, 1] = -1.0
    y = torch.empty(two.n, dtype=torch.float64, device="cuda")
    with pytest.raises(UnphysicalStateError):
        two.rhs(torch.tensor(x.ravel(), device="cuda"), y)
    got = y.cpu().numpy().reshape(x.shape)[:, 0]
    one = context(M.hex_grid(1, 1, 1, periodic=(False,) * 3), order, rs, avg, prec, (1, 2, 4, 5, 6))  # x = max is open
    one.set_tuning(TUNE_HEX_KERNEL, variant)
    y1 = torch.empty(one.n, dtype=torch.float64, device="cuda")
    one.rhs(torch.tensor(np.ascontiguousarray(x[:, 0]).ravel(), device="cuda"), y1)
    ref = y1.cpu().numpy().reshape(got.shape)
    assert np.abs(got - ref).max() <= (1e-12 if prec == FP64 else 1e-5) * np.abs(ref).max()


@pytest.mark.parametrize("prec", [FP64, FP32_BULK])
@pytest.mark.parametrize("geom", [M.GEOM_SQUARE, M.GEOM_CUBE])
def test_failed_hanging_face_has_no_flux(cuda, geom, prec):
    """A coarse element beside a refined one whose elements are non-physical."""
    if geom == M.GEOM_CUBE:
        base, lone, attrs = (M.hex_grid(2, 1, 1, box=((0, 2), (0, 1), (0, 1)), periodic=(False,) * 3),
                             M.hex_grid(1, 1, 1, periodic=(False,) * 3), (1, 2, 4, 5, 6))
    else:
        base, lone = M.quad_grid(2, 1, 0, 2, 0, 1), M.quad_grid(1, 1, 0, 1, 0, 1)
        right = [a for a, v in zip(lone.bdr_attr, lone.bdr_vertices) if np.allclose(
            [lone.elem_coords[0][list(lone.elem_vertices[0]).index(i)][0] for i in v], 1.0)]
        attrs = [a for a in range(1, 5) if a not in right]
    mesh = M.refine_nc(base, [1])
    ctx = context(mesh, 1, RS_HLLC, AVG_EINFELDT, prec, range(1, 7))
    coarse = int(np.argmin(mesh.elem_coords[..., 0].mean(1)))
    x = random_state(ctx.node_coords(), seed=72, amp=0.1, vel=0.2).reshape(base.dim + 2, mesh.num_elements, -1)
    bad = np.arange(mesh.num_elements) != coarse
    x[0, bad] = -1.0
    y = torch.empty(ctx.n, dtype=torch.float64, device="cuda")
    with pytest.raises(UnphysicalStateError):
        ctx.rhs(torch.tensor(x.ravel(), device="cuda"), y)
    got = y.cpu().numpy().reshape(x.shape)[:, coarse]
    one = context(lone, 1, RS_HLLC, AVG_EINFELDT, prec, attrs)
    y1 = torch.empty(one.n, dtype=torch.float64, device="cuda")
    one.rhs(torch.tensor(np.ascontiguousarray(x[:, coarse]).ravel(), device="cuda"), y1)
    ref = y1.cpu().numpy().reshape(got.shape)
    assert np.abs(got - ref).max() <= (1e-12 if prec == FP64 else 1e-5) * np.abs(ref).max()
