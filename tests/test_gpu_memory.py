"""The face pass's slots are as wide as the context's precision, and the
hexahedral variants of one kernel hold none: what a context gives back when such a
variant is chosen (in pages of 2 MiB)."""
import pytest
import torch

from rkdg3d_gb300 import cases
from rkdg3d_gb300.solver import FP32_BULK, FP64, TUNE_HEX_KERNEL, Context
from tests.helpers import random_state, rel_l1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,width", [(FP64, 8), (FP32_BULK, 4)])
def test_face_slots_follow_precision_and_variant(cuda, prec, width):
    case = cases.pulse3d(n=32, order=2)
    ctx = Context(case.mesh, case.order, device=0, precision=prec)
    cases.configure_context(case, ctx)
    slots = 3 * 32 ** 3 * 5 * 9 * width
    torch.cuda.synchronize()
    free = [torch.cuda.mem_get_info()[0]]
    for variant in (2, 3, 1, 0):
        ctx.set_tuning(TUNE_HEX_KERNEL, variant)
        free.append(torch.cuda.mem_get_info()[0])
    page = 2 << 20
    assert abs(free[1] - free[0] - slots) <= page
    assert abs(free[2] - free[0]) <= page and abs(free[4] - free[0]) <= page
    assert abs(free[3] - free[0] - slots) <= page
    # and the precision can be changed after the mesh
    x = torch.tensor(random_state(ctx.node_coords(), seed=96, amp=0.02, vel=0.05), device="cuda")
    y, z = torch.empty_like(x), torch.empty_like(x)
    ctx.rhs(x, y)
    ctx.set_precision(FP32_BULK if prec == FP64 else FP64)
    ctx.rhs(x, z)
    assert rel_l1(z.cpu().numpy(), y.cpu().numpy()) < 1e-5
    torch.cuda.synchronize()
    ctx.set_tuning(TUNE_HEX_KERNEL, 2)
    before = torch.cuda.mem_get_info()[0]
    ctx.set_tuning(TUNE_HEX_KERNEL, 0)
    assert abs(before - torch.cuda.mem_get_info()[0] - slots * (12 - width) // width) <= page


@pytest.mark.parametrize("stages", [1, 3])
def test_adjoint_scratch_follows_the_tableau(cuda, stages):
    """Order 1 hexahedra and SSP-RK3: the reverse step's vectors, the traces'
    cotangents (6.75 state vectors) and the limiter's derivatives take no more than
    22 state vectors."""
    case = cases.pulse3d(n=40, order=1)
    ctx = Context(case.mesh, case.order, device=0, precision=FP64)
    cases.configure_context(case, ctx)
    if stages == 1:
        ctx.set_tableau(1, [0.0], [1.0], [0.0])
    x = torch.tensor(random_state(ctx.node_coords(), seed=97, amp=0.02, vel=0.05), device="cuda")
    k, out, g = torch.randn_like(x), torch.empty_like(x), torch.randn_like(x)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ctx.rhs_vjp(x, k, out)
    used = free - torch.cuda.mem_get_info()[0]
    vectors = used / (8 * ctx.n)
    assert vectors < (22 if stages == 3 else 14.2)
    ctx.step_vjp(x, 1e-4, g)  # runs within them
    assert free - torch.cuda.mem_get_info()[0] == used
    assert torch.isfinite(g).all()
