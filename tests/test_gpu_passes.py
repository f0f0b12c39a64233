"""The two-pass right-hand sides, the limiter's teams, the wave-speed kernels and
the limiter VJP at the edges of their tiles: one element, one CTA and one
more element, the line between the small and the large CTA, and remainders.

Tolerances: FP64 against the oracle 1e-12, the parity contract of
test_gpu_parity.py; FP32 1e-5, its contract for one right-hand side (a unit
roundoff of 6e-8, at most ~100 terms of one sign in the sums)."""
import numpy as np
import pytest
import torch

from oracle.refcpu import Oracle
from rkdg3d_gb300 import cases
from rkdg3d_gb300 import mesh as M
from rkdg3d_gb300.solver import (AVG_EINFELDT, AVG_TRRS, BC_SLIP, FP32_BULK, FP64, FUN_BJ, FUN_MICHALAK,
                                 FUN_VENKATAKRISHNAN, IND_BJ, IND_EVERYWHERE, LIM_FINDIFF, LIM_MULTI,
                                 RS_HLL, RS_HLLC, RS_RUSANOV, TUNE_LIMITER_BLOCK, Context)
from tests.helpers import random_state, rel_l1
from tests.test_gpu_adjoint import fd_check

pytestmark = pytest.mark.gpu

TOL = {FP64: 1e-12, FP32_BULK: 1e-5}
QUAD, TRI, HEX = M.GEOM_SQUARE, M.GEOM_TRIANGLE, M.GEOM_CUBE


def box(geom, n, order, rs=RS_HLLC, avg=AVG_TRRS):
    """A walled box; hexahedra with a dyadic spacing (their normals are exact)."""
    if geom == HEX:
        mesh = M.hex_grid(*n, box=tuple((0.0, k / 16) for k in n), periodic=(False,) * 3)
    elif geom == QUAD:
        mesh = M.quad_grid(*n, 0, 1, 0, 0.7)
    else:
        mesh = M.tri_grid(*n, 0, 1, 0, 1, jitter=0.2, seed=3)
    return cases.Case("box", mesh, order, rs, avg, covolume=0.005,
                      bcs=[(a, BC_SLIP, None) for a in range(1, 7 if geom == HEX else 5)])


def pair(case, prec):
    ctx = Context(case.mesh, case.order, device=0, precision=prec)
    cases.configure_context(case, ctx)
    orc = Oracle(case.mesh, case.order)
    cases.configure_oracle(case, orc)
    return ctx, orc


def dev(a):
    return torch.tensor(a, dtype=torch.float64, device="cuda:0")


@pytest.mark.parametrize("prec", [FP64, FP32_BULK])
@pytest.mark.parametrize("geom,order,n", [
    (QUAD, 1, (1, 1)), (QUAD, 1, (3, 3)), (QUAD, 1, (33, 1)), (QUAD, 1, (67, 73)), (QUAD, 1, (141, 139)),
    (QUAD, 2, (1, 1)), (QUAD, 2, (4, 2)), (QUAD, 2, (67, 73)),
    (QUAD, 3, (1, 1)), (QUAD, 3, (5, 1)), (QUAD, 3, (43, 43)),
    (TRI, 1, (1, 1)), (TRI, 1, (3, 2)), (TRI, 1, (17, 1)), (TRI, 1, (70, 70)), (TRI, 1, (99, 99)),
    (TRI, 2, (1, 1)), (TRI, 2, (3, 1)), (TRI, 2, (50, 49)),
    (HEX, 1, (1, 1, 1)), (HEX, 1, (3, 1, 1)), (HEX, 1, (5, 5, 1)), (HEX, 1, (25, 1, 1)),
    (HEX, 2, (1, 1, 1)), (HEX, 2, (3, 1, 1)), (HEX, 2, (7, 1, 1)), (HEX, 2, (2, 2, 2)), (HEX, 2, (5, 4, 3))])
def test_rhs_tile_edges(cuda, geom, order, n, prec):
    case = box(geom, n, order, avg=AVG_TRRS if order == 1 else AVG_EINFELDT)
    ctx, orc = pair(case, prec)
    x = random_state(ctx.node_coords(), b=0.005, seed=31)
    y_ref, m_ref = orc.rhs(x)
    y = torch.empty(ctx.n, dtype=torch.float64, device="cuda")
    m = ctx.rhs(dev(x), y)
    assert rel_l1(y.cpu().numpy(), y_ref) < TOL[prec]
    assert abs(m - m_ref) <= (1e-13 if prec == FP64 else 1e-6) * m_ref
    xs_ref, _ = orc.step(x, 1e-4)
    xd = dev(x)
    ctx.step(xd, 1e-4)
    assert rel_l1(xd.cpu().numpy(), xs_ref) < TOL[prec]


@pytest.mark.parametrize("prec", [FP64, FP32_BULK])
@pytest.mark.parametrize("block", [0, 32, 256])
@pytest.mark.parametrize("geom,order,n,fun", [
    (QUAD, 1, (3, 3), FUN_MICHALAK), (QUAD, 2, (13, 5), FUN_BJ), (QUAD, 3, (13, 5), FUN_VENKATAKRISHNAN),
    (TRI, 1, (13, 5), FUN_VENKATAKRISHNAN), (TRI, 2, (9, 1), FUN_MICHALAK), (TRI, 2, (13, 5), FUN_BJ),
    (HEX, 1, (11, 3, 1), FUN_BJ), (HEX, 2, (5, 1, 1), FUN_VENKATAKRISHNAN), (HEX, 2, (11, 3, 1), FUN_MICHALAK)])
def test_limiter_team_edges(cuda, geom, order, n, fun, block, prec):
    case = box(geom, n, order)
    case.limiter = (LIM_MULTI, IND_BJ, fun, 1, 0)
    ctx, orc = pair(case, prec)
    if block:
        ctx.set_tuning(TUNE_LIMITER_BLOCK, block)
    x = random_state(ctx.node_coords(), b=0.005, seed=32)
    xd = dev(x)
    ctx.limit(xd)
    ref = orc.limit(x)
    assert rel_l1(ref, x) > 1e-3  # it limits
    assert rel_l1(xd.cpu().numpy(), ref) < TOL[prec]


@pytest.mark.parametrize("prec", [FP64, FP32_BULK])
@pytest.mark.parametrize("rs", [RS_HLL, RS_RUSANOV])
@pytest.mark.parametrize("geom,order,n", [(QUAD, 1, (19, 7)), (QUAD, 2, (19, 7)), (QUAD, 3, (5, 1)),
                                          (TRI, 1, (9, 7)), (TRI, 2, (9, 7)), (HEX, 1, (7, 5, 3)),
                                          (HEX, 2, (5, 4, 3))])
def test_face_speed_of_strong_jumps(cuda, geom, order, n, rs, prec):
    """The speed kernels skip a point whose FP32 estimate with its margin stays
    below the maximum so far: a constant state per element, orders of magnitude
    apart, the last element's far above the others (HLLC's
    signed speed of such jumps is an error, as it is for the reference)."""
    case = box(geom, n, order, rs=rs)
    ctx, orc = pair(case, prec)
    rng = np.random.default_rng(33)
    X = ctx.node_coords()
    dim, nd = X.shape
    ne = case.mesh.elem_vertices.shape[0]
    ndof = nd // ne
    cell = np.arange(nd) // ndof
    rho = 10.0 ** rng.uniform(-2, 1, ne)[cell]
    p = 10.0 ** rng.uniform(-2, 1, ne)[cell]
    p[cell == ne - 1] = 40.0
    vel = [0.3 * rng.uniform(-1, 1, ne)[cell] for _ in range(dim)]
    x = cases.conservative([rho, *vel, p], 1.4, 0.005)
    s_ref = orc.face_speed(x)
    assert abs(ctx.face_speed(dev(x)) - s_ref) <= (1e-12 if prec == FP64 else 1e-6) * s_ref


@pytest.mark.parametrize("limiter,indicator,fun", [(LIM_MULTI, IND_BJ, FUN_BJ), (LIM_MULTI, IND_BJ, FUN_MICHALAK),
                                                   (LIM_MULTI, IND_EVERYWHERE, FUN_BJ),
                                                   (LIM_FINDIFF, IND_BJ, FUN_VENKATAKRISHNAN)])
@pytest.mark.parametrize("geom,order,n", [(QUAD, 1, (1, 1)), (QUAD, 2, (11, 3)), (TRI, 1, (13, 5)), (TRI, 2, (17, 1)),
                                          (HEX, 1, (17, 1, 1)), (HEX, 2, (3, 3, 1))])
def test_limit_vjp_tile_edges(cuda, geom, order, n, limiter, indicator, fun):
    case = box(geom, n, order)
    case.limiter = (limiter, indicator, fun, 1, 0)
    ctx, _ = pair(case, FP64)
    x = random_state(ctx.node_coords(), b=0.005, seed=34, amp=0.1, vel=0.2)

    def apply(xx):
        y = dev(xx)
        ctx.limit(y)
        return y.cpu().numpy()

    def vjp(w):
        out = torch.empty(ctx.n, dtype=torch.float64, device="cuda")
        ctx.limit_vjp(dev(x), dev(w), out)
        return out.cpu().numpy()

    fd_check(apply, vjp, x, seed=3, eps=1e-7)


def test_float_pair_split_and_join_are_exact(cuda):
    """A step of length 0 with the one-stage scheme returns each value rounded to
    its float pair, hi = float(x) and lo = float(x - hi)."""
    case = box(QUAD, (33, 7), 1)
    ctx, _ = pair(case, FP32_BULK)
    ctx.set_tableau(1, [0.0], [1.0], [0.0])
    rng = np.random.default_rng(35)
    # elements orders of magnitude apart, each smooth enough to be physical at its faces
    scale = np.repeat(10.0 ** rng.uniform(-3, 3, ctx.n // 16), 4)
    x = random_state(ctx.node_coords(), seed=36, amp=0.05, vel=0.1) * np.tile(scale, 4)
    hi = x.astype(np.float32)
    want = hi.astype(np.float64) + (x - hi).astype(np.float32).astype(np.float64)
    xd = dev(x)
    ctx.step(xd, 0.0)
    assert np.array_equal(xd.cpu().numpy(), want)


@pytest.mark.parametrize("limited", [False, True])
def test_batch_fp32_q2_close_to_fp64(cuda, limited):
    """FP32 Q2 batches take the element pass: two steps against the FP64 batch
    (node pass), a smooth state; and the failed problem between them, whose
    state is non-physical, ends with finite values."""
    meshes = [M.quad_grid(n, 3, 2 * i, 2 * i + 1, 0, 0.7) for i, n in enumerate((5, 4, 33))]
    off = np.concatenate([[0], np.cumsum([m.num_elements for m in meshes])])
    case = box(QUAD, (2, 2), 2)
    if limited:
        case.limiter = (LIM_MULTI, IND_BJ, FUN_VENKATAKRISHNAN, 1, 0)
    case.mesh = cases.union_mesh(meshes)
    out = {}
    for prec in (FP64, FP32_BULK):
        ctx = Context(case.mesh, 2, device=0, precision=prec)
        cases.configure_context(case, ctx)
        ctx.batch_setup(off, [1.4] * 3, [0.005] * 3)
        x = random_state(ctx.node_coords(), b=0.005, seed=38, amp=0.01, vel=0.1).reshape(4, -1)
        x[3, 9 * off[1]:9 * off[2]] = 1e-3  # less than the kinetic energy
        xd = dev(x.ravel())
        info = ctx.batch_run(xd, 1e19, dt0=1e-3, dt_mode=2, max_steps=2, limit_initial=False)
        out[prec] = xd.cpu().numpy().reshape(4, -1)
        assert np.isfinite(out[prec]).all()
        assert list(info["steps"][[0, 2]]) == [2, 2] and info["steps"][1] < 0
    for cut in (slice(0, 9 * off[1]), slice(9 * off[2], None)):
        assert rel_l1(out[FP32_BULK][:, cut], out[FP64][:, cut]) < TOL[FP32_BULK]


def test_batch_larger_than_its_grid(cuda):
    """A batch whose CTAs loop over the active work, also when it starts in the
    middle of the lists: a small problem that ends after a few steps before a
    large one.  Each is bit-identical to the same problem run alone."""
    meshes = [M.quad_grid(20, 20, 0, 1, 0, 0.7), M.quad_grid(900, 700, 2, 3, 0, 0.7)]
    ne = [m.num_elements for m in meshes]
    case = box(QUAD, (2, 2), 1)
    case.limiter = (LIM_MULTI, IND_BJ, FUN_MICHALAK, 1, 0)
    case.mesh = cases.union_mesh(meshes)
    ctx = Context(case.mesh, 1, device=0, precision=FP64)
    cases.configure_context(case, ctx)
    ctx.batch_setup([0, ne[0], sum(ne)], [1.4, 1.4], [0.005, 0.005])
    x = random_state(ctx.node_coords(), b=0.005, seed=37, amp=0.05, vel=0.1)
    xd = dev(x)
    info = ctx.batch_run(xd, 5e-4, 0.3)
    assert 0 < info["steps"][0] < info["steps"][1]
    got = xd.cpu().numpy().reshape(4, -1)
    for p, cut in enumerate((slice(0, 4 * ne[0]), slice(4 * ne[0], None))):
        case.mesh = meshes[p]
        one = Context(case.mesh, 1, device=0, precision=FP64)
        cases.configure_context(case, one)
        xs = dev(np.ascontiguousarray(x.reshape(4, -1)[:, cut]).ravel())
        assert one.run(xs, 5e-4, 0.3)["steps"] == info["steps"][p]
        assert np.array_equal(got[:, cut], xs.cpu().numpy().reshape(4, -1))
