"""The initial wave speed is the FP64 maximum over all face points, whatever its
kernels leave at their FP32 bound (rkdg_speed_bound.h): hexahedra whose z faces
are slightly tilted, gases with other TRRS powers, near ties, and HLLC's
negative speeds, which are errors.

On hexahedra against the team kernel, which evaluates every point in FP64 with
the same functions: 1e-14.  (The oracle takes the pressure from the rotated state; a
normal within 1e-3 of the z axis makes that rotation lose the more digits the
closer it is, 1e-7 at 1e-5.)  Planar elements against the oracle: 1e-12, the FP64
parity contract."""
import numpy as np
import pytest
import torch

from oracle.refcpu import Oracle, OracleError
from rkdg3d_gb300 import cases
from rkdg3d_gb300 import mesh as M
from rkdg3d_gb300.solver import (AVG_EINFELDT, AVG_TRRS, BC_SLIP, FP32_BULK, FP64, RS_HLL, RS_HLLC, RS_LLF, RS_RUSANOV,
                                 TUNE_HEX_KERNEL, Context, RkdgError)
from tests.helpers import random_state

pytestmark = pytest.mark.gpu


def pair(case, prec=FP64):
    ctx = Context(case.mesh, case.order, device=0, precision=prec)
    cases.configure_context(case, ctx)
    orc = Oracle(case.mesh, case.order)
    cases.configure_oracle(case, orc)
    return ctx, orc


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def all_points_speed(ctx, x):
    ctx.set_tuning(TUNE_HEX_KERNEL, 2)
    s = ctx.face_speed(dev(x))
    ctx.set_tuning(TUNE_HEX_KERNEL, 0)
    return s


def sheared(n, tilt):
    """An open box whose z faces' normals lean towards x by `tilt`; the boundary
    carries no integrator."""
    mesh = M.hex_grid(*n, periodic=(False,) * 3)
    mesh.elem_coords[..., 2] -= tilt * mesh.elem_coords[..., 0]
    return mesh


@pytest.mark.parametrize("order,n", [(1, (26, 26, 24)), (2, (20, 20, 20))])
@pytest.mark.parametrize("rs,avg", [(RS_HLL, AVG_EINFELDT), (RS_HLLC, AVG_EINFELDT), (RS_LLF, AVG_TRRS),
                                    (RS_RUSANOV, AVG_TRRS)])
@pytest.mark.parametrize("tilt", [1e-5, 1e-4, 2.4e-4, 1e-3])
def test_tilted_hexahedra(cuda, order, n, rs, avg, tilt):
    """A uniform flow along x and z: the z faces, the last in the list, carry
    the maximum, and only by what their tilt adds."""
    case = cases.Case("tilt", sheared(n, tilt), order, rs, avg)
    ctx, _ = pair(case)
    X = ctx.node_coords()
    w = 0.85
    a = w + 0.95 * tilt * w  # the x faces come just below
    one = np.ones(X.shape[1])
    x = cases.conservative([one, a * one, 0 * one, w * one, one / 1.4], 1.4, 0.0)
    s_ref = all_points_speed(ctx, x)
    assert abs(ctx.face_speed(dev(x)) - s_ref) <= 1e-14 * s_ref


@pytest.mark.parametrize("geom,order,n", [(M.GEOM_CUBE, 1, (26, 26, 24)), (M.GEOM_CUBE, 2, (20, 20, 20)),
                                          (M.GEOM_SQUARE, 1, (300, 200)), (M.GEOM_SQUARE, 3, (200, 150)),
                                          (M.GEOM_TRIANGLE, 1, (200, 150)), (M.GEOM_TRIANGLE, 2, (150, 120))])
@pytest.mark.parametrize("rs,avg", [(RS_LLF, AVG_TRRS), (RS_HLLC, AVG_TRRS), (RS_HLL, AVG_EINFELDT),
                                    (RS_RUSANOV, AVG_TRRS)])
@pytest.mark.parametrize("gamma", [1.05, 1.4, 5 / 3])
def test_near_ties(cuda, geom, order, n, rs, avg, gamma):
    """States that vary inside the elements, with a fluctuation near FP32
    rounding: the speeds of all points lie within a few 1e-6."""
    if geom == M.GEOM_CUBE:
        mesh = M.hex_grid(*n)
    elif geom == M.GEOM_SQUARE:
        mesh = M.quad_grid(*n, 0, 1, 0, 0.7)
    else:
        mesh = M.tri_grid(*n, 0, 1, 0, 1, jitter=0.2, seed=3)
    case = cases.Case("ties", mesh, order, rs, avg, gamma=gamma)
    ctx, orc = pair(case)
    rng = np.random.default_rng(41)
    X = ctx.node_coords()
    k = X.shape[1]
    for amp in (1e-6, 3e-5, 1e-2):
        f = lambda: 1 + amp * rng.uniform(-1, 1, k)
        x = cases.conservative([f(), *[0.3 * f() for _ in range(X.shape[0])], f()], gamma, 0.0)
        hexa = geom == M.GEOM_CUBE
        s_ref = all_points_speed(ctx, x) if hexa else orc.face_speed(x)
        assert abs(ctx.face_speed(dev(x)) - s_ref) <= (1e-14 if hexa else 1e-12) * s_ref


def test_negative_hllc_speed_is_an_error(cuda):
    """A flow against the z faces' normals a little faster than sound: HLLC's
    max(SL, SR) is negative there, by less than FP32 resolves, and the reference
    stops; the x and y faces, evaluated before, have ordinary speeds."""
    case = cases.Case("neg", sheared((26, 26, 24), 0.0), 1, RS_HLLC, AVG_EINFELDT)
    ctx, orc = pair(case)
    k = ctx.node_coords().shape[1]
    one = np.ones(k)
    for rho in (1.0, 0.7, 1.9):
        c = np.sqrt(1.4 / rho)
        for d in (1e-11, 1e-9, 3e-8, 1e-6):
            x = cases.conservative([rho * one, 0 * one, 0 * one, -c * (1 + d) * one, one], 1.4, 0.0)
            with pytest.raises(OracleError):
                orc.face_speed(x)
            with pytest.raises(RkdgError):
                ctx.face_speed(dev(x))


@pytest.mark.parametrize("prec", [FP64, FP32_BULK])
def test_first_step_of_a_batch_problem(cuda, prec):
    """Each problem's first time step follows from its own maximum."""
    meshes = [M.quad_grid(n, 7, 2 * i, 2 * i + 1, 0, 0.7) for i, n in enumerate((40, 33, 21))]
    off = np.concatenate([[0], np.cumsum([m.num_elements for m in meshes])])
    case = cases.Case("b", cases.union_mesh(meshes), 2, RS_HLL, AVG_TRRS, bcs=[(a, BC_SLIP, None) for a in range(1, 5)])
    ctx = Context(case.mesh, 2, device=0, precision=prec)
    cases.configure_context(case, ctx)
    ctx.batch_setup(off, [1.4, 1.1, 5 / 3], [0.0, 0.0, 0.005])
    x = random_state(ctx.node_coords(), seed=9, amp=0.02, vel=0.2).reshape(4, -1)
    info = ctx.batch_run(dev(x.ravel()), 0.5, 0.3, max_steps=1, limit_initial=False)
    for p, (g, b) in enumerate(((1.4, 0.0), (1.1, 0.0), (5 / 3, 0.005))):
        one = cases.Case("one", meshes[p], 2, RS_HLL, AVG_TRRS, gamma=g, covolume=b,
                         bcs=[(a, BC_SLIP, None) for a in range(1, 5)])
        c1, _ = pair(one, prec)
        i1 = c1.run(dev(x[:, 9 * off[p]:9 * off[p + 1]].ravel()), 0.5, 0.3, max_steps=1, limit_initial=False)
        assert info["sum_dt"][p] == i1["sum_dt"]
