"""rkdg_riemann_batch of an FP32-bulk context returns the flux that its hexahedra,
Q1 and Q2 quads and hanging faces compute, to the bit."""
import ctypes as C

import numpy as np
import pytest
import torch

from rkdg3d_gb300 import mesh as M
from rkdg3d_gb300.solver import (AVG_EINFELDT, AVG_TRRS, FP32_BULK, Context, Physics, RiemannSolverHLL, RiemannSolverHLLC,
                                 RiemannSolverLLF, RiemannSolverRusanov)
from tests import device_math

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("avg", [AVG_TRRS, AVG_EINFELDT])
@pytest.mark.parametrize("rs", [0, 1, 2, 3])
@pytest.mark.parametrize("dim", [2, 3])
def test_pointwise_flux_is_the_elements(cuda, dim, rs, avg):
    lib = device_math.load()
    mesh = M.hex_grid(3, 3, 3) if dim == 3 else M.quad_grid(3, 3, 0, 1, 0, 1, periodic=(True, True))
    ctx = Context(mesh, 1, device=0, precision=FP32_BULK)
    solver = (RiemannSolverRusanov, RiemannSolverLLF, RiemannSolverHLL, RiemannSolverHLLC)[rs]
    ctx.set_physics(solver(avg), Physics(1.4, 0.005, 1.0))
    rng = np.random.default_rng(93)
    n = 20000
    nor = rng.normal(size=(n, dim))
    nor /= np.linalg.norm(nor, axis=1, keepdims=True)

    def state():
        rho, p = 10.0 ** rng.uniform(-1, 1, n), 10.0 ** rng.uniform(-1, 1, n)
        v = rng.normal(size=(n, dim))
        e = p * (1 - 0.005 * rho) / 0.4 + 0.5 * rho * (v * v).sum(1)
        return np.concatenate([rho[:, None], rho[:, None] * v, e[:, None]], 1)

    t = [torch.tensor(a, device="cuda") for a in (state(), state(), nor)]
    flux, sp = torch.zeros_like(t[0]), torch.zeros(n, dtype=torch.float64, device="cuda")
    f2, s2 = torch.zeros_like(flux), torch.zeros_like(sp)
    torch.cuda.synchronize()
    ctx.riemann_batch(*t, flux, sp)
    P = device_math.ptr
    assert lib.check_plain(dim, n, P(t[0]), P(t[1]), P(t[2]), P(f2), P(s2), C.c_float(1.4), C.c_float(0.005), rs, avg) == 0
    assert torch.equal(sp, s2) and torch.equal(flux, f2)
