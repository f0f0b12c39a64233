"""Performance cases: the calls a solver built on this package makes, over the
element types, orders, precisions and sizes it is used with.

A case is a dict of plain values:

  op        "run"      the time loop (``Context.run``), ``steps`` RK steps
            "step"     ``ExplicitRKLimitedSolver.Step``, ``steps`` times
            "mult"     one right-hand side (``FE_Evolution.Mult``)
            "limit"    one limiter pass (``Limiter.update``)
            "batch"    ``Context.batch_run`` over ``nprob`` strip problems
            "adjoint"  ``Context.adjoint_run`` over ``steps`` RK steps
  geom      2 triangles, 3 quadrilaterals, 5 hexahedra;  order: polynomial order
  nx ny nz  cells per direction (triangles: two per cell)
  rs avg    Riemann solver 0 Rusanov, 1 LLF, 2 HLL, 3 HLLC; wave speeds 0 TRRS, 1 Einfeldt
  fp32      FP32-bulk precision (else FP64)
  lim fun   limiter 0 none, 1 FinDiff, 2 Multi, both with the BJ-family
            indicator; fun 0 BJ, 1 Venkatakrishnan, 2 Michalak
  ic        "smooth" periodic waves, "shock" a jump across an oblique plane with
            waves on both sides, "mach10" the double-Mach-reflection states
  dynamic   a new CFL time step after every step (else fixed after the first)

Every pass starts from the state that ``prepare`` made (an ensemble restarted
from its initial field).  A program reads an FP32-bulk result as FP32 fields:
the mode evaluates its fluxes in FP32, so that is what the outputs carry.
"""
from __future__ import annotations

import itertools
import math

import numpy as np
import torch

from rkdg3d_gb300 import cases as C
from rkdg3d_gb300 import mesh as M
from rkdg3d_gb300 import solver as S

DEV = torch.device("cuda")
GAMMA = 1.4


def _case(name, op, geom, order, n, rs, avg, fp32, lim=0, fun=2, ic="smooth", steps=1, dynamic=False,
          nprob=0):
    nx, ny, nz = (tuple(n) + (1,))[:3]
    c = dict(op=op, geom=geom, order=order, nx=nx, ny=ny, nz=nz, rs=rs, avg=avg, fp32=fp32, lim=lim,
             fun=fun, ic=ic, steps=steps, dynamic=dynamic, nprob=nprob)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the acoustic pulse workload of the benchmark in the mixed mode: state far larger than L2
        _case("hex_q2_run_fp32", "run", 5, 2, (48, 48, 48), 0, 0, True, steps=4),
        # the same scheme in plain FP64, the precision of the reference
        _case("hex_q2_step_fp64", "step", 5, 2, (32, 32, 32), 0, 0, False, steps=1),
        # 3D channel with walls and open ends, order 1, shocks, limited, FP64, ragged sizes
        _case("hex_q1_limited_fp64", "run", 5, 1, (33, 27, 21), 3, 1, False, 2, 2, "shock", 3, True),
        # the same physics in the mixed mode on a larger mesh
        _case("hex_q1_limited_fp32", "run", 5, 1, (48, 45, 51), 2, 0, True, 2, 1, "shock", 4, True),
        # order 2 with the limiter in the mixed mode, ragged sizes
        _case("hex_q2_limited_fp32", "run", 5, 2, (31, 29, 23), 1, 1, True, 2, 2, "shock", 3),
        # the 200 x 4 shock tube: launches and latency, a time step read back after every step
        _case("tube_quad_q1_fp64", "run", 3, 1, (200, 4), 3, 1, False, 2, 0, "shock", 20, True),
        # the double Mach reflection mesh (524,288 triangles) with its limiter
        _case("dmr_tri_p1_fp32", "run", 2, 1, (1024, 256), 2, 0, True, 2, 1, "mach10", 4, True),
        # order-2 triangles in FP64 with the FinDiff limiter
        _case("tri_p2_limited_fp64", "run", 2, 2, (151, 101), 3, 1, False, 1, 2, "shock", 2, True),
        # a bare right-hand side, as a host-side time integrator calls it
        _case("quad_q2_mult_fp64", "mult", 3, 2, (301, 203), 3, 0, False, ic="smooth"),
        # the highest quad order in the mixed mode, no limiter
        _case("quad_q3_run_fp32", "run", 3, 3, (317, 211), 0, 0, True, steps=4),
        # a batch of uneven Riemann problems (perfect gas and covolume) in one graph launch
        _case("batch_q1_fp32", "batch", 3, 1, (1000, 4), 3, 1, True, 2, 2, "shock", 20, True, 64),
        # the discrete adjoint of limited steps
        _case("adjoint_hex_q1_fp64", "adjoint", 5, 1, (20, 20, 20), 3, 0, False, 2, 1, "smooth", 3),
    ]


def draw(rng):
    log = lambda a, b: math.exp(rng.uniform(math.log(a), math.log(b)))  # noqa: E731
    op = rng.choice(["run"] * 5 + ["step", "step", "mult", "limit", "batch", "adjoint"])
    geom, order = rng.choice([(5, 1), (5, 2), (5, 1), (5, 2), (3, 1), (3, 2), (3, 3), (2, 1), (2, 2)])
    fp32 = rng.random() < 0.5
    if op == "batch":
        geom, order = 3, rng.choice([1, 1, 2])
    if op in ("adjoint", "limit", "mult"):  # FP64 entry points; FP32-bulk is a mode of the steps
        fp32 = False
    lim = rng.choice([0, 0, 1, 2, 2]) if op != "limit" else rng.choice([1, 2])
    if op in ("mult",):
        lim = 0
    ic = rng.choice(["smooth", "shock"]) if lim else "smooth"
    if op == "adjoint":
        ic = "smooth"
    rs, avg = rng.choice([(0, 0), (1, 0), (1, 1), (2, 0), (2, 1), (3, 0), (3, 1)])
    # cells: up to the FP32 and FP64 sizes of the listed cases
    per = {(5, 1): 40, (5, 2): 135, (3, 1): 16, (3, 2): 36, (3, 3): 64, (2, 1): 24, (2, 2): 48}[geom, order]
    top = (8e6 if fp32 else 1.5e6) / per
    if op == "adjoint":
        top = 3e5 / per
    cells = int(log(60, top))
    nprob = 0
    if geom == 5:
        a, b = rng.uniform(0.6, 1.6), rng.uniform(0.6, 1.6)
        m = cells ** (1.0 / 3.0)
        n = (max(3, round(m * a)), max(3, round(m * b)), max(3, round(m / (a * b))))
    elif op == "batch":
        nprob = rng.randint(3, 64)
        n = (max(12, cells // (4 * nprob)), 4)
    else:
        a = log(0.25, 4.0)
        m = math.sqrt(cells)
        n = (max(3, round(m * a)), max(3, round(m / a)))
    steps = 1 if op in ("mult", "limit") else rng.randint(1, 3)
    if op == "batch":
        ic = "shock"
        steps = rng.randint(4, 16)
    return _case("", op, geom, order, n, rs, avg, fp32, lim, rng.randrange(3), ic, steps,
                 op in ("run", "batch") and rng.random() < 0.5, nprob)


# ---- inputs ------------------------------------------------------------------
def _mach10():
    """Pre- and post-shock states (rho, u, v, p) of the double Mach reflection."""
    rho1, p1, mach = 1.4, 1.0, 10.0
    ws = mach * math.sqrt(GAMMA * p1 / rho1)
    rho2 = rho1 * (GAMMA + 1) * mach ** 2 / ((GAMMA - 1) * mach ** 2 + 2)
    p2 = p1 * (2 * GAMMA * mach ** 2 - (GAMMA - 1)) / (GAMMA + 1)
    u2 = ws * (1.0 - rho1 / rho2)
    nx, ny = math.sin(math.pi / 3), -math.cos(math.pi / 3)
    return (rho1, 0.0, 0.0, p1), (rho2, u2 * nx, u2 * ny, p2), (nx, ny)


def _strips(case):
    """The batch's strip lengths (cells along x), uneven and the same for every seed."""
    rng = np.random.default_rng(case["nprob"] * 7919 + case["nx"])
    return [max(8, int(v)) for v in rng.uniform(0.1, 1.9, case["nprob"]) * case["nx"]]


def _mesh(case):
    """Mesh, boundary conditions (attribute, type, state), batch offsets."""
    nx, ny, nz, wall = case["nx"], case["ny"], case["nz"], case["ic"] != "smooth"
    if case["op"] == "batch":
        parts = [M.quad_grid(n, ny, 0.0, 1.0, 0.0, ny / n) for n in _strips(case)]
        off = np.concatenate([[0], np.cumsum([m.num_elements for m in parts])])
        return C.union_mesh(parts), [(1, S.BC_SLIP, None), (3, S.BC_SLIP, None), (2, S.BC_OPEN, None),
                                     (4, S.BC_OPEN, None)], off
    if case["geom"] == 5:
        m = M.hex_grid(nx, ny, nz, ((0.0, 1.0), (0.0, ny / nx), (0.0, nz / nx)), (not wall,) * 3)
        bcs = [(1, S.BC_SLIP, None), (6, S.BC_SLIP, None), (2, S.BC_SLIP, None), (4, S.BC_SLIP, None),
               (3, S.BC_OPEN, None), (5, S.BC_OPEN, None)]
    else:
        bcs = [(1, S.BC_SLIP, None), (3, S.BC_SLIP, None), (2, S.BC_OPEN, None), (4, S.BC_OPEN, None)]
        if case["geom"] == 3:
            m = M.quad_grid(nx, ny, 0.0, 1.0, 0.0, ny / nx, (not wall, not wall))
        else:
            m = M.tri_grid(nx, ny, 0.0, 1.0, 0.0, ny / nx, jitter=0.2, seed=0)
            if case["ic"] == "mach10":
                r, u, v, p = _mach10()[1]
                post = np.array([r, r * u, r * v, p / (GAMMA - 1) + 0.5 * r * (u * u + v * v)])
                bcs = [(1, S.BC_SLIP, None), (3, S.BC_OPEN, None), (2, S.BC_OPEN, None),
                       (4, S.BC_SUPERSONIC_INLET, post)]
    return m, bcs, None


def _initial(case, seed, X, prob, ext):
    """Conservative state [neq, ne, nd] at the nodes X [dim, ne, nd] (CUDA, FP64):
    random waves or jumps from the seed alone; prob: element -> problem, cov [ne]."""
    rng = np.random.default_rng(seed)
    dim = X.shape[0]
    dev = X.device
    tau = 2.0 * math.pi

    def waves(amp):
        f = torch.zeros_like(X[0])
        for _ in range(4):
            ph = rng.uniform(0, tau)
            for d in range(dim):
                ph = ph + tau * int(rng.integers(1, 4)) * X[d] / ext[d]
            f += amp * float(rng.uniform(0.3, 1.0)) * torch.sin(ph)
        return f

    if case["ic"] == "mach10":
        pre, post, n = _mach10()
        x0 = rng.uniform(0.1, 0.3)
        behind = n[0] * (X[0] - x0) + n[1] * X[1] < 0
        w = 1.0 + waves(0.004)
        prim = [torch.where(behind, torch.full_like(w, b), torch.full_like(w, a)) for a, b in zip(pre, post)]
        prim[0], prim[-1] = prim[0] * w, prim[-1] * w
    elif case["ic"] == "shock":
        npb = int(prob.max()) + 1 if prob is not None else 1
        rr = torch.from_numpy(rng.uniform(0.3, 1.0, (2, 2, npb))).to(dev)
        uu = torch.from_numpy(rng.uniform(-0.3, 0.3, (2, dim, npb))).to(dev)
        nrm = rng.normal(size=dim)
        nrm[0] = abs(nrm[0]) + 1.0
        if prob is not None:
            nrm[1:] = 0.0
        nrm /= np.linalg.norm(nrm)
        mid = torch.from_numpy(rng.uniform(0.4, 0.6, npb)).to(dev)
        pb = prob if prob is not None else torch.zeros(X.shape[1], dtype=torch.long, device=dev)
        s = sum(nrm[d] * (X[d] - ext[d] * (0.5 if d else 0.0)) for d in range(dim)) - (mid * nrm[0])[pb][:, None]
        left = s < 0
        pick = lambda a: torch.where(left, a[0][pb][:, None], a[1][pb][:, None])  # noqa: E731
        w = 1.0 + waves(0.004)
        prim = [pick(rr[:, 0]) * w] + [pick(uu[:, d]) for d in range(dim)] + [pick(rr[:, 1]) * w]
    else:
        rho = 1.0 + waves(0.01)
        prim = [rho] + [0.1 + waves(0.01) for _ in range(dim)] + [rho ** GAMMA]
    rho, vel, p = prim[0], prim[1:-1], prim[-1]
    cov = _cov(case, X.shape[1], prob, dev)
    E = p / (GAMMA - 1) * (1 - rho * cov[:, None]) + 0.5 * rho * sum(v * v for v in vel)
    return torch.stack([rho] + [rho * v for v in vel] + [E])


def _cov(case, ne, prob, dev):
    """Covolume per element: the second half of a batch's problems is a covolume gas."""
    cov = torch.zeros(ne, dtype=torch.float64, device=dev)
    if prob is not None:
        cov[prob >= case["nprob"] // 2] = 0.001
    return cov


def _prob(off, dev):
    if off is None:
        return None
    return torch.from_numpy(np.repeat(np.arange(len(off) - 1), np.diff(off))).to(dev)


def _node_coords(mesh, nodes, dev):
    """Physical node coordinates [dim, ne, nd] of affine elements."""
    X = torch.from_numpy(mesh.elem_coords).to(dev)
    cols = [1, 2] if mesh.geom == 2 else ([1, 3] if mesh.geom == 3 else [1, 3, 4])
    J = torch.stack([X[:, c] - X[:, 0] for c in cols], 2)
    xi = torch.from_numpy(nodes).to(dev)
    return (X[:, 0, :, None] + J @ xi.T).permute(1, 0, 2).contiguous(), J


def _ext(case):
    return [1.0, case["ny"] / case["nx"], case["nz"] / case["nx"]]


def _speed_bound(case):
    """A wave speed that the inputs stay below, for the cases with a given dt."""
    return 1.6 if case["ic"] == "smooth" else 3.0


def _fixed_dt(case):
    h = 1.0 / case["nx"] * (0.3 if case["geom"] == 2 else 1.0)
    return 0.2 * h / _speed_bound(case) / (2 * case["order"] + 1)


CFL = 0.2


def prepare(case, seed):
    dev = DEV
    mesh, bcs, off = _mesh(case)
    ctx = S.Context(mesh, case["order"], precision=S.FP32_BULK if case["fp32"] else S.FP64)
    stream = torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    rs = S.RiemannSolver(case["avg"])
    rs.code = case["rs"]
    ctx.set_physics(rs, S.Physics(GAMMA, 0.0, 1.0))
    ctx.set_solver_quirks(S.QUIRK_HLLC_NEGATIVE_SPEED_OK if case["rs"] == 3 else 0)
    for attr, kind, state in bcs:
        ctx.set_bc(attr, kind, state)
    ind = S.IndicatorBJ(case["fun"]) if case["lim"] else S.IndicatorNowhere()
    limiter = (S.LimiterMultiplier if case["lim"] == 2 else S.LimiterFinDiff)(ctx, ind)
    ctx.set_tableau(*S.TABLEAU_SSPRK3)
    prob = _prob(off, dev)
    if off is not None:
        npb = case["nprob"]
        ctx.batch_setup(off, np.full(npb, GAMMA), np.where(np.arange(npb) < npb // 2, 0.0, 0.001))
    X, _ = _node_coords(mesh, _Ref(case["geom"], case["order"]).nodes, dev)
    u = _initial(case, seed, X, prob, _ext(case)).reshape(-1).contiguous()
    st = dict(case=case, ctx=ctx, limiter=limiter, stream=stream, u0=u, u=u.clone())
    torch.cuda.synchronize()
    if case["lim"] and case["op"] != "limit" and off is None:
        limiter.update(u)  # a limited field, as every program starts from
    if case["op"] == "mult":
        st["evolution"], st["y"] = S.FE_Evolution(ctx), torch.empty_like(u)
    if case["op"] == "step":
        st["evolution"] = S.FE_Evolution(ctx)
        st["solver"] = S.ExplicitRKLimitedSolver(*S.TABLEAU_SSPRK3, limiter)
        st["solver"].Init(st["evolution"])
    if case["op"] == "adjoint":
        g = torch.Generator(device=dev)
        g.manual_seed(seed)
        st["bar0"] = torch.randn(u.shape, generator=g, device=dev, dtype=torch.float64)
        st["bar"], st["end"] = torch.empty_like(u), torch.empty_like(u)
    torch.cuda.synchronize()
    return st


def run(st):
    case, ctx, u = st["case"], st["ctx"], st["u"]
    num = np.float32 if case["fp32"] else float
    with torch.cuda.stream(st["stream"]):
        if case["op"] == "mult":
            speed = st["evolution"].Mult(st["u0"], st["y"])
            return {"y": st["y"], "speed": speed}
        u.copy_(st["u0"])
        if case["op"] == "limit":
            st["limiter"].update(u)
            return {"u": u}
        if case["op"] == "adjoint":
            st["bar"].copy_(st["bar0"])
            ctx.adjoint_run(u, case["steps"], _fixed_dt(case), 2, st["bar"], st["end"])
            return {"bar": st["bar"], "end": st["end"]}
        if case["op"] == "step":
            dt = _fixed_dt(case)
            for i in range(case["steps"]):
                last = st["solver"].Step(u, i * dt, dt)
        elif case["op"] == "batch":
            r = ctx.batch_run(u, 1e19, cfl=CFL, dt_mode=0 if case["dynamic"] else 1, max_steps=case["steps"])
            last = r["sum_dt"].astype(np.float32) if case["fp32"] else r["sum_dt"]
        else:
            r = ctx.run(u, 1e30, cfl=CFL, dt_mode=0 if case["dynamic"] else 1, max_steps=case["steps"])
            last = r["dt"]
        last = last if isinstance(last, np.ndarray) else num(last)
        return {"u": u.to(torch.float32) if case["fp32"] else u, "last": last}


# ---- what a pass cannot do without ---------------------------------------------
def work(case):
    geom, p = case["geom"], case["order"]
    dim, n1 = (3 if geom == 5 else 2), p + 1
    neq = dim + 2
    if geom == 2:
        ne, nd, nf, nq, nql = 2 * case["nx"] * case["ny"], n1 * (p + 2) // 2, 3, n1, 2
    elif geom == 3:
        cells = sum(_strips(case)) if case["op"] == "batch" else case["nx"]
        ne, nd, nf, nq, nql = cells * case["ny"], n1 ** 2, 4, n1, 2
    else:
        ne, nd, nf, nq, nql = case["nx"] * case["ny"] * case["nz"], n1 ** 3, 6, (p + 2) ** 2, 4
    n = ne * nd * neq
    # one sweep over an element: dense for triangles, sum-factorised for tensor elements
    vol = 2 * neq * dim * nd * (nd if geom == 2 else n1)
    if geom == 5:
        trace = 2 * neq * (n1 ** 3 + (p + 2) * n1 ** 2 + (p + 2) ** 2 * n1)
    else:
        trace = 2 * neq * (nq * nd if geom == 2 else n1 ** 2 + (0 if nq == n1 else nq * n1))
    rhs = nf * 2 * trace + nf / 2 * nq * (90 if case["rs"] == 0 else 150) + nd * (20 + 12 * dim) + 2 * vol
    lim = nf * nql * (2 * nd + 12) * (1 if case["lim"] == 2 else neq) + 4 * nd * neq
    stage = rhs + 8 * nd * neq + (lim if case["lim"] else 0)
    io = 8 + (4 if case["fp32"] else 8)
    if case["op"] == "mult":
        return {"bytes": n * io, "flops": ne * rhs}
    if case["op"] == "limit":
        return {"bytes": 16 * n, "flops": ne * lim}
    if case["op"] == "adjoint":  # forward, recomputation, and a reverse sweep of twice the forward work
        return {"bytes": 32 * n, "flops": case["steps"] * 3 * ne * stage * 4}
    return {"bytes": n * io, "flops": case["steps"] * 3 * ne * stage}


# ---- the same in plain torch, 64 bits --------------------------------------------
def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (x + 1), 0.5 * w


class _Ref:
    """Reference element: Lagrange basis on Gauss-Legendre nodes (triangles:
    the open barycentric nodes), and dense operators from exact rules."""

    VERTS = {2: [(0, 0), (1, 0), (0, 1)], 3: [(0, 0), (1, 0), (1, 1), (0, 1)],
             5: [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]}
    FACES = {2: [(0, 1), (1, 2), (2, 0)], 3: [(0, 1), (1, 2), (2, 3), (3, 0)],
             5: [(3, 2, 1, 0), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7), (4, 5, 6, 7)]}

    def __init__(self, geom, p):
        self.geom, self.p, self.dim = geom, p, 3 if geom == 5 else 2
        g, _ = _gauss(p + 1)
        if geom == 2:
            self.exps = [(a, b) for b in range(p + 1) for a in range(p + 1 - b)]
            nodes = []
            for j in range(p + 1):
                for i in range(p + 1 - j):
                    w = g[i] + g[j] + g[p - i - j]
                    nodes.append((g[i] / w, g[j] / w))
            self.nodes = np.array(nodes)
        else:
            self.nodes = np.array([t[::-1] for t in itertools.product(g, repeat=self.dim)])
            self.exps = list(t[::-1] for t in itertools.product(range(p + 1), repeat=self.dim))
        self.nd = len(self.nodes)
        self.coef = np.linalg.inv(self._mono(self.nodes))

    def _mono(self, x, d=None):
        cols = []
        for e in self.exps:
            v = np.ones(len(x))
            for k in range(self.dim):
                if k == d:
                    v = v * (e[k] * x[:, k] ** max(e[k] - 1, 0))
                else:
                    v = v * x[:, k] ** e[k]
            cols.append(v)
        return np.stack(cols, 1)

    def basis(self, x, d=None):
        return self._mono(np.asarray(x), d) @ self.coef

    def rule(self):
        g, w = _gauss(self.p + 2)
        if self.geom == 2:
            x = np.array([(a, b * (1 - a)) for a in g for b in g])
            return x, np.array([u * v * (1 - a) for a, u in zip(g, w) for v in w])
        x = np.array([t[::-1] for t in itertools.product(g, repeat=self.dim)])
        return x, np.array([np.prod(t) for t in itertools.product(w, repeat=self.dim)])

    def face_points(self, n):
        """Points [nf, nq, dim] of the n-point (per direction) Gauss rule on every face, weights."""
        g, w = _gauss(n)
        V = np.array(self.VERTS[self.geom], float)
        pts, out = list(itertools.product(g, repeat=self.dim - 1)), []
        for f in self.FACES[self.geom]:
            rows = []
            for t in pts:
                s = t[::-1]
                N = [1 - s[0], s[0]] if self.dim == 2 else [(1 - s[0]) * (1 - s[1]), s[0] * (1 - s[1]),
                                                            s[0] * s[1], (1 - s[0]) * s[1]]
                rows.append(sum(c * V[v] for c, v in zip(N, f)))
            out.append(rows)
        return np.array(out), np.array([np.prod(t) for t in itertools.product(w, repeat=self.dim - 1)])


class _Plain:
    """DG right-hand side, limiter and RK steps on an affine conforming mesh."""

    def __init__(self, case, mesh, bcs, prob):
        self.case, self.dev = case, DEV
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)  # noqa: E731
        r = self.r = _Ref(case["geom"], case["order"])
        self.dim, self.nd, self.neq = r.dim, r.nd, r.dim + 2
        ne = self.ne = mesh.num_elements
        self.X, J = _node_coords(mesh, r.nodes, self.dev)
        self.det = torch.linalg.det(J)
        self.Ji = torch.linalg.inv(J)
        JJ = J
        if case["geom"] == 2:
            A = torch.tensor([[1.0, -1 / math.sqrt(3)], [0.0, 2 / math.sqrt(3)]], dtype=J.dtype, device=self.dev)
            JJ = J @ A
        self.hmin = torch.linalg.svdvals(JJ).min(1).values
        x, w = r.rule()
        phi = r.basis(x)
        mass = phi.T @ (w[:, None] * phi)
        self.Minv = t(np.linalg.inv(mass))
        self.D = t(np.stack([np.einsum("q,qm,qj->jm", w, phi, r.basis(x, d)) for d in range(r.dim)]))
        self.wm = t((w @ phi) / w.sum())
        n = case["order"] + (2 if case["geom"] == 5 else 1)
        fp, self.fw = r.face_points(n)
        self.fw = t(self.fw)
        self.nq, nf = fp.shape[1], fp.shape[0]
        self.B = t(np.stack([r.basis(q) for q in fp]))                       # [nf, nq, nd]
        lp, _ = r.face_points(2)
        self.Bl = t(np.stack([r.basis(q) for q in lp]))
        self.Bv = t(r.basis(np.array(r.VERTS[case["geom"]], float)))
        # faces: pairs of element sides with the same vertices
        ev = mesh.elem_vertices
        nvf = len(r.FACES[case["geom"]][0])
        sides = np.stack([ev[:, list(f)] for f in r.FACES[case["geom"]]], 1).reshape(ne * nf, nvf)
        key = np.sort(sides, 1)
        order = np.lexsort(key.T[::-1])
        same = (key[order][1:] == key[order][:-1]).all(1)
        a, b = order[:-1][same], order[1:][same]
        a, b = np.minimum(a, b), np.maximum(a, b)
        nbr = np.full(ne * nf, -1)
        nbr[a], nbr[b] = b // nf, a // nf
        self.nbr = t(nbr.reshape(ne, nf))
        lone = np.ones(ne * nf, bool)
        lone[a] = lone[b] = False
        lone = np.nonzero(lone)[0]
        attr = {tuple(sorted(v)): c for v, c in zip(mesh.bdr_vertices.tolist(), mesh.bdr_attr.tolist())}
        kinds = {c: (k, s) for c, k, s in bcs}
        self.bnd = {}
        for c, (k, s) in kinds.items():
            idx = np.array([i for i in lone if attr.get(tuple(sorted(sides[i].tolist()))) == c], dtype=np.int64)
            if idx.size:
                self.bnd[c] = (k, s, t(idx))
        # side s of element e on local face f is row e * nf + f
        ec = t(mesh.elem_coords)
        fv = [list(f) for f in r.FACES[case["geom"]]]
        E = torch.stack([ec[:, f] for f in fv], 1)                            # [ne, nf, nvf, dim]
        if r.dim == 2:
            d = E[:, :, 1] - E[:, :, 0]
            nor = torch.stack([d[..., 1], -d[..., 0]], -1)
        else:
            nor = torch.linalg.cross(E[:, :, 1] - E[:, :, 0], E[:, :, 3] - E[:, :, 0])
        self.area = nor.norm(dim=-1).reshape(-1)
        self.nor = nor.reshape(-1, r.dim) / self.area[:, None]
        # point q of side a <-> point perm[q] of side b: positions about the face's middle
        P = torch.einsum("fqd,edc->efqc", t(fp), J.transpose(1, 2)).reshape(ne * nf, self.nq, r.dim)
        P = P - P.mean(1, keepdim=True)
        self.a, self.b = t(a), t(b)
        perm = torch.empty((len(a), self.nq), dtype=torch.long, device=self.dev)
        for i in range(0, len(a), 1 << 16):
            s = slice(i, i + (1 << 16))
            perm[s] = (P[self.a[s]][:, :, None] - P[self.b[s]][:, None]).square().sum(-1).argmin(2)
        self.perm = perm
        self.prob = prob
        self.cov_e = _cov(case, ne, prob, self.dev)

    # pointwise physics; s: [neq, ...], n: list of normal components, b: covolume
    def pressure(self, s, b):
        return (GAMMA - 1) * (s[-1] - 0.5 * (s[1:-1] ** 2).sum(0) / s[0]) / (1 - s[0] * b)

    def sound(self, s, p, b):
        return torch.sqrt(GAMMA * p / s[0] / (1 - s[0] * b))

    def normal_flux(self, s, n, p):
        un = sum(s[1 + d] * n[d] for d in range(self.dim)) / s[0]
        return torch.stack([un * s[0]] + [un * s[1 + d] + p * n[d] for d in range(self.dim)]
                           + [un * (s[-1] + p)]), un

    def riemann(self, s1, s2, n, b):
        p1, p2 = self.pressure(s1, b), self.pressure(s2, b)
        c1, c2 = self.sound(s1, p1, b), self.sound(s2, p2, b)
        f1, u1 = self.normal_flux(s1, n, p1)
        f2, u2 = self.normal_flux(s2, n, p2)
        rs = self.case["rs"]
        if rs == 0:
            e1 = (s1[1:-1] ** 2).sum(0).sqrt() / s1[0] + c1
            e2 = (s2[1:-1] ** 2).sum(0).sqrt() / s2[0] + c2
            m = torch.maximum(e1, e2)
            return 0.5 * (f1 + f2) - 0.5 * m * (s2 - s1), m
        if self.case["avg"] == 1:
            r1, r2 = s1[0].sqrt(), s2[0].sqrt()
            t = r1 + r2
            u = (u1 * r1 + u2 * r2) / t
            c = ((r1 * c1 ** 2 + r2 * c2 ** 2) / t + 0.5 * r1 * r2 / t ** 2 * (u2 - u1) ** 2).sqrt()
            SL, SR = u - c, u + c
        else:
            z = 0.5 * (GAMMA - 1) / GAMMA
            ps = ((c1 + c2 - 0.5 * (GAMMA - 1) * (u2 - u1)) / (c1 / p1 ** z + c2 / p2 ** z)) ** (1 / z)
            one = torch.ones_like(ps)
            q = lambda p: torch.where(ps > p, (1 + 0.5 * (GAMMA + 1) * (torch.maximum(ps / p, one) - 1) / GAMMA)  # noqa: E731
                                      .sqrt(), one)
            SL, SR = u1 - q(p1) * c1, u2 + q(p2) * c2
        m = torch.maximum(SL.abs(), SR.abs())
        if rs == 1:
            return 0.5 * (f1 + f2) - 0.5 * m * (s2 - s1), m
        if rs == 2:
            mid = (SR * f1 - SL * f2 + SL * SR * (s2 - s1)) / (SR - SL)
        else:
            k1, k2 = SL - u1, SR - u2
            ss = (p2 - p1 + s1[0] * u1 * k1 - s2[0] * u2 * k2) / (s1[0] * k1 - s2[0] * k2)
            left = ss > 0
            w = lambda x, y: torch.where(left, x, y)  # noqa: E731
            SK, sK, fK = w(SL, SR), w(s1, s2), w(f1, f2)
            ex = SK * (w(p1, p2) + sK[0] * w(k1, k2) * (ss - w(u1, u2)))
            D = torch.stack([torch.zeros_like(ss)] + [n[d] * torch.ones_like(ss) for d in range(self.dim)] + [ss])
            mid = (ss * (sK * SK - fK) + D * ex) / (SK - ss)
            m = torch.maximum(SL, SR)
        return torch.where(SL >= 0, f1, torch.where(SR <= 0, f2, mid)), m

    def rhs(self, u, faces_only=False):
        """Right-hand side [neq, ne, nd] and the wave speed per element."""
        neq, ne, nd, nf = self.neq, self.ne, self.nd, self.B.shape[0]
        tr = torch.einsum("fqj,kej->kefq", self.B, u).reshape(neq, ne * nf, self.nq)
        S = tr.shape[1:]
        speeds = torch.zeros(ne * nf, dtype=u.dtype, device=u.device)
        n = [self.nor[self.a, d][:, None] for d in range(self.dim)]
        s1 = tr[:, self.a]
        s2 = torch.gather(tr[:, self.b], 2, self.perm[None].expand(neq, -1, -1))
        b = self.cov_e[self.a // nf][:, None]
        F, m = self.riemann(s1, s2, n, b)
        w = self.fw * self.area[self.a][:, None] * F
        out = torch.zeros((neq,) + tuple(S), dtype=u.dtype, device=u.device)
        out = out.index_add(1, self.a, -w)
        back = torch.zeros_like(w).scatter(2, self.perm[None].expand(neq, -1, -1), w)
        out = out.index_add(1, self.b, back)
        m = m.detach().amax(1)
        speeds[self.a] = m
        speeds[self.b] = m
        for kind, state, idx in self.bnd.values():
            s1 = tr[:, idx]
            n = [self.nor[idx, d][:, None] for d in range(self.dim)]
            if kind == S_OPEN:
                s2 = s1
            elif kind == S_SLIP:
                mn = sum(s1[1 + d] * n[d] for d in range(self.dim))
                s2 = torch.stack([s1[0]] + [s1[1 + d] - 2 * mn * n[d] for d in range(self.dim)] + [s1[-1]])
            else:
                s2 = torch.from_numpy(state).to(u.device)[:, None, None].expand_as(s1)
            F, m = self.riemann(s1, s2, n, self.cov_e[idx // nf][:, None])
            out = out.index_add(1, idx, -self.fw * self.area[idx][:, None] * F)
            speeds[idx] = m.detach().amax(1)
        speed = speeds.reshape(ne, nf).amax(1)
        if faces_only:
            return None, speed
        z = torch.einsum("fqj,kefq->kej", self.B, out.reshape(neq, ne, nf, self.nq))
        b = self.cov_e[:, None]
        p = self.pressure(u, b)
        vel = u[1:-1] / u[0]
        node = (vel.square().sum(0).sqrt() + self.sound(u, p, b)).detach().amax(1)
        for r in range(self.dim):
            # contravariant component along r: det J sum_d (J^-1)[r, d] F_d
            g = self.Ji[:, r] * self.det[:, None]
            un = sum(g[:, d, None] * vel[d] for d in range(self.dim))
            G = torch.stack([un * u[0]] + [un * u[1 + d] + g[:, d, None] * p for d in range(self.dim)]
                            + [un * (u[-1] + p)])
            z = z + torch.einsum("jm,kem->kej", self.D[r], G)
        y = torch.einsum("ij,kej->kei", self.Minv, z) / self.det[:, None]
        return y, torch.maximum(speed, node)

    def limit(self, u):
        lim, fun = self.case["lim"], self.case["fun"]
        if not lim:
            return u
        um = u @ self.wm                                                       # [neq, ne]
        inner = self.nbr >= 0
        st = torch.cat([um[:, :, None], torch.where(inner, um[:, self.nbr.clamp(min=0)], um[:, :, None])], 2)
        lo, hi = st.amin(2)[:, :, None, None], st.amax(2)[:, :, None, None]
        if lim == 2:  # the density's indicator alone counts
            lo, hi = lo[:1], hi[:1]
        k = lo.shape[0]
        diff = torch.einsum("fqj,kej->kefq", self.Bl, u[:k]) - um[:k, :, None, None]
        safe = torch.where(diff.abs() > 1e-3, diff, torch.ones_like(diff))
        y = torch.where(diff > 1e-3, (hi - um[:k, :, None, None]) / safe,
                        torch.where(diff < -1e-3, (lo - um[:k, :, None, None]) / safe, torch.ones_like(diff)))
        if fun == 0:
            y = torch.clamp(y, max=1.0)
        elif fun == 1:
            y = (y * y + 2 * y) / (y * y + y + 2)
        else:
            y = torch.where(y < 1, y - 0.5 * (y / 1.5) ** 3, torch.ones_like(y))
        y = torch.where(inner[None, :, :, None], y, torch.full_like(y, 1e9))
        ind = y.reshape(k, self.ne, -1).amin(2)
        if fun == 0:
            ind = torch.clamp(ind, max=1.0)
        d = u - um[:, :, None]
        if lim == 1:
            return torch.where((ind[-1] < 0.999)[None, :, None], um[:, :, None].expand_as(u), u)
        v = um[:, :, None] + (ind[0] ** self.nd)[None, :, None] * d
        ver = torch.einsum("vj,kej->kev", self.Bv, v)
        bad = (ver[0] < 0) | (ver[-1] <= 0) | (self.pressure(ver, self.cov_e[:, None]) <= 0)
        return torch.where(bad.any(1)[None, :, None], um[:, :, None].expand_as(u), v)

    def step(self, u, dt):
        """SSP-RK3 in Butcher form, limited after every stage; dt per element."""
        dt = dt[None, :, None] if torch.is_tensor(dt) and dt.dim() else dt
        k0, _ = self.rhs(u)
        k1, _ = self.rhs(self.limit(u + dt * k0))
        k2, m = self.rhs(self.limit(u + dt * (0.25 * k0 + 0.25 * k1)))
        return self.limit(u + dt * (k0 / 6 + k1 / 6 + 2 * k2 / 3)), m

    def per_problem(self, v, how):
        if self.prob is None:
            return getattr(v, how)().expand(self.ne)
        out = torch.zeros(int(self.prob.max()) + 1, dtype=v.dtype, device=v.device)
        return out.scatter_reduce(0, self.prob, v, how, include_self=False)[self.prob]

    def run(self, u, steps, dynamic):
        u = self.limit(u)
        h = self.per_problem(self.hmin, "amin")
        den = 2 * self.case["order"] + 1
        dt = CFL * h / self.per_problem(self.rhs(u, True)[1], "amax") / den
        total = torch.zeros_like(dt)
        for _ in range(steps):
            total = total + dt
            u, m = self.step(u, dt)
            if dynamic:
                dt = CFL * h / self.per_problem(m, "amax") / den
        return u, dt, total


S_OPEN, S_SLIP = S.BC_OPEN, S.BC_SLIP


def exact(case, seed):
    mesh, bcs, off = _mesh(case)
    prob = _prob(off, DEV)
    d = _Plain(case, mesh, bcs, prob)
    u = _initial(case, seed, d.X, prob, _ext(case))
    flat = lambda v: v.reshape(-1)  # noqa: E731
    if case["op"] == "limit":
        return {"u": flat(d.limit(u))}
    if prob is None:
        u = d.limit(u)
    if case["op"] == "mult":
        y, m = d.rhs(u)
        return {"y": flat(y), "speed": float(m.max())}
    dt = _fixed_dt(case)
    if case["op"] == "adjoint":
        g = torch.Generator(device=u.device)
        g.manual_seed(seed)
        bar = torch.randn(u.numel(), generator=g, device=u.device, dtype=torch.float64).reshape(u.shape)
        states = [u]
        for _ in range(case["steps"]):
            states.append(d.step(states[-1], dt)[0])
        for x in reversed(states[:-1]):
            x = x.detach().requires_grad_(True)
            with torch.enable_grad():
                y = d.step(x, dt)[0]
                (bar,) = torch.autograd.grad(y, x, bar)
        return {"bar": flat(bar), "end": flat(states[-1])}
    if case["op"] == "step":
        for _ in range(case["steps"]):
            u, m = d.step(u, dt)
        return {"u": flat(u), "last": float(m.max())}
    u, dt, total = d.run(u, case["steps"], case["dynamic"])
    if prob is not None:
        first = torch.from_numpy(np.asarray(off[:-1])).to(u.device)
        return {"u": flat(u), "last": total[first]}
    return {"u": flat(u), "last": float(dt[0])}
