"""The work that this library's users have it do, as cases to be timed.

A case is a dict of plain values; `prepare` builds what a user's program holds
before the call (a mesh, a solver handle with its material, growth and
boundary conditions), `run` is one call sequence through the public interface
(`tissuefolding_paperversion_gb300.api`), host arrays in and out.

Kinds of cases:
  step      one implicit time step of one tissue (the whole of
            Simulation::updateStepNR) and its node positions: what a
            simulation does thousands of times
  sequence  the same step through the NewtonRaphsonSolver call sequence,
            driven by the host program
  batch     one time step of many independent tissues in one handle
  residual  K and g assembled at a state the caller gives, g read back
  adjoint   loss and gradients through a few steps, forward and backward
  packing   a step of two facing sheets with implicit packing
  static    the linear solve that allocates nothing, on the caller's matrix

A simulation goes on from step to step: `run` of a step case advances the
handle's tissue in time.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from tissuefolding_paperversion_gb300 import api, mesh

DEV = "cuda"
F64 = torch.float64
#: Degrees of freedom up to which `exact` solves its systems densely.
DENSE_DOFS = 9000


def listed():
    return [
        # the smallest call: a patch of tissue as in a quick parameter scan, where latency is all
        dict(name="step-patch-256", kind="step", nx=8, ny=8, layers=2, eta=0.0, material="uniform", growth="uniform"),
        # the small reference sheet: 1,600 prisms, elastic (CG, block-Jacobi)
        dict(name="step-small-1600", kind="step", nx=20, ny=20, layers=2, eta=0.0, material="uniform",
             growth="uniform"),
        # a viscous tissue of ordinary size through the solver's own call sequence (BiCGStab, block-Jacobi)
        dict(name="sequence-viscous-9k", kind="sequence", nx=31, ny=37, layers=4, eta=100.0, material="lognormal",
             growth="bump"),
        # an ordinary elastic tissue whose growth comes from growth functions, as a model file sets them (CG, multigrid)
        dict(name="step-functions-46k", kind="step", nx=83, ny=70, layers=4, eta=0.0, material="lognormal",
             growth="functions"),
        # the large viscous sheet: 320,000 prisms (BiCGStab, multigrid)
        dict(name="step-large-320k", kind="step", nx=200, ny=200, layers=4, eta=100.0, material="lognormal",
             growth="bump"),
        # the wing-disc-like sheet: about 1.0M prisms, elastic (CG, multigrid)
        dict(name="step-wing-1m", kind="step", shape="ellipse", nx=358, ny=224, layers=8, spacing=2.236, eta=0.0,
             material="layered", growth="bump", dt=120.0),
        # a parameter sweep: 32 tissues of uneven size in one handle
        dict(name="batch-32", kind="batch", n=32, min_prisms=1000, max_prisms=50000),
        # assembly for a caller with its own outer loop: elastic, an odd size
        dict(name="residual-elastic-97k", kind="residual", nx=127, ny=191, layers=2, eta=0.0, material="lognormal"),
        # the same on the large viscous sheet
        dict(name="residual-viscous-320k", kind="residual", nx=200, ny=200, layers=4, eta=100.0,
             material="lognormal"),
        # gradients for an inverse problem on a small sheet, every solve tight, order-fixed assembly
        dict(name="adjoint-3200", kind="adjoint", nx=20, ny=20, layers=4, eta=100.0, steps=6, every=3),
        # two surfaces pressed together
        dict(name="packing-28k", kind="packing", n=60, layers=2, eta=0.0),
        # a host that owns all device memory, with a matrix of its own
        dict(name="static-8405", kind="static", nx=41, ny=41, layers=5),
    ]


def draw(rng):
    """One more case of the ranges that the listed ones stand for."""
    def logu(a, b):
        return math.exp(rng.uniform(math.log(a), math.log(b)))

    def sheet(lo, hi, layers):
        cells = logu(lo, hi) / (2 * layers)
        aspect = rng.uniform(0.6, 1.6)
        nx = max(3, round(math.sqrt(cells * aspect)))
        return dict(nx=nx, ny=max(3, round(cells / nx)), layers=layers)

    kind = rng.choice(["step"] * 5 + ["sequence", "batch", "residual", "residual", "adjoint", "packing", "static"])
    layers = rng.choice([1, 2, 2, 3, 4, 4, 5, 8])
    eta = rng.choice([0.0, 100.0])
    if kind == "step":
        c = dict(kind=kind, **sheet(150, 300000, layers), eta=eta,
                 material=rng.choice(["uniform", "lognormal", "layered"]),
                 growth=rng.choice(["uniform", "bump", "bump", "functions"]),
                 shape=rng.choice(["rect", "rect", "ellipse"]))
        if rng.random() < 0.15:
            c["deterministic"] = True  # order-fixed assembly, for runs that have to be repeated bit by bit
        return c
    if kind == "sequence":
        return dict(kind=kind, **sheet(500, 60000, layers), eta=eta, material="lognormal", growth="bump")
    if kind == "batch":
        hi = logu(1500, 50000)
        return dict(kind=kind, n=rng.randint(2, 32), min_prisms=max(300, round(hi / logu(2, 50))),
                    max_prisms=round(hi))
    if kind == "residual":
        return dict(kind=kind, **sheet(300, 320000, layers), eta=eta, material="lognormal",
                    deterministic=rng.random() < 0.2)
    if kind == "adjoint":
        steps = rng.randint(2, 6)
        return dict(kind=kind, **sheet(300, 3200, rng.choice([2, 3, 4])), eta=eta, steps=steps,
                    every=rng.randint(1, steps))
    if kind == "packing":
        return dict(kind=kind, n=round(logu(6, 60)), layers=rng.choice([1, 2, 3]), eta=eta)
    n = logu(300, 16000)
    layers = rng.randint(2, 6)
    nx = max(3, round(math.sqrt(n / layers) * rng.uniform(0.7, 1.2)))
    return dict(kind=kind, nx=nx, ny=max(3, int(n / layers / nx)), layers=layers)


# ---- tissues -----------------------------------------------------------------------------


def _tissue(case, seed):
    """The sheet of a case: a jittered grid (or the part of it inside an
    ellipse) extruded into layers; basal nodes fixed in z, external viscosity
    on both surfaces."""
    rng = np.random.default_rng(seed)
    h = case.get("spacing", 5.0)
    nx, ny, layers = case["nx"], case["ny"], case["layers"]
    thick = (2.5 if h < 5.0 else 5.0) * layers
    if case.get("shape", "rect") == "ellipse" and min(nx, ny) >= 6:
        pos, conn, pl = mesh.ellipse_sheet(0.5 * nx * h, 0.5 * ny * h, h, layers, thick, 0.09 * h, rng)
    else:
        pos, conn, pl = mesh.rect_sheet(nx + 1, ny + 1, h, layers, thick, 0.1 * h, rng)
    ne, nn = conn.size // 6, pl.size
    fixed = np.zeros((nn, 3), dtype=np.uint8)
    fixed[pl == 0, 2] = 1
    ev = np.zeros((nn, 3))
    ev[pl != 2] = 10.0
    t = mesh.Tissue(pos=pos, conn=conn, fixed=fixed.reshape(-1), ext_visc=ev.reshape(-1), node_placement=pl,
                    E=np.full(ne, 1000.0), nu=np.full(ne, 0.3), eta=np.full(ne, float(case["eta"])),
                    rates=np.zeros(3 * ne), dt=float(case.get("dt", 60.0)))
    c = t.centroids()
    apical = c[:, 2] >= 0.5 * thick
    if case.get("material") == "lognormal":
        t.E = rng.lognormal(math.log(1000.0) - 0.045, 0.3, size=ne)
    elif case.get("material") == "layered":
        t.E = np.where(apical, 2000.0, 500.0)
    else:
        t.E = t.E * rng.uniform(0.98, 1.02, size=ne)
    lo, hi = c[:, :2].min(axis=0), c[:, :2].max(axis=0)
    centre = lo + rng.uniform(0.25, 0.75, size=2) * (hi - lo)
    width = rng.uniform(0.1, 0.25) * float((hi - lo).max())
    growth = case.get("growth", "bump")
    if growth == "uniform":
        g = (0.01 + 0.005 * apical) * rng.uniform(0.9, 1.1) / mesh.HOUR
    else:
        d2 = ((c[:, :2] - centre) ** 2).sum(axis=1)
        g = 0.02 / mesh.HOUR * np.exp(-d2 / (2.0 * width * width))
    rates = np.zeros((ne, 3))
    rates[:, 0] = rates[:, 1] = g
    t.rates = rates.reshape(-1)
    return t


def _solver(t, case, **kw):
    return api.Solver(t, deterministic=bool(case.get("deterministic", False)), **kw)


def _add_growth_functions(s, t, seed):
    """A uniform function in the apical half, a ring and a grid over the sheet."""
    p = t.pos.reshape(-1, 3)
    lo, hi = p.min(axis=0), p.max(axis=0)
    rates, angles = mesh.grid_growth_inputs(seed, 12, 9, scale=5e-6)
    s.add_uniform_growth([2e-6, 1e-6, 0.0], angle_rad=0.6, zmin=0.0, zmax=0.5)
    s.add_ring_growth((lo[:2] + hi[:2]) / 2, 0.1 * (hi[0] - lo[0]), 0.45 * (hi[0] - lo[0]), [4e-6, 4e-6, 0.0])
    s.add_grid_growth(rates, angles)


def _loss_params(t):
    xy = t.pos.reshape(-1, 3)
    c = 0.5 * (xy[:, :2].min(axis=0) + xy[:, :2].max(axis=0))
    return np.array([c[0], c[1], 5.0, 40.0])


def _static_system(case, seed):
    """A symmetric 3x3-block system on a grid of nx x ny x layers nodes coupled
    to their neighbours (27-point): springs of seeded stiffness and direction
    with a weak support at every node.  Rows, columns and blocks on the GPU."""
    rng = np.random.default_rng(seed)
    nx, ny, nl = case["nx"], case["ny"], case["layers"]
    ids = np.arange(nx * ny * nl).reshape(nl, ny, nx)
    src, dst, vec = [], [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                if (dz, dy, dx) <= (0, 0, 0):
                    continue
                a = ids[max(0, -dz):nl - max(0, dz), max(0, -dy):ny - max(0, dy), max(0, -dx):nx - max(0, dx)]
                b = ids[max(0, dz):nl - max(0, -dz), max(0, dy):ny - max(0, -dy), max(0, dx):nx - max(0, -dx)]
                src.append(a.reshape(-1))
                dst.append(b.reshape(-1))
                vec.append(np.tile([float(dx), float(dy), float(dz)], (a.size, 1)))
    src, dst, vec = np.concatenate(src), np.concatenate(dst), np.concatenate(vec)
    vec = vec + rng.uniform(-0.1, 0.1, size=vec.shape)
    vec /= np.linalg.norm(vec, axis=1, keepdims=True)
    k = rng.lognormal(0.0, 0.3, size=src.size)
    blk = k[:, None, None] * (vec[:, :, None] * vec[:, None, :] + 0.2 * np.eye(3))
    n = ids.size
    diag = np.zeros((n, 3, 3))
    np.add.at(diag, src, blk)
    np.add.at(diag, dst, blk)
    diag += 0.02 * np.eye(3)
    row = np.concatenate([src, dst, np.arange(n)])
    col = np.concatenate([dst, src, np.arange(n)])
    val = np.concatenate([-blk, -blk, diag])
    order = np.lexsort((col, row))
    row, col, val = row[order], col[order], val[order]
    rowptr = np.searchsorted(row, np.arange(n + 1)).astype(np.int32)
    to = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
    return n, to(rowptr), to(col.astype(np.int32)), to(val.reshape(-1)), to(rng.standard_normal(3 * n))


# ---- what is timed ---------------------------------------------------------------------------


def prepare(case, seed):
    kind = case["kind"]
    if kind == "static":
        n, rowptr, col, val, b = _static_system(case, seed)
        return dict(kind=kind, n=n, rowptr=rowptr, col=col, val=val, b=b, x=torch.empty_like(b), lib=api.load())
    if kind == "batch":
        # the sweep's meshes are the same for every seed, their stiffness and growth are not
        ts = [mesh.config_batch_instance(i, case["min_prisms"], case["max_prisms"]) for i in range(case["n"])]
        rng = np.random.default_rng(seed)
        for t in ts:
            t.E = t.E * rng.uniform(0.7, 1.4)
            t.rates = t.rates * rng.uniform(0.5, 1.0)
        s = api.Batch(ts)
        s.set_growth_rates()
        return dict(kind=kind, s=s, dt=ts[0].dt)
    if kind == "packing":
        t = mesh.config_facing_sheets(seed=seed, n=case["n"], n_layers=case["layers"], gap=1.5, E=100000.0,
                                      eta=case["eta"])
        s = _solver(t, case, krylov_rtol=1e-10)
        s.set_packing(True)
        rng = np.random.default_rng(seed + 1)
        starts = [t.pos + rng.uniform(-0.02, 0.02, size=t.pos.shape) for _ in range(4)]
        return dict(kind=kind, s=s, dt=t.dt, starts=starts, turn=0)
    t = _tissue(case, seed)
    if kind == "adjoint":
        s = api.Solver(t, newton_tol=1e-11, krylov_rtol=1e-13, deterministic=True)
        return dict(kind=kind, s=s, dt=t.dt, pos=t.pos, rate=t.rates.reshape(-1, 3)[:, 0].copy(), logE=np.log(t.E),
                    params=_loss_params(t), steps=case["steps"], every=case["every"])
    s = _solver(t, case)
    if kind == "residual":
        uk, un = mesh.perturbed_state(t, seed=seed + 1)
        s.set_Fg(mesh.growth_Fg(t, seed=seed + 2))
        s.set_positions(un)
        s.begin_step(t.dt)  # the viscosity surfaces of the step's start shape
        return dict(kind=kind, s=s, dt=t.dt, uk=uk, un=un)
    if case["growth"] == "functions":
        _add_growth_functions(s, t, seed)
    else:
        s.set_growth_rates(t.rates)
    return dict(kind=kind, s=s, dt=t.dt)


def run(state):
    kind, s = state["kind"], state.get("s")
    if kind == "step":
        s.newton_step(state["dt"])
        return {"positions": s.positions()}
    if kind == "sequence":
        s.begin_step(state["dt"])
        for _ in range(21):
            s.assemble()
            s.solve()
            if s.update()[0]:
                break
        s.end_step()
        return {"positions": s.positions()}
    if kind == "batch":
        s.step(state["dt"])
        return {"positions": s.positions()}
    if kind == "packing":
        s.set_positions(state["starts"][state["turn"] % len(state["starts"])])
        state["turn"] += 1
        s.newton_step(state["dt"])
        return {"positions": s.positions()}
    if kind == "residual":
        s.set_state(state["uk"], state["un"], state["dt"])
        s.assemble()
        return {"residual": s.residual()}
    if kind == "adjoint":
        s.set_positions(state["pos"])
        loss, saved = s.adjoint_forward(state["rate"], state["logE"], state["steps"], state["dt"], state["every"],
                                        state["params"])
        gr, ge = s.adjoint_backward(saved)
        saved.free()
        return {"loss": loss, "grad_rate": gr, "grad_logE": ge, "positions": s.positions()}
    p = lambda a: ctypes.c_void_p(a.data_ptr())  # noqa: E731
    it, rr = ctypes.c_int32(0), ctypes.c_double(0.0)
    st = state["lib"].tf_solve_bsr_static(state["n"], p(state["rowptr"]), p(state["col"]), p(state["val"]),
                                          p(state["b"]), p(state["x"]), 1e-12, 5000,
                                          ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
                                          ctypes.byref(it), ctypes.byref(rr))
    if st != api.TF_OK:
        raise RuntimeError("tf_solve_bsr_static: status %d" % st)
    return {"x": state["x"]}


def _sizes(case):
    """(prisms, nodes) of a case, on average over the seeds."""
    kind = case["kind"]
    if kind == "batch":
        lo, hi = case["min_prisms"], case["max_prisms"]
        ne = case["n"] * (hi - lo) / max(math.log(hi / lo), 1e-9)
        return ne, ne / 1.55
    if kind == "packing":
        n, layers = case["n"], case["layers"]
        return 4 * (n - 1) ** 2 * layers, 2 * n * n * (layers + 1)
    nx, ny, layers = case["nx"], case["ny"], case["layers"]
    part = math.pi / 4 if case.get("shape", "rect") == "ellipse" else 1.0
    return 2 * nx * ny * layers * part, (nx + 1) * (ny + 1) * (layers + 1) * part


def work(case):
    """One assembly reads a prism's connectivity, reference shape, growth
    tensor and material (324 B) and the node states, and writes g and the
    blocks of K (about 18 a node); its arithmetic is that of the 18 x 18
    tangent at six Gauss points.  A step assembles three times and reads K
    once more for each of its solves."""
    if case["kind"] == "static":
        n = case["nx"] * case["ny"] * case["layers"]
        return {"bytes": 27 * n * 76 + 48 * n, "flops": 2 * 9 * 27 * n}
    ne, nn = _sizes(case)
    visc = case.get("eta", 0.0) != 0.0
    k_bytes = 18 * 72 * nn
    a_bytes, a_flops = 324 * ne + 72 * nn + k_bytes, ne * (24000 if visc else 13000)
    if case["kind"] == "residual":
        return {"bytes": a_bytes, "flops": a_flops}
    times = 3
    if case["kind"] == "adjoint":
        steps = case["steps"]
        times = 3 * (2 * steps - math.ceil(steps / case["every"])) + steps
    return {"bytes": times * (a_bytes + k_bytes), "flops": times * (a_flops + 2 * 9 * 18 * nn)}


# ---- the same in plain torch, 64 bits ------------------------------------------------------------


class _Plain:
    """The implicit prism step in plain torch: g as a differentiable function
    of the shape, dense Newton and adjoint solves."""

    def __init__(self, t):
        to = lambda a: torch.as_tensor(np.asarray(a), device=DEV)  # noqa: E731
        self.t, self.dt, self.nn, self.ne = t, t.dt, t.n_nodes, t.n_elems
        self.conn = to(t.conn.reshape(-1, 6).astype(np.int64))
        self.pos0 = to(t.pos).to(F64)
        self.free = to(t.fixed.astype(np.float64) == 0.0).to(F64)
        self.ev = to(t.ext_visc).to(F64)
        self.eta = to(t.eta).to(F64)
        self.nu = to(np.clip(t.nu, 0.0, 0.5)).to(F64)
        self.logE = to(np.log(t.E)).to(F64)
        self.rates = to(t.rates.reshape(-1, 3)).to(F64)
        self.eye = torch.eye(3, dtype=F64, device=DEV)
        s = 1.0 / math.sqrt(3.0)
        dn = np.zeros((6, 3, 6))
        for q, (a, b, z) in enumerate([(1 / 6, 1 / 6, s), (2 / 3, 1 / 6, s), (1 / 6, 2 / 3, s),
                                       (1 / 6, 1 / 6, -s), (2 / 3, 1 / 6, -s), (1 / 6, 2 / 3, -s)]):
            lo, up, c = (1 - z) / 2, (1 + z) / 2, 1 - a - b
            dn[q] = [[-lo, lo, 0, -up, up, 0], [-lo, 0, lo, -up, 0, up],
                     [-c / 2, -a / 2, -b / 2, c / 2, a / 2, b / 2]]
        X = self.pos0.reshape(-1, 3)[self.conn]
        X = X - X[:, :1]
        D = to(dn).to(F64)
        M = torch.einsum("qja,eai->eqij", D, X)  # dX/dxi
        inv = torch.linalg.inv(M)
        self.gX = torch.einsum("eqjk,qja->eqak", inv, D)
        self.w = torch.linalg.det(M) / 6.0
        pl = np.asarray(t.node_placement)[t.conn.reshape(-1, 6)]
        self.faces = torch.cat([self.conn[to((pl == 1).any(axis=1))][:, 3:], self.conn[to((pl == 0).any(axis=1))][:, :3]])

    def areas(self, u):
        """Viscosity surface of every node on the shape u."""
        x = u.reshape(-1, 3)[self.faces]
        n = torch.linalg.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0])
        a = 0.5 * torch.linalg.norm(n, dim=1)
        out = torch.zeros(self.nn, dtype=F64, device=DEV)
        for k in range(3):
            out = out.index_add(0, self.faces[:, k], a / 3.0)
        return out

    def forces(self, x, x0, Fg, logE, eta, nu, gX, w):
        """Nodal forces (e, 6, 3) of elements with node positions x now and x0 at the step's start."""
        E = torch.exp(logE)
        lam = (E * nu / (1 + nu) / (1 - 2 * nu))[..., None]
        mu = (E / 2.0 / (1 + nu))[..., None]
        r = x - x[..., :1, :]
        F = torch.einsum("...ai,...qaj->...qij", r, gX)
        Fe = F @ torch.linalg.inv(Fg)[..., None, :, :]
        det = lambda m: (m[..., 0, :] * torch.linalg.cross(m[..., 1, :], m[..., 2, :])).sum(-1)  # noqa: E731
        J, dF = det(Fe), det(F)
        cols = torch.stack([torch.linalg.cross(F[..., :, 1], F[..., :, 2]), torch.linalg.cross(F[..., :, 2], F[..., :, 0]),
                            torch.linalg.cross(F[..., :, 0], F[..., :, 1])], dim=-1)  # cofactors
        dn = torch.einsum("...qik,...qak->...qai", cols, gX) / dF[..., None, None]
        b = Fe @ Fe.transpose(-1, -2)
        sig = (mu[..., None, None] * (b - self.eye) + (lam * torch.log(J))[..., None, None] * self.eye) / J[..., None, None]
        v = (x - x0) / self.dt
        L = torch.einsum("...ai,...qaj->...qij", v - v[..., :1, :], dn)
        sig = sig + 0.5 * eta[..., None, None, None] * (L + L.transpose(-1, -2))
        return -torch.einsum("...q,...qij,...qaj->...ai", w * dF, sig, dn)

    def g(self, u, un, Fg, logE, area):
        x, x0 = u.reshape(-1, 3)[self.conn], un.reshape(-1, 3)[self.conn]
        f = self.forces(x, x0, Fg, logE, self.eta, self.nu, self.gX, self.w)
        out = -(area[:, None] * self.ev.reshape(-1, 3)) * (u - un).reshape(-1, 3) / self.dt
        return out.index_add(0, self.conn.reshape(-1), f.reshape(-1, 3)).reshape(-1) * self.free

    def jacobian(self, u, un, Fg, logE, area):
        """-dg/du, dense, unit rows and columns at fixed DOFs."""
        x, x0 = u.reshape(-1, 3)[self.conn], un.reshape(-1, 3)[self.conn]
        jac = torch.func.vmap(torch.func.jacfwd(self.forces), chunk_size=4096)
        K = -jac(x, x0, Fg, logE, self.eta, self.nu, self.gX, self.w).reshape(-1, 18, 18)
        dof = (3 * self.conn[:, :, None] + torch.arange(3, device=DEV)).reshape(-1, 18)
        n = 3 * self.nn
        A = torch.zeros(n * n, dtype=F64, device=DEV)
        A.index_add_(0, (dof[:, :, None] * n + dof[:, None, :]).reshape(-1), K.reshape(-1))
        A = A.view(n, n)
        A.diagonal().add_(area.repeat_interleave(3) * self.ev / self.dt)
        A.mul_(self.free[:, None]).mul_(self.free[None, :])
        A.diagonal().add_(1.0 - self.free)
        return A

    def step(self, un, Fg, logE):
        """The converged end shape of one step, to the rounding of g."""
        area, u, last = self.areas(un), un.clone(), math.inf
        for _ in range(25):
            du = torch.linalg.solve(self.jacobian(u, un, Fg, logE, area), self.g(u, un, Fg, logE, area))
            u = u + du
            size = float(du.norm())
            if size < 1e-11 or (size < 1e-7 and size > 0.3 * last):
                break
            last = size
        return u

    def grown(self, k):
        return torch.diag_embed(torch.exp(self.rates * (self.dt * k)))


def _exact_adjoint(case, seed):
    t = _tissue(case, seed)
    p = _Plain(t)
    N = case["steps"]
    rate = p.rates[:, 0].clone()
    us = [p.pos0]
    for n in range(1, N + 1):
        us.append(p.step(us[-1], p.grown(n), p.logE))
    cx, cy, amp, wid = (float(v) for v in _loss_params(t))
    apical = torch.as_tensor(t.node_placement == 1, device=DEV)

    def loss(u):
        x = u.reshape(-1, 3)[apical]
        return ((x[:, 2] - amp * torch.exp(-((x[:, 0] - cx) ** 2 + (x[:, 1] - cy) ** 2) / (2 * wid * wid))) ** 2).sum()

    uN = us[N].clone().requires_grad_(True)
    val = loss(uN)
    (bar,) = torch.autograd.grad(val, uN)
    gr, ge = torch.zeros(p.ne, dtype=F64, device=DEV), torch.zeros(p.ne, dtype=F64, device=DEV)
    for n in range(N, 0, -1):
        r, e, prev = (v.clone().requires_grad_(True) for v in (rate, p.logE, us[n - 1]))
        rr = torch.stack([r, r, torch.zeros_like(r)], dim=1)
        Fg = torch.diag_embed(torch.exp(rr * (p.dt * n)))
        with torch.no_grad():
            A = p.jacobian(us[n], us[n - 1], Fg.detach(), p.logE, p.areas(us[n - 1]))
            lam = torch.linalg.solve(A.T, bar * p.free)
            del A
        dr, de, dp = torch.autograd.grad((p.g(us[n], prev, Fg, e, p.areas(prev)) * lam).sum(), (r, e, prev))
        gr, ge, bar = gr + dr, ge + de, dp
    return {"loss": float(val), "grad_rate": gr, "grad_logE": ge, "positions": us[N]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "static":
        n, rowptr, col, val, b = _static_system(case, seed)
        A = torch.sparse_bsr_tensor(rowptr.long(), col.long(), val.view(-1, 3, 3), size=(3 * n, 3 * n), dtype=F64)
        A = A.to_sparse_coo().to_sparse_csr()
        x = torch.zeros_like(b)
        r = b.clone()
        q, rho = r.clone(), r @ r
        stop = 1e-32 * float(rho)
        for _ in range(20000):
            Aq = A @ q
            alpha = rho / (q @ Aq)
            x, r = x + alpha * q, r - alpha * Aq
            new = r @ r
            q, rho = r + (new / rho) * q, new
            if float(rho) < stop:
                break
        return {"x": x}
    if kind in ("batch", "packing"):
        return None
    if kind == "residual":
        t = _tissue(case, seed)
        p = _Plain(t)
        uk, un = (torch.as_tensor(v, device=DEV) for v in mesh.perturbed_state(t, seed=seed + 1))
        Fg = torch.as_tensor(mesh.growth_Fg(t, seed=seed + 2), device=DEV).reshape(-1, 3, 3)
        return {"residual": p.g(uk, un, Fg, p.logE, p.areas(un))}
    if 3 * _sizes(case)[1] > DENSE_DOFS:
        return None
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    if case["growth"] == "functions":
        return None
    p = _Plain(_tissue(case, seed))
    return {"positions": p.step(p.pos0, p.grown(1), p.logE)}
