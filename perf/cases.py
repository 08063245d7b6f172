"""The work that users of this framework have it do, as timed cases over its public entry points.

Kinds of case (``case["kind"]``):
  energy   one evaluation of the incremental potential and its gradient at a new displacement, as an external
           optimiser drives it (update_energy_and_gradients): tets or a mass-spring sheet
  hessian  the SPD-projected Hessian assembled at a new displacement and applied to a vector, as an external
           Krylov or eigen solver drives it (update_hessian + spmv)
  step     one whole backward-Euler Newton step from a given state (prepare, solve, next): the simulation loop
  lbfgs    one whole step of the L-BFGS stepper with a fixed budget of iterations a frame, as interactive
           programs run it
  adjoint  the reverse pass of one step, as a differentiable rollout runs it once per step (adjoint_step)

Solver settings are the benchmark's (inexact Newton, block-Jacobi PCG); a step is solved to the residual ``tol``,
the benchmark's 1e-6 in full precision, 1e-7 for large mixed-precision scenes (where their results carry FP32
accuracy) and the tests' 1e-8 for small bodies.  States live on the GPU: a pass writes its state into the
handle's own buffers (device_ptr, as a torch tensor), calls the entry point and returns the handle's buffers.  A
mixed-precision handle's results carry FP32 accuracy; its user keeps them as float32.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ssim_gb300 as sg
from ssim_gb300 import adjoint as sg_adjoint
from ssim_gb300 import mesh, scenes

SOLVER = dict(stop_mode=1, cg_forcing=1, cg_rtol=1e-1, cg_eta_min=5e-2, cg_max_iters=5000,
              max_newton_iters=100, precond=2, cg_check_every=16)
NU, RHO, DT = 0.45, 1000.0, 1e-2
GRAVITY = (0.0, 0.0, -9.8)


def listed():
    return [
        # the plain 6,000-tet cube: the smallest evaluation, where a launch and a host wait count
        {"name": "energy_box_small", "kind": "energy", "scene": "box", "precision": "fp64", "nx": 10, "ny": 10, "nz": 10},
        # the same evaluation on the million-tet beam
        {"name": "energy_beam_1m", "kind": "energy", "scene": "box", "precision": "fp64", "nx": 100, "ny": 50, "nz": 34},
        # the mass-spring sheet of 512 x 512 vertices (1.57M springs)
        {"name": "energy_cloth_512", "kind": "energy", "scene": "cloth", "precision": "fp64", "nx": 512},
        # a Hessian for an external solver, the 192,000-tet bar
        {"name": "hessian_bar_mixed", "kind": "hessian", "scene": "box", "precision": "mixed", "nx": 80, "ny": 20, "nz": 20},
        # ... and in full precision on a ragged box
        {"name": "hessian_box_fp64", "kind": "hessian", "scene": "box", "precision": "fp64", "nx": 23, "ny": 17, "nz": 13},
        # the plain FP64 cube stepped: small systems, every launch and wait of the Newton loop counts
        {"name": "step_box_fp64", "kind": "step", "scene": "box", "precision": "fp64", "nx": 10, "ny": 10, "nz": 10, "tol": 1e-8},
        # the bar stepped in full precision, odd sizes
        {"name": "step_bar_fp64", "kind": "step", "scene": "box", "precision": "fp64", "nx": 57, "ny": 19, "nz": 13, "tol": 1e-6},
        # the 192,000-tet bar in mixed precision
        {"name": "step_bar_mixed", "kind": "step", "scene": "box", "precision": "mixed", "nx": 80, "ny": 20, "nz": 20, "tol": 1e-7},
        # the headline: the 1.02M-tet beam in mixed precision
        {"name": "step_beam_mixed", "kind": "step", "scene": "box", "precision": "mixed", "nx": 100, "ny": 50, "nz": 34, "tol": 1e-7},
        # many independent bodies in one handle, each with its own stopping test
        {"name": "step_batch_mixed", "kind": "step", "scene": "batch", "precision": "mixed", "n": 64, "kmin": 4, "kmax": 24, "tol": 1e-8},
        # L-BFGS, a fixed number of iterations a frame
        {"name": "lbfgs_bar_fp64", "kind": "lbfgs", "scene": "box", "precision": "fp64", "nx": 40, "ny": 14, "nz": 14, "iters": 20},
        # the reverse pass of the differentiable rollout's cube
        {"name": "adjoint_cube_fp64", "kind": "adjoint", "scene": "box", "precision": "fp64", "nx": 24, "ny": 24, "nz": 24},
    ]


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    def box(most):
        # hex counts a side of an elongated box of 6 tets a hex; the sizes come out odd and even alike
        hexes = log_int(500, most)
        ratio, squash = rng.uniform(1.0, 4.0), rng.uniform(0.7, 1.4)
        side = (hexes / ratio) ** (1.0 / 3.0)
        nx, ny, nz = (max(3, int(v)) for v in (side * ratio, side * squash, side / squash))
        return {"scene": "box", "nx": nx, "ny": ny, "nz": nz}

    kind = rng.choice(["energy", "energy", "energy_cloth", "hessian", "hessian", "step_fp64", "step_fp64", "step_mixed",
                       "step_mixed", "step_mixed", "batch", "lbfgs", "adjoint"])
    if kind == "energy":
        return {"kind": "energy", "precision": "fp64", **box(165000)}
    if kind == "energy_cloth":
        return {"kind": "energy", "precision": "fp64", "scene": "cloth", "nx": log_int(40, 500)}
    if kind == "hessian":
        p = rng.choice(["fp64", "mixed"])
        return {"kind": "hessian", "precision": p, **box(30000)}
    if kind == "step_fp64":
        return {"kind": "step", "precision": "fp64", "tol": rng.choice([1e-6, 1e-8]), **box(14000)}
    if kind == "step_mixed":
        b = box(165000)
        return {"kind": "step", "precision": "mixed", **b, "tol": 1e-8 if b["nx"] * b["ny"] * b["nz"] < 20000 else 1e-7}
    if kind == "batch":
        return {"kind": "step", "scene": "batch", "precision": "mixed", "tol": 1e-8, "n": log_int(6, 60), "kmin": rng.randint(3, 6),
                "kmax": rng.randint(12, 24)}
    if kind == "lbfgs":
        return {"kind": "lbfgs", "precision": "fp64", **box(16000), "iters": rng.randint(8, 20)}
    return {"kind": "adjoint", "precision": "fp64", **box(13000)}


# ---------------------------------------------------------------- scenes
def _smooth(X, gen, amplitude, ramp):
    """A smooth random vector field on the points X [V, 3]: a few sine modes, zero where ramp is zero."""
    lo, hi = X.min(0).values, X.max(0).values
    Y = (X - lo) / torch.clamp((hi - lo).max(), min=1e-12)
    out = torch.zeros_like(X)
    for _ in range(4):
        k = math.pi * (1.0 + 2.0 * torch.rand(3, 3, generator=gen, dtype=torch.float64))
        ph = 2 * math.pi * torch.rand(3, generator=gen, dtype=torch.float64)
        a = torch.randn(3, generator=gen, dtype=torch.float64)
        out += (a.to(X.device) * torch.sin(Y @ k.to(X.device).T + ph.to(X.device)))
    return amplitude * 0.5 * out * ramp[:, None]


def _scene(case, seed):
    """Mesh, material, Dirichlet set and start state of a case (numpy / torch, host and GPU)."""
    gen = torch.Generator().manual_seed(1000003 + int(seed))
    rng = np.random.default_rng(77 + int(seed))
    s = {}
    if case["scene"] == "box":
        h = 0.02
        n = (case["nx"], case["ny"], case["nz"])
        X, T = mesh.kuhn_box(n, tuple(h * k for k in n))
        X = mesh.jitter_interior(X, 0.1 * h, 11 + int(seed))
        s.update(X=X, cells=T, E=10.0 ** rng.uniform(4.0, 6.0, T.shape[0]), nu=None, fixed=np.where(X[:, 0] == 0.0)[0],
                 size=h * max(n), offsets=None)
    elif case["scene"] == "batch":
        b = scenes.batch_cubes(case["n"], case["kmin"], case["kmax"], seed=4)
        E = 10.0 ** rng.uniform(4.0, 6.0, case["n"])
        tets = 6 * b["k"].astype(np.int64) ** 3
        s.update(X=b["X"], cells=b["cells"], E=np.repeat(E, tets), nu=b["nu_cells"], fixed=b["fixed"], size=1.0,
                 offsets=b["vertex_offsets"])
    else:
        c = scenes.cloth(case["nx"])
        s.update(X=c["X"], cells=c["cells"], fixed=c["fixed"], size=float(c["X"].max()), k=c["k"], offsets=None,
                 vertex_mass=c["vertex_mass"])
    dev = torch.device("cuda")
    Xd = torch.from_numpy(s["X"]).to(dev)
    mask = torch.ones(Xd.shape[0], dtype=torch.float64, device=dev)
    mask[torch.from_numpy(np.ascontiguousarray(s["fixed"])).to(dev)] = 0.0
    if case["scene"] == "box":
        ramp = torch.clamp(Xd[:, 0] / (0.5 * Xd[:, 0].max()), max=1.0)
    elif case["scene"] == "batch":
        ramp = torch.clamp(Xd[:, 2] / 0.5, max=1.0)
    else:
        ramp = mask
    s["Xd"], s["free"] = Xd, mask
    s["u"] = _smooth(Xd, gen, 0.003 * s["size"], ramp)
    s["v"] = _smooth(Xd, gen, 0.3, ramp)
    s["xt"] = (s["u"] + DT * s["v"] + DT * DT * torch.tensor(GRAVITY, dtype=torch.float64, device=dev)) * mask[:, None]
    s["gen"] = gen
    return s


class _Buffer:
    """A [V, 3] float64 device buffer of a handle, for torch's zero-copy view; the view keeps the handle alive."""

    def __init__(self, ts, field):
        self.ts = ts
        self.__cuda_array_interface__ = {"shape": (ts.num_vertices, 3), "typestr": "<f8", "version": 3,
                                         "data": (ts.device_ptr(field), False)}


def _view(ts, field):
    return torch.as_tensor(_Buffer(ts, field), device="cuda")


def prepare(case, seed):
    s = _scene(case, seed)
    kind = case["kind"]
    stream = torch.cuda.Stream()
    params = sg.default_params(**SOLVER)
    params.rel_tol = case.get("tol", 1e-6)
    if kind == "lbfgs":
        params.max_lbfgs_iters = case["iters"]
    if kind == "adjoint":
        eng = sg_adjoint.RolloutEngine(s["X"], s["cells"], s["fixed"], dt=DT, nu=NU, rho=RHO, gravity=GRAVITY,
                                       precision=case["precision"], params=params)
        eng.ts.set_stream(stream.cuda_stream)
        eng.start(torch.from_numpy(s["E"]), s["v"])
        g = s["gen"]
        st = {"kind": kind, "stream": stream, "ts": eng.ts, "eng": eng, "u1": s["u"],
              "ubar": torch.randn(s["X"].shape, generator=g, dtype=torch.float64).cuda(),
              "vbar": 1e-2 * torch.randn(s["X"].shape, generator=g, dtype=torch.float64).cuda()}
        torch.cuda.synchronize()
        return st
    if case["scene"] == "cloth":
        ts = sg.TimeStep.springs(s["X"], s["cells"], s["k"], vertex_mass=s["vertex_mass"], time_step=DT)
    else:
        ts = sg.TimeStep(s["X"], s["cells"], DT, 1e5, NU, RHO)
    ts.set_precision(case["precision"])
    if case["scene"] != "cloth":
        ts.set_material(s["E"], s["nu"])
    ts.mark_dirichlet_batched(s["fixed"], np.zeros((len(s["fixed"]), 3)))
    ts.add_gravity(GRAVITY)
    if s["offsets"] is not None:
        ts.set_instances(s["offsets"])
    ts.set_params(params)
    ts.reset({"step": "newton", "lbfgs": "lbfgs"}.get(kind, "none"))
    ts.set_stream(stream.cuda_stream)
    st = {"kind": kind, "stream": stream, "ts": ts, "u": s["u"], "v": s["v"], "mixed": case["precision"] == "mixed",
          "deformation": _view(ts, "deformation"), "prev": _view(ts, "prev_deform"), "velocity": _view(ts, "velocity"),
          "next": _view(ts, "next_deform"), "forces": _view(ts, "forces")}
    if kind in ("energy", "hessian"):
        _view(ts, "inertia_deform").copy_(s["xt"])
    if kind == "hessian":
        st["x"] = np.random.default_rng(5 + int(seed)).normal(size=s["X"].shape)
    torch.cuda.synchronize()
    return st


def run(st):
    ts, kind = st["ts"], st["kind"]
    with torch.cuda.stream(st["stream"]):
        if kind == "energy":
            st["next"].copy_(st["u"])
            e = ts.update_energy_and_gradients()
            return {"energy": e, "forces": st["forces"]}
        if kind == "hessian":
            st["next"].copy_(st["u"])
            ts.update_hessian(make_spsd=True)
            y = ts.spmv(st["x"])
            return {"y": y.astype(np.float32) if st["mixed"] else y}
        if kind == "adjoint":
            ubar, vbar = st["ubar"].clone(), st["vbar"].clone()
            ebar = torch.zeros(st["eng"].num_cells, dtype=torch.float64, device="cuda")
            st["eng"].adjoint_step(st["u1"], ubar, vbar, ebar)
            return {"ubar": ubar, "vbar": vbar, "ebar": ebar}
        st["deformation"].copy_(st["u"])
        st["prev"].copy_(st["u"])
        st["velocity"].copy_(st["v"])
        ts.step()
        if st["mixed"]:
            return {"u": st["deformation"].float(), "v": st["velocity"].float()}
        return {"u": st["deformation"], "v": st["velocity"]}


# ---------------------------------------------------------------- what a pass cannot do without
def _sizes(case):
    """(cells, vertices, vertex pairs of the upper block triangle) of a case's mesh."""
    if case["scene"] == "box":
        a, b, c = case["nx"], case["ny"], case["nz"]
        nt, nv = 6 * a * b * c, (a + 1) * (b + 1) * (c + 1)
    elif case["scene"] == "batch":
        # the mean cube of kmin..kmax hexes a side
        ks = range(case["kmin"], case["kmax"] + 1)
        nt = case["n"] * sum(6 * k**3 for k in ks) // len(ks)
        nv = case["n"] * sum((k + 1) ** 3 for k in ks) // len(ks)
    else:
        n = case["nx"]
        return 2 * n * (n - 1) + 2 * (n - 1) ** 2 + 2 * n * (n - 2), n * n, 0
    return nt, nv, 8 * nv


def work(case):
    """Inputs read once and outputs written once; operations of the stated passes.  Per tet: 300 for energy and
    forces, 1,500 for the projected Hessian; 18 per block of the full matrix in a product.  A Newton step is
    counted as 6 iterations of one evaluation, one Hessian and 50 PCG products, the adjoint as 300 products."""
    nt, nv, up = _sizes(case)
    kind = case["kind"]
    if case["scene"] == "cloth":
        return {"bytes": 24.0 * nt + 24.0 * 4 * nv, "flops": 40.0 * nt}
    mesh_bytes = (16 + 88 + 24) * nt  # cells, Dm^-1 (9) and volume, material
    if case["precision"] == "mixed":
        mesh_bytes = (16 + 40 + 12) * nt
    blocks = 2 * up - nv
    if kind == "energy":
        return {"bytes": mesh_bytes + 24.0 * 4 * nv, "flops": 300.0 * nt}
    if kind == "hessian":
        return {"bytes": mesh_bytes + 24.0 * 4 * nv, "flops": 1500.0 * nt + 18.0 * blocks}
    if kind == "adjoint":
        return {"bytes": mesh_bytes + 24.0 * 6 * nv + 16.0 * nt, "flops": 1800.0 * nt + 300 * 18.0 * blocks}
    if kind == "lbfgs":
        return {"bytes": mesh_bytes + 24.0 * 5 * nv, "flops": case["iters"] * 300.0 * nt}
    return {"bytes": mesh_bytes + 24.0 * 5 * nv, "flops": 6 * (1800.0 * nt + 50 * 18.0 * blocks)}


# ---------------------------------------------------------------- the same results in plain torch, 64 bits
class _Tets:
    """The incremental potential 1/2 |x - x~|^2_M + dt^2 sum_e V_e Psi(F_e) of stable Neo-Hookean tets in plain
    torch: energy, gradient, element Hessians.  Psi = 1/2 [mu (Ic - 3) + lambda (J - alpha)^2 - mu log(Ic + 1)]
    - Psi(I), alpha = 1 + 3/4 mu / lambda; consistent mass rho V_e / 20 (1 + delta_ij)."""

    def __init__(self, s):
        self.T = torch.from_numpy(s["cells"].astype(np.int64)).cuda()
        self.X, self.nv = s["Xd"], s["Xd"].shape[0]
        x = self.X[self.T]
        D = torch.stack([x[:, 1] - x[:, 0], x[:, 2] - x[:, 0], x[:, 3] - x[:, 0]], dim=2)
        B = torch.linalg.inv(D)
        self.V = torch.linalg.det(D).abs() / 6
        self.D = torch.cat([-B.sum(1, keepdim=True), B], dim=1)  # shape gradients [T, 4, 3]
        E = torch.from_numpy(np.ascontiguousarray(s["E"])).cuda()
        nu = torch.full_like(E, NU) if s["nu"] is None else torch.from_numpy(s["nu"]).cuda()
        self.E, self.mu, self.lam = E, E / (2 * (1 + nu)), E * nu / ((1 + nu) * (1 - 2 * nu))
        self.alpha = 1 + 0.75 * self.mu / self.lam
        self.psi0 = 0.5 * (self.lam * (1 - self.alpha) ** 2 - self.mu * math.log(4.0))
        self.free = s["free"][:, None]
        self.xt = s["xt"]

    def F(self, u):
        G = torch.einsum("tvi,tvj->tij", u[self.T], self.D)
        return G + torch.eye(3, dtype=torch.float64, device=u.device)

    @staticmethod
    def cof(F):
        return torch.stack([torch.linalg.cross(F[:, 1], F[:, 2]), torch.linalg.cross(F[:, 2], F[:, 0]),
                            torch.linalg.cross(F[:, 0], F[:, 1])], dim=1)

    def mass(self, w):
        we = w[self.T]
        m = (RHO * self.V / 20)[:, None, None] * (we + we.sum(1, keepdim=True))
        return torch.zeros_like(w).index_add_(0, self.T.reshape(-1), m.reshape(-1, 3))

    def stress(self, F):
        Ic, C = (F * F).sum((1, 2)), self.cof(F)
        J = (F[:, 0] * C[:, 0]).sum(1)
        return ((self.lam * (J - self.alpha))[:, None, None] * C + (self.mu * (1 - 1 / (Ic + 1)))[:, None, None] * F), Ic, J, C

    def evaluate(self, u):
        F = self.F(u)
        P, Ic, J, _ = self.stress(F)
        psi = 0.5 * (self.mu * (Ic - 3) + self.lam * (J - self.alpha) ** 2 - self.mu * torch.log(Ic + 1)) - self.psi0
        f = DT * DT * self.V[:, None, None] * torch.einsum("tij,tvj->tvi", P, self.D)
        w = u - self.xt
        Mw = self.mass(w)
        g = Mw + torch.zeros_like(u).index_add_(0, self.T.reshape(-1), f.reshape(-1, 3))
        return float(0.5 * (w * Mw).sum() + DT * DT * (self.V * psi).sum()), g * self.free

    def element_hessians(self, u, spsd, lo=0, hi=None):
        """dt^2 V_e times the 12 x 12 element Hessians of tets lo..hi; spsd: eigenvalues of d2Psi/dF2 raised to
        1e-3."""
        hi = self.T.shape[0] if hi is None else hi
        F = self.F(u)[lo:hi]
        mu, lam, alpha = self.mu[lo:hi], self.lam[lo:hi], self.alpha[lo:hi]
        Ic, C = (F * F).sum((1, 2)), self.cof(F)
        J = (F[:, 0] * C[:, 0]).sum(1)
        f, c = F.reshape(-1, 9), C.reshape(-1, 9)
        H = (mu * (1 - 1 / (Ic + 1)))[:, None, None] * torch.eye(9, dtype=torch.float64, device=u.device)
        H = H + (2 * mu / (Ic + 1) ** 2)[:, None, None] * f[:, :, None] * f[:, None, :] + lam[:, None, None] * c[:, :, None] * c[:, None, :]
        d2J = torch.zeros_like(H)  # d cof / dF: antisymmetric blocks of the rows of F
        for a, b, r, sg_ in ((0, 1, 2, 1.0), (1, 2, 0, 1.0), (2, 0, 1, 1.0)):
            x = F[:, r]
            K = torch.zeros(F.shape[0], 3, 3, dtype=torch.float64, device=u.device)
            K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -x[:, 2], x[:, 1], -x[:, 0]
            K = K - K.transpose(1, 2)
            # J = row_r . (row_a x row_b): d2J / d row_a d row_b = -[row_r]x
            d2J[:, 3 * a:3 * a + 3, 3 * b:3 * b + 3] = -sg_ * K
            d2J[:, 3 * b:3 * b + 3, 3 * a:3 * a + 3] = sg_ * K
        H = H + (lam * (J - alpha))[:, None, None] * d2J
        if spsd:
            w, Q = np.linalg.eigh(H.cpu().numpy())
            w, Q = torch.from_numpy(np.maximum(w, 1e-3)).cuda(), torch.from_numpy(Q).cuda()
            H = torch.einsum("tik,tk,tjk->tij", Q, w, Q)
        H = H.reshape(-1, 3, 3, 3, 3)
        K = torch.einsum("tvj,tijkl,twl->tviwk", self.D[lo:hi], H, self.D[lo:hi])
        return (DT * DT * self.V[lo:hi])[:, None, None] * K.reshape(-1, 12, 12)

    def apply(self, K, x, tau=0.0):
        """((1 + tau) M + K) x with the Dirichlet identity."""
        xf = x * self.free
        y = torch.bmm(K, xf[self.T].reshape(-1, 12, 1)).reshape(-1, 3)
        y = (1 + tau) * self.mass(xf) + torch.zeros_like(x).index_add_(0, self.T.reshape(-1), y)
        return y * self.free + x * (1 - self.free)

    def diagonal(self, K, tau=0.0):
        m = ((1 + tau) * RHO * self.V / 10)[:, None, None]
        d = torch.diagonal(K, dim1=1, dim2=2).reshape(-1, 4, 3) + m
        d = torch.zeros_like(self.X).index_add_(0, self.T.reshape(-1), d.reshape(-1, 3))
        return d * self.free + (1 - self.free)

    def solve(self, K, b, tol=1e-13, most=4000, tau=0.0):
        """Jacobi-preconditioned CG on (1 + tau) M + K; None on a direction of negative curvature."""
        d = self.diagonal(K, tau)
        if float(d.min()) <= 0:
            return None
        x, r = torch.zeros_like(b), b.clone()
        z = r / d
        p, rz, n0 = z.clone(), (r * z).sum(), float(b.norm())
        low = torch.full((), math.inf, dtype=torch.float64, device=b.device)
        for k in range(most):
            if k % 16 == 0 and (float(r.norm()) <= tol * n0 or float(low) <= 0):
                break
            q = self.apply(K, p, tau)
            pq = (p * q).sum()
            low = torch.minimum(low, pq)
            a = rz / pq
            x, r = x + a * p, r - a * q
            z = r / d
            rz, old = (r * z).sum(), rz
            p = z + (rz / old) * p
        return x if float(low) > 0 else None

    def minimise(self):
        """The minimiser of the incremental potential from x~, to round-off; None if it was not reached."""
        u = self.xt.clone()
        E, g = self.evaluate(u)
        g0 = gn = float(g.norm())
        tau = 0.0
        for _ in range(60):
            if gn <= 1e-13 * g0:
                break
            K = self.element_hessians(u, False)
            d = None
            while d is None and tau < 1e6:  # more mass until the Hessian is positive definite
                d = self.solve(K, -g, tol=1e-3 if gn > 1e-3 * g0 else 1e-7, tau=tau)
                tau = tau / 4 if d is not None else max(1.0, 4 * tau)
            tau = tau if tau >= 0.25 else 0.0
            if d is None:
                return None
            a, slope = 1.0, float((g * d).sum())
            while True:
                En, gt = self.evaluate(u + a * d)
                if En <= E + 1e-4 * a * slope or (abs(slope) < 1e-12 * abs(E) and float(gt.norm()) < gn) or a < 1e-8:
                    break
                a *= 0.5
            if float(gt.norm()) >= gn and gn <= 1e-10 * g0:
                break  # at round-off
            u, E, g, gn = u + a * d, En, gt, float(gt.norm())
        return u if gn <= 1e-10 * g0 else None


def exact(case, seed):
    kind = case["kind"]
    if kind == "lbfgs":
        return None  # the iterate after a fixed number of iterations has no value but the algorithm's own
    s = _scene(case, seed)
    if case["scene"] == "cloth":
        c = torch.from_numpy(s["cells"].astype(np.int64)).cuda()
        X, u = s["Xd"], s["u"]
        L = (X[c[:, 0]] - X[c[:, 1]]).norm(dim=1)
        e = (X + u)[c[:, 0]] - (X + u)[c[:, 1]]
        l = e.norm(dim=1)
        m = torch.from_numpy(s["vertex_mass"]).cuda()[:, None]
        w = u - s["xt"]
        f = (DT * DT * s["k"] * (l - L) / l)[:, None] * e
        g = m * w
        g.index_add_(0, c[:, 0], f).index_add_(0, c[:, 1], -f)
        E = 0.5 * float((m * w * w).sum()) + DT * DT * 0.5 * s["k"] * float(((l - L) ** 2).sum())
        return {"energy": E, "forces": g * s["free"][:, None]}
    nt = s["cells"].shape[0]
    if kind == "energy":
        E, g = _Tets(s).evaluate(s["u"])
        return {"energy": E, "forces": g}
    if kind == "hessian":
        t = _Tets(s)
        x = torch.from_numpy(np.random.default_rng(5 + int(seed)).normal(size=s["X"].shape)).cuda()
        y = torch.zeros_like(x)
        xf = x * t.free
        for lo in range(0, nt, 32768):  # the 9 x 9 eigenproblems of one block of tets at a time
            hi = min(nt, lo + 32768)
            K = t.element_hessians(s["u"], True, lo, hi)
            y.index_add_(0, t.T[lo:hi].reshape(-1), torch.bmm(K, xf[t.T[lo:hi]].reshape(-1, 12, 1)).reshape(-1, 3))
        y = (y + t.mass(xf)) * t.free + x * (1 - t.free)
        return {"y": y}
    if kind == "adjoint":
        t, g = _Tets(s), s["gen"]
        ubar = torch.randn(s["X"].shape, generator=g, dtype=torch.float64).cuda()
        vbar = 1e-2 * torch.randn(s["X"].shape, generator=g, dtype=torch.float64).cuda()
        lam = t.solve(t.element_hessians(s["u"], False), (ubar + vbar / DT) * t.free)
        xb = t.mass(lam) * t.free
        P = t.stress(t.F(s["u"]))[0]
        W = torch.einsum("tvi,tvj->tij", lam[t.T], t.D)
        return {"ubar": xb - vbar / DT, "vbar": DT * xb, "ebar": -DT * DT * t.V * (W * P).sum((1, 2)) / t.E}
    if nt > 2000000:
        return None  # the minimiser of larger systems takes this plain Newton-CG over 20 seconds
    t = _Tets(s)
    u1 = t.minimise()
    return None if u1 is None else {"u": u1, "v": (u1 - s["u"]) / DT}
