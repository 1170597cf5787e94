"""Performance cases: the time steps that users of this library run.

A case is one *pass* of a running simulation, through the calls a driver
makes: the max wave speed (the CFL time step), then SSP-RK3 steps at the
reference drivers' cadence -- one step per wave speed for WENO5, ten for DG
(or a fixed time step and many steps, as a convergence or batch job does) --
on a context whose state stays on the device and is read in place
(zk_state_device).  Running a pass again continues the simulation.  The
batched case is a whole batch job: add every problem from host arrays, run,
read every state back.

Initial states are seeded:
  quadrants  four constant states meeting at the centre, transmissive ring --
             shocks, contacts and rarefactions (the library's benchmark
             problem).  Drawn from rho, p in [0.5, 2], |u|, |v| <= 0.5, inside
             the benchmark's [0.1, 2] and 1, because the schemes have no
             positivity fix that carries every such draw through a long run
  wave       a smooth density wave on a periodic grid (the accuracy problem)
  jet        a dense supersonic jet entering from frozen inflow columns

`exact` integrates the same pass in 64-bit torch, written from the scheme's
definition and independent of the library.
"""
import ctypes
import math

import numpy as np
import torch

from zuikakucfd_b200 import Solver, _native
from zuikakucfd_b200.batch import Batch

WENO_CFL = 0.4   # the WENO driver's CFL number
DG_CFL = 0.5     # fraction of the DG driver's CFL limit
TVB_M = 50.0


def _case(name, method, precision, ny, nx, steps, problem="quadrants", order=0, limiter="none", fixed_dt=False):
    c = dict(kind="step", method=method, order=order, precision=precision, limiter=limiter, ny=ny, nx=nx,
             steps=steps, problem=problem, fixed_dt=fixed_dt)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest driver loop (teaching and unit-test grids): launch and read-back latency
        _case("weno_fp64_64", "weno", "fp64", 64, 64, 1),
        # the 256^2 reference run: fixed time step, many steps in one call
        _case("weno_fp64_256", "weno", "fp64", 256, 256, 50, fixed_dt=True),
        # a ragged periodic grid on the fast path
        _case("weno_mixed_173x301", "weno", "mixed", 173, 301, 1, problem="wave"),
        # the large shock problem on the fast path, and in plain FP64 at half the side
        _case("weno_mixed_2048", "weno", "mixed", 2048, 2048, 1),
        _case("weno_fp64_1024", "weno", "fp64", 1024, 1024, 1),
        # DG P=1 with the reference's limiter on the jet
        _case("dg1_mixed_jet_512x1024", "dg", "mixed", 512, 1024, 10, problem="jet", order=1, limiter="reference"),
        # the smooth-wave accuracy study: DG P=2 with TVB on a periodic grid
        _case("dg2_mixed_wave_1030", "dg", "mixed", 1030, 1030, 10, problem="wave", order=2, limiter="tvb"),
        # plain FP64 DG with the reference's limiter on a ragged grid
        _case("dg2_fp64_203x331", "dg", "fp64", 203, 331, 10, order=2, limiter="reference"),
        # the plain FP64 baseline of the flagship problem at half its side
        _case("dg3_fp64_1024", "dg", "fp64", 1024, 1024, 10, order=3, limiter="tvb"),
        # the flagship: DG P=3, mixed precision, TVB gated by the learned indicator
        _case("dg3_mixed_2048", "dg", "mixed", 2048, 2048, 10, order=3, limiter="tvb_mlp"),
        # FP64 with fused multiply-adds and the reference's limiter
        _case("dg3_fma_768", "dg", "fp64_fma", 768, 768, 10, order=3, limiter="reference"),
        # batched serving: uneven problems, half WENO5 and half DG P=2
        dict(name="batch_8", kind="batch", problems=8, min_side=128, max_side=512, steps=180),
    ]


def draw(rng):
    """One more case of the same ranges: methods, precisions, orders, limiters
    and problems at random, sides log-uniform from 64 to 2048 (odd ones too),
    no larger than the listed cases."""
    if rng.random() < 0.08:
        n = rng.randint(4, 10)
        return dict(kind="batch", problems=n, min_side=64, max_side=rng.choice([192, 256, 384]),
                    steps=rng.randint(40, 1400 // n))
    side = lambda hi: int(round(64 * (hi / 64) ** rng.random()))  # noqa: E731
    if rng.random() < 0.4:
        precision = rng.choice(["fp64", "mixed", "mixed", "fp64_fma"])
        hi = 2048 if precision == "mixed" else 1448
        fixed = rng.random() < 0.25
        ny, nx = side(hi), side(hi)
        steps = max(1, min(50, int(6e6 / (ny * nx)))) if fixed else 1
        return _case(None, "weno", precision, ny, nx, steps, problem=rng.choice(["quadrants", "quadrants", "wave"]),
                     fixed_dt=fixed)
    order = rng.randint(1, 3)
    precision = rng.choice(["fp64", "mixed", "mixed", "fp64_fma"])
    problem = rng.choice(["quadrants", "quadrants", "wave"] + (["jet"] if order == 1 else []))
    if problem == "jet":
        limiter = "reference"
    else:
        limiter = rng.choice(["reference", "tvb"] + (["tvb_mlp"] if order > 1 and precision == "mixed" else [])
                             + (["none"] if problem == "wave" else []))
    cells = (1.0 if precision != "mixed" else 3.0) * 2 ** 20 * 4 / (order + 1) ** 2 * (2.5 if order == 3 else 1.5)
    ny, nx = side(2048), side(2048)
    while ny * nx > min(cells, 4e6):
        ny, nx = max(64, int(ny * 0.8)), max(64, int(nx * 0.8))
    return _case(None, "dg", precision, ny, nx, 10, problem=problem, order=order, limiter=limiter)


# ---- problems -------------------------------------------------------------------

def _bctype(c):
    ny, nx = c["ny"], c["nx"]
    b = np.full((ny, nx), -3 if c["problem"] == "wave" else -1, np.int32)
    b[3:-3, 3:-3] = 0
    if c["problem"] == "jet":
        b[3:-3, :3] = 0  # frozen inflow columns
    return b


def _grid(c):
    """(cell size, gamma): the wave spans [0, 2] inside its ring, the others [0, 1]."""
    if c["problem"] == "wave":
        return 2.0 / (max(c["ny"], c["nx"]) - 6), 1.4
    return 1.0 / max(c["ny"], c["nx"]), 5.0 / 3.0 if c["problem"] == "jet" else 1.4


def _conserved(rho, u, v, p, gamma):
    return torch.stack([rho, rho * u, rho * v, p / (gamma - 1.0) + 0.5 * rho * (u * u + v * v)])


def _initial(c, seed, device):
    """The state, [4, ny, nx] (WENO) or [4, NM, ny, nx] (DG)."""
    r = np.random.default_rng([int(seed), c["ny"], c["nx"]])
    ny, nx, (da, gamma) = c["ny"], c["nx"], _grid(c)
    kw = dict(device=device, dtype=torch.float64)
    nm = (c["order"] + 1) ** 2 if c["method"] == "dg" else 1
    one = torch.ones(ny, nx, **kw)
    if c["problem"] == "wave":
        a, phase, u, v, p = r.uniform(0.15, 0.25), r.uniform(0, 2 * math.pi), *r.uniform(-1, 1, 2), r.uniform(0.8, 1.2)
        q = c["order"] + 1 if c["method"] == "dg" else 1
        t, w = np.polynomial.legendre.leggauss(q)
        i = torch.arange(ny, **kw).sub(3).remainder(ny - 6).add(0.5)[:, None]
        j = torch.arange(nx, **kw).sub(3).remainder(nx - 6).add(0.5)[None, :]
        modes = [torch.zeros(ny, nx, **kw) for _ in range(nm)]
        for k in range(q * q):  # L2 projection at the Gauss points (a point value for WENO)
            x, y = (j + 0.5 * t[k // q]) / (nx - 6), (i + 0.5 * t[k % q]) / (ny - 6)
            rho = 1.0 + a * torch.sin(2 * math.pi * (x + y) + phase)
            for m in range(nm):
                px, py = m // q, m % q
                f = (2 * px + 1) * (2 * py + 1) / 4.0 * w[k // q] * w[k % q]
                modes[m] += f * _legendre(px, t[k // q]) * _legendre(py, t[k % q]) * rho
        rho = torch.stack(modes)
        s = torch.stack([rho, u * rho, v * rho, 0.5 * (u * u + v * v) * rho])
        s[3, 0] += p / (gamma - 1.0)
        return s if c["method"] == "dg" else s[:, 0]
    if c["problem"] == "jet":
        rho, u, v, p = 0.5 * one, 0 * one, 0 * one, 0.4127 * one
        y = (torch.arange(ny, **kw) + 0.5) / ny - 0.5
        band = y.abs() < r.uniform(0.08, 0.12)
        rho[band, :3] = r.uniform(4.0, 5.0)
        u[band, :3] = r.uniform(4.0, 6.0)
    else:
        q = np.stack([r.uniform(0.5, 2.0, 4), r.uniform(-0.5, 0.5, 4), r.uniform(-0.5, 0.5, 4), r.uniform(0.5, 2.0, 4)])
        at = (2 * (torch.arange(ny, device=device) >= ny // 2)[:, None].long()
              + (torch.arange(nx, device=device) >= nx // 2)[None, :].long())
        rho, u, v, p = (torch.tensor(q[k], **kw)[at] for k in range(4))
    U = _conserved(rho, u, v, p, gamma)
    if c["method"] != "dg":
        return U
    s = torch.zeros(4, nm, ny, nx, **kw)
    s[:, 0] = U
    return s


def _legendre(n, x):
    return [1.0, x, 0.5 * (3 * x * x - 1), 0.5 * (5 * x * x * x - 3 * x)][n]


def _dlegendre(n, x):
    return [0.0, 1.0, 3 * x, 0.5 * (15 * x * x - 3)][n]


def _dt(c, da, lam):
    if c["method"] == "dg":
        return DG_CFL * 0.9 / (2.0 * (2 * c["order"] + 1)) * da / max(lam, 1e-7)
    return (0.3 if c["fixed_dt"] else WENO_CFL) * da / lam


# ---- a pass through the library -----------------------------------------------------

class _DeviceState:
    """The context's FP64 state as a CUDA array of [planes, ny, pitch]; keeps
    the context, which owns the memory, alive."""

    def __init__(self, solver, planes):
        self.solver = solver
        ptr, pitch = ctypes.POINTER(ctypes.c_double)(), ctypes.c_int()
        _native.check(_native.lib().zk_state_device(solver._h, ctypes.byref(ptr), ctypes.byref(pitch)))
        self.__cuda_array_interface__ = dict(
            shape=(planes, solver.ny, pitch.value), typestr="<f8", version=3, strides=None,
            data=(ctypes.cast(ptr, ctypes.c_void_p).value, False))


def _batch_members(c, seed):
    """The batch's problems as step cases, with their seeds: sides evenly over
    the case's range, the first half WENO5, the second half DG P=2 with the
    reference's limiter."""
    half = c["problems"] // 2
    sides = np.linspace(c["min_side"], c["max_side"], c["problems"] - half).round().astype(int)
    sides = np.concatenate([sides[:half], sides])
    out = []
    for k, s in enumerate(sides):
        m = _case(None, "weno" if k < half else "dg", "mixed", int(s), int(s), c["steps"],
                  order=0 if k < half else 2, limiter="none" if k < half else "reference")
        out.append((m, int(seed) * 1009 + k))
    return out


def prepare(case, seed):
    c = case
    if c["kind"] == "batch":
        return dict(case=c, members=[(m, _bctype(m), _initial(m, s, "cuda").cpu().numpy())
                                     for m, s in _batch_members(c, seed)])
    da, gamma = _grid(c)
    solver = Solver(method=c["method"], order=max(1, c["order"]), precision=c["precision"],
                    limiter=c["limiter"] if c["method"] == "dg" else "reference",
                    boundary="periodic" if c["problem"] == "wave" else "exchange", tvb_M=TVB_M)
    solver.set_mesh(c["ny"], c["nx"], da, gamma, _bctype(c))
    if c["limiter"] == "tvb_mlp":
        solver.set_indicator()
    init = _initial(c, seed, "cuda")
    view = torch.as_tensor(_DeviceState(solver, init[..., 0, 0].numel()), device="cuda")
    view = view.view(*init.shape[:-2], *view.shape[-2:])[..., : c["nx"]]
    view.copy_(init)
    torch.cuda.synchronize()
    st = dict(case=c, solver=solver, view=view, da=da)
    if c["fixed_dt"]:
        st["dt"] = _dt(c, da, solver.max_speed())
    return st


def run(state):
    c = state["case"]
    if c["kind"] == "batch":
        with Batch(policy="all") as b:
            ids = [b.add(bt, *_grid(m), s, m["steps"], WENO_CFL if m["method"] == "weno" else DG_CFL,
                         method=m["method"], order=max(1, m["order"]), precision=m["precision"], limiter="reference")
                   for m, bt, s in state["members"]]
            b.run()
            return [b.get_state(k) for k in ids]
    solver = state["solver"]
    if c["fixed_dt"]:
        solver.step(state["dt"], c["steps"])
        return {"state": state["view"]}
    lam = solver.max_speed()
    solver.step(_dt(c, state["da"], lam), c["steps"])
    return {"state": state["view"], "max_speed": lam}


def work(case):
    """Face-deduplicated operations per updated cell and stage (add, sub, mul,
    div, sqrt, min, max: WENO5 1,330; DG P = 1, 2, 3: 1,700, 5,300, 13,200);
    the state read once and written once."""
    if case["kind"] == "batch":
        parts = [work(m) for m, _ in _batch_members(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    cells = (case["ny"] - 6) * (case["nx"] - 6)
    dg = case["method"] == "dg"
    planes = 4 * (case["order"] + 1) ** 2 if dg else 4
    flops = {0: 1330, 1: 1700, 2: 5300, 3: 13200}[case["order"] if dg else 0]
    return {"bytes": 2 * 8.0 * planes * case["ny"] * case["nx"], "flops": 3.0 * flops * cells * case["steps"]}


# ---- the same pass in 64-bit torch ------------------------------------------------------

def _ghost_sources(n, periodic, frozen):
    """Source index of each index of one axis: periodic images, or the largest
    interior index within 3 cells (the fill order of the scheme's row sweep)."""
    if periodic:
        return [3 + (k - 3) % (n - 6) for k in range(n)]
    lo = list(range(3)) if frozen else [min(k + 3, n - 4) for k in range(3)]
    return lo + list(range(3, n - 3)) + [n - 4] * 3


class _Exact:
    def __init__(self, c, device):
        self.c, (self.da, self.gamma) = c, _grid(c)
        self.periodic = c["problem"] == "wave"
        ix = lambda n, f: torch.tensor(_ghost_sources(n, self.periodic, f), device=device)  # noqa: E731
        self.rows, self.cols = ix(c["ny"], False), ix(c["nx"], c["problem"] == "jet")
        if c["method"] == "dg":
            q = c["order"] + 1
            t, w = np.polynomial.legendre.leggauss(q)
            self.q, nm = q, q * q
            kw = dict(device=device, dtype=torch.float64)
            L, D = _legendre, _dlegendre
            pts = [(a, b) for a in range(q) for b in range(q)]
            tab = lambda f, g: torch.tensor([[f(m // q, t[a]) * g(m % q, t[b]) for m in range(nm)]  # noqa: E731
                                             for a, b in pts], **kw)
            wv = torch.tensor([w[a] * w[b] for a, b in pts], **kw)[:, None]
            self.phi, self.dxi, self.det = tab(L, L), tab(D, L) * wv, tab(L, D) * wv
            face = lambda f: torch.tensor([[f(m // q, m % q, x) for m in range(nm)] for x in t], **kw)  # noqa: E731
            self.tr = [face(lambda a, b, x: L(a, 1.0) * L(b, x)), face(lambda a, b, x: L(a, -1.0) * L(b, x)),
                       face(lambda a, b, x: L(a, x) * L(b, 1.0)), face(lambda a, b, x: L(a, x) * L(b, -1.0))]
            self.bv = [x * torch.tensor(w, **kw)[:, None] for x in self.tr]
            self.scale = torch.tensor([(2 * (m // q) + 1) * (2 * (m % q) + 1) * 0.5 / self.da for m in range(nm)],
                                      **kw)[:, None, None]
            cut = lambda n, x: L(n, x) if n < 3 else 0.0  # noqa: E731  positivity points drop the cubic factors
            g4 = np.polynomial.legendre.leggauss(4)[0]
            self.zs = torch.tensor([[cut(m // q, x) * cut(m % q, y) for m in range(nm)] for x in g4 for y in g4], **kw)
            self.corner = torch.tensor([[L(m // q, x) * L(m % q, y) for m in range(nm)]
                                        for y in (-1.0, 1.0) for x in (-1.0, 1.0)], **kw)
            self.high = torch.tensor([m // q == q - 1 or m % q == q - 1 for m in range(nm)], device=device)

    def fill(self, U):
        V = U.clone()
        if self.periodic:
            return V[..., self.rows, :][..., self.cols]
        V[..., 3:-3, :] = U[..., 3:-3, :][..., self.cols]
        V[..., :, 3:-3] = V[..., self.rows, :][..., 3:-3]
        return V

    def max_speed(self, U):
        g = self.gamma
        if self.c["method"] == "dg":
            lo = 0 if self.c["problem"] == "jet" else 3  # the frozen inflow columns count
            U = torch.einsum("cmij,km->ckij", U[..., 3:-3, lo:-3], self.corner)
            rho = U[0].clamp(min=1e-12)
            p = ((g - 1) * (U[3] - 0.5 * (U[1] ** 2 + U[2] ** 2) / rho)).clamp(min=1e-12)
        else:
            rho = U[0]
            p = (g - 1) * (U[3] - 0.5 * (U[1] ** 2 + U[2] ** 2) / rho)
        return float((torch.sqrt(U[1] ** 2 + U[2] ** 2) / rho + torch.sqrt(g * p / rho)).max())

    def hllc(self, L, R, eps):
        """HLLC flux along the first momentum; L, R = 4 tensors each."""
        g = self.gamma

        def side(U):
            rho = U[0].clamp(min=eps)
            u, v, E = U[1] / rho, U[2] / rho, U[3] / rho
            p = ((g - 1) * (U[3] - 0.5 * rho * (u * u + v * v))).clamp(min=eps)
            return rho, u, v, E, p, torch.sqrt((g * p / rho).clamp(min=eps)), torch.sqrt(rho)

        rl, ul, vl, El, pl, al, sl = side(L)
        rr, ur, vr, Er, pr, ar, sr = side(R)
        den = sl + sr
        u = (sl * ul + sr * ur) / den
        h = (sl * (El + pl / rl) + sr * (Er + pr / rr)) / den
        a = torch.sqrt(((g - 1) * (h - 0.5 * u * u)).clamp(min=eps))
        SL, SR = torch.minimum(ul - al, u - a), torch.maximum(ur + ar, u + a)
        away = lambda x: torch.where(x.abs() < eps, torch.where(x >= 0, eps, -eps).to(x), x)  # noqa: E731
        Ss = (pr - pl + rl * ul * (SL - ul) - rr * ur * (SR - ur)) / away(rl * (SL - ul) - rr * (SR - ur))
        left = Ss >= 0
        pick = lambda x, y: torch.where(left, x, y)  # noqa: E731
        left = left & (SR > 0) | (SL >= 0)
        rho, u, v, E, p, S = (pick(x, y) for x, y in ((rl, rr), (ul, ur), (vl, vr), (El, Er), (pl, pr), (SL, SR)))
        Us = [pick(x, y) for x, y in zip(L, R)]
        k = rho * (S - u) / away(S - Ss)
        star = [k, k * Ss, k * v, k * (E + (Ss - u) * (Ss + p / (rho * (S - u))))]
        F = [rho * u, rho * u * u + p, rho * u * v, (Us[3] + p) * u]
        whole = (SL >= 0) | (SR <= 0)
        return [torch.where(whole, f, f + S * (s - x)) for f, s, x in zip(F, star, Us)]

    # -- WENO5 ----------------------------------------------------------------------
    @staticmethod
    def weno5(a, b, c, d, e):
        q = ((2 * a - 7 * b + 11 * c) / 6, (-b + 5 * c + 2 * d) / 6, (2 * c + 5 * d - e) / 6)
        s = (13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2,
             13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2,
             13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2)
        w = [x / (1e-6 + y) ** 2 for x, y in zip((0.1, 0.6, 0.3), s)]
        return (w[0] * q[0] + w[1] * q[1] + w[2] * q[2]) / (w[0] + w[1] + w[2])

    def weno_rhs(self, V, dt):
        d = torch.zeros_like(V)

        def flux(W):  # faces between cells 2|3 .. n-4|n-3 of the last axis
            n = W.shape[-1]
            s = [W[..., k: n - 5 + k] for k in range(6)]
            return torch.stack(self.hllc(list(self.weno5(*s[:5])), list(self.weno5(*s[:0:-1])), 1e-12))

        F = flux(V[:, 3:-3, :])
        swap = [0, 2, 1, 3]
        G = flux(V[swap][:, :, 3:-3].transpose(1, 2)).transpose(1, 2)[swap]
        d[:, 3:-3, 3:-3] = -(dt / self.da) * ((F[..., 1:] - F[..., :-1]) + (G[:, 1:] - G[:, :-1]))
        return d

    # -- DG ---------------------------------------------------------------------------
    def dg_rhs(self, V):
        g = self.gamma
        d = torch.zeros_like(V)
        I = V[..., 3:-3, 3:-3]
        U = torch.einsum("cmij,pm->cpij", I, self.phi)
        rho = U[0].clamp(min=1e-3)
        u, v = U[1] / rho, U[2] / rho
        p = ((g - 1) * (U[3] - 0.5 * rho * (u * u + v * v))).clamp(min=1e-3)
        F = torch.stack([rho * u, rho * u * u + p, rho * u * v, (U[3] + p) * u])
        out = torch.einsum("cpij,pm->cmij", F, self.dxi)
        F = torch.stack([rho * v, rho * u * v, rho * v * v + p, (U[3] + p) * v])
        out += torch.einsum("cpij,pm->cmij", F, self.det)
        del F, U
        trace = lambda W, k: torch.einsum("cmij,qm->cqij", W, self.tr[k])  # noqa: E731
        X, Y = V[..., 3:-3, 2:-2], V[..., 2:-2, 3:-3]
        Fx = torch.stack(self.hllc(list(trace(X[..., :-1], 0)), list(trace(X[..., 1:], 1)), 1e-5))
        swap = [0, 2, 1, 3]
        Fy = torch.stack(self.hllc(list(trace(Y[..., :-1, :], 2)[swap]), list(trace(Y[..., 1:, :], 3)[swap]), 1e-5))[swap]
        for k, f in enumerate((Fx[..., 1:], Fx[..., :-1], Fy[..., 1:, :], Fy[..., :-1, :])):
            out += (-1.0 if k % 2 == 0 else 1.0) * torch.einsum("cqij,qm->cmij", f, self.bv[k])
        d[..., 3:-3, 3:-3] = out * self.scale
        return d

    def limit_reference(self, U):
        """Persson modal filter, then Zhang-Shu positivity, per cell."""
        g, floor, eps = self.gamma, 1e-5, 1e-5
        o = U[..., 3:-3, 3:-3].clone()
        P = self.q - 1
        s0 = (-3.0 if P >= 3 else -4.0) * math.log10(P)
        s = torch.log10((o * o)[:, self.high].sum(1) / ((o * o).sum(1) + eps))
        ramp = 0.5 * (1.0 + torch.sin(math.pi * (s - s0 - 0.5)))
        cut = torch.where(s > s0, torch.where(s > s0 + 1.0, torch.ones_like(s), ramp), torch.zeros_like(s))
        o[:, self.high] *= (1.0 - cut)[:, None]
        o[0, 0] = o[0, 0].clamp(min=floor)
        ke = 0.5 * (o[1, 0] ** 2 + o[2, 0] ** 2) / o[0, 0]
        o[3, 0] = torch.where((g - 1) * (o[3, 0] - ke) < floor, floor / (g - 1) + ke, o[3, 0])
        rho = torch.einsum("mij,km->kij", o[0], self.zs)
        one = torch.ones_like(rho)
        th = torch.where(rho < floor, (o[0, 0] - floor) / (o[0, 0] - rho + eps), one).amin(0).clamp(max=1.0)
        o[:, 1:] *= th
        Z = torch.einsum("cmij,km->ckij", o, self.zs)
        p = (g - 1) * (Z[3] - 0.5 * (Z[1] ** 2 + Z[2] ** 2) / Z[0])
        avg = (g - 1) * (o[3, 0] - 0.5 * (o[1, 0] ** 2 + o[2, 0] ** 2) / o[0, 0])
        th = torch.where((Z[0] > floor) & (p < floor), (avg - floor) / (avg - p + eps), one).amin(0).clamp(max=1.0)
        o[:, 1:] *= th
        U[..., 3:-3, 3:-3] = o

    def limit_tvb(self, U):
        """Cockburn-Shu TVB minmod on characteristic slopes, neighbour means through the ghost fill."""
        q, g, mh2 = self.q, self.gamma, TVB_M * self.da ** 2
        M = self.fill(U[:, 0])
        b = M[:, 3:-3, 3:-3]
        rho = b[0]
        vel = b[1:3] / rho
        q2 = vel[0] ** 2 + vel[1] ** 2
        p = (g - 1) * (b[3] - 0.5 * rho * q2)
        phys = (rho > 0) & (p > 0)
        a = torch.sqrt(g * torch.where(phys, p / rho, torch.ones_like(p)))
        H, b1 = (b[3] + p) / rho, (g - 1) / (a * a)
        b2 = 0.5 * q2 * b1

        def direction(slope, dp, dm, n):
            t = 3 - n
            un, ut = vel[n - 1], vel[t - 1]

            def project(w):  # left eigenvectors
                s, m = 0.5 * (b2 * w[0] - b1 * un * w[n] - b1 * ut * w[t] + b1 * w[3]), 0.5 * (un * w[0] - w[n]) / a
                return [s + m, w[0] - 2 * s, w[t] - ut * w[0], s - m]

            lims, changed = [], torch.zeros_like(phys)
            plain = [list(slope), list(dp), list(dm)]
            char = [project(w) for w in plain]
            for r in range(4):
                w, x, y = (torch.where(phys, char[k][r], plain[k][r]) for k in range(3))
                up = torch.where((w > 0) & (x > 0) & (y > 0), torch.minimum(w, torch.minimum(x, y)), torch.zeros_like(w))
                dn = torch.where((w < 0) & (x < 0) & (y < 0), torch.maximum(w, torch.maximum(x, y)), up)
                lim = torch.where(w.abs() <= mh2, w, dn)
                changed |= lim != w
                lims.append(lim)
            l0, l1, l2, l3 = lims
            out = [None] * 4
            out[0] = l0 + l1 + l3
            out[n] = (un - a) * l0 + un * l1 + (un + a) * l3
            out[t] = ut * (l0 + l1 + l3) + l2
            out[3] = (H - un * a) * l0 + 0.5 * q2 * l1 + ut * l2 + (H + un * a) * l3
            return torch.stack([torch.where(phys, x, y) for x, y in zip(out, lims)]), changed

        o = U[..., 3:-3, 3:-3]
        lx, tx = direction(o[:, q], M[:, 3:-3, 4:-2] - b, b - M[:, 3:-3, 2:-4], 1)
        ly, ty = direction(o[:, 1], M[:, 4:-2, 3:-3] - b, b - M[:, 2:-4, 3:-3], 2)
        o[:, q] = torch.where(tx, lx, o[:, q])
        o[:, 1] = torch.where(ty, ly, o[:, 1])
        for m in range(q * q):
            if m // q + m % q > 1:
                o[:, m] = torch.where(tx | ty, torch.zeros_like(b), o[:, m])

    def step(self, U, dt):
        cur = U
        for a, b in ((0.0, 1.0), (0.75, 0.25), (1.0 / 3.0, 2.0 / 3.0)):
            V = self.fill(cur)
            d = dt * self.dg_rhs(V) if self.c["method"] == "dg" else self.weno_rhs(V, dt)
            cur = U + d if a == 0.0 else a * U + b * (V + d)
            if self.c["limiter"] == "reference":
                self.limit_reference(cur)
            elif self.c["limiter"] == "tvb":
                self.limit_tvb(cur)
        return cur


def exact(case, seed):
    c = case
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if c["kind"] == "batch":
        out = []
        for m, s in _batch_members(c, seed):
            X, U = _Exact(m, device), _initial(m, s, device)
            for _ in range(m["steps"]):
                U = X.step(U, _dt(m, X.da, X.max_speed(U)))
            out.append(U)
        return out
    if c["limiter"] == "tvb_mlp":
        return None  # which cells are limited is a BF16 network's decision
    X, U = _Exact(c, device), _initial(c, seed, device)
    lam = X.max_speed(U)
    dt = _dt(c, X.da, lam)
    for _ in range(c["steps"]):
        U = X.step(U, dt)
    return {"state": U} if c["fixed_dt"] else {"state": U, "max_speed": lam}
