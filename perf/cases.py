"""Performance cases of the flux-reconstruction solver.

Each case is work that a user of the library has it do, through its public entry points: time
steps from a given vorticity (``HO_2D``), an outer step of the coupled (hybrid) operation,
gradients by the discrete adjoint (``ho2d.adjoint.rollout``), and the Poisson operator on the
caller's own device buffers. ``listed`` names the fixed ones, ``draw`` gives more of the same
ranges, ``prepare`` makes what a user's program holds before the call, ``run`` is one pass,
``work`` the bytes and operations a pass cannot do without, and ``exact`` the answer in 64 bits
from plain torch, for the lid-driven cavities (the meshes with a logical n x n grid).

A case is a dict of plain values:

kind        "steps", "gradient", "hybrid" or "operator"
mesh        "cavity<n>", "cavityj<n>" (interior nodes moved by +/-0.1h), "bfs<m>" (backward-facing
            step of h = 1/m; m = 15 has 14,625 quads), "cyl<nr>x<nt>" (O-grid), "channel<nr>x<nt>"
            (cylinder in a channel) or "annulus<nr>x<nt>" (wall inside, open boundary outside)
knod        solution points per direction, K = P + 1
reyn        Reynolds number
precision   "fp64", "mixed" or "mixed_krylov"
smoother    of the FP32 preconditioner: "blocks", "bf16" or "kron" (steps in the mixed modes)
rk, adv     time integrator (1, 2, 4) and advection scheme (1, 2)
steps       time steps of a pass
ckpt, fp32  checkpoint interval and FP32 storage of the adjoint's states (gradient)
"""

from __future__ import annotations

import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ho-cxx_b200"))

from ho2d import FP64, HO_2D, MIXED, MIXED_KRYLOV, capi, meshgen  # noqa: E402
from ho2d.adjoint import rollout  # noqa: E402
from ho2d.adjoint_case import cavity_dt  # noqa: E402

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
PRECISION = {"fp64": FP64, "mixed": MIXED, "mixed_krylov": MIXED_KRYLOV}
SMOOTHER = {"blocks": capi.SMOOTHER_BLOCKS, "bf16": capi.SMOOTHER_BF16, "kron": capi.SMOOTHER_KRON}


def _steps(name, mesh, knod, reyn, precision, smoother, steps, rk=4, adv=1):
    return dict(name=name, kind="steps", mesh=mesh, knod=knod, reyn=reyn, precision=precision, smoother=smoother,
                rk=rk, adv=adv, steps=steps)


def listed():
    return [
        # the smallest run, where launches and latency count: the 16 x 16 cavity that the CPU code runs for
        # 2,000 steps, a stretch of 20 of them
        _steps("cavity16_k4_fp64", "cavity16", 4, 100.0, "fp64", "blocks", 20),
        # an odd, small mesh at low order with the continuous-flux advection and RK2, default smoother
        _steps("cavityj37_k3_adv2_krylov", "cavityj37", 3, 400.0, "mixed_krylov", "blocks", 10, rk=2, adv=2),
        # the shedding run's channel (73,728 points, pulsatile inflow), which takes tens of thousands of steps
        _steps("channel48x96_k4_mixed", "channel48x96", 4, 100.0, "mixed", "kron", 10),
        # the backward-facing step of 14,625 jittered quads, FP64 and mixed side by side: an ordinary mesh
        _steps("bfs15_k5_fp64", "bfs15", 5, 400.0, "fp64", "blocks", 6),
        _steps("bfs15_k5_mixed", "bfs15", 5, 400.0, "mixed", "kron", 6),
        # the large cylinder O-grid (4.7M points), the benchmark's workload, in both precisions
        _steps("cyl256x512_k6_mixed", "cyl256x512", 6, 100.0, "mixed", "kron", 4),
        _steps("cyl256x512_k6_fp64", "cyl256x512", 6, 100.0, "fp64", "blocks", 3),
        # the largest mesh: a jittered cavity of 12.8M points at high order, a step of it. (FP64: the FP32
        # inner solves of the mixed modes break down on such a mesh for some start fields.)
        _steps("cavityj512_k7_fp64", "cavityj512", 7, 5000.0, "fp64", "blocks", 1),
        # gradients of a final-time objective: the differentiation case's mesh in FP64, and a larger jittered
        # one with the mixed Poisson solves and FP32 states
        dict(name="gradient64_k5_fp64", kind="gradient", mesh="cavity64", knod=5, reyn=1000.0, precision="fp64",
             steps=4, ckpt=2, fp32=False),
        dict(name="gradientj80_k5_krylov", kind="gradient", mesh="cavityj80", knod=5, reyn=5000.0,
             precision="mixed_krylov", steps=4, ckpt=2, fp32=True),
        # one outer step of a vortex-method coupling: 10 RK2 steps at the default order 3
        dict(name="hybrid24x96_k3", kind="hybrid", mesh="annulus24x96", knod=3, reyn=200.0, precision="fp64", rk=2,
             steps=10),
        # the Poisson operator on the caller's device buffers: a single short call
        dict(name="operator96_k5", kind="operator", mesh="cavityj96", knod=5, reyn=1000.0, precision="fp64"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "gradient", "hybrid", "operator"])
    precision = rng.choice(["fp64", "mixed", "mixed_krylov"])
    if kind == "operator":
        knod = rng.randint(2, 7)
        return dict(kind=kind, mesh="cavityj%d" % _log(rng, 9, int(math.sqrt(131072 // knod))), knod=knod, reyn=1000.0,
                    precision="fp64")
    if kind == "hybrid":
        nr = rng.randint(6, 40)
        return dict(kind=kind, mesh="annulus%dx%d" % (nr, rng.randint(24, 160)), knod=rng.choice([3, 3, 4]),
                    reyn=float(rng.randint(50, 400)), precision="fp64", rk=2, steps=rng.randint(4, 12))
    if kind == "gradient":
        precision = rng.choice(["fp64", "mixed_krylov"])
        knod = rng.randint(3, 7 if precision == "fp64" else 5)
        family = rng.choice(["cavity", "cavityj"]) if precision == "fp64" else "cavity"
        return dict(kind=kind, mesh="%s%d" % (family, _log(rng, 10, 64)), knod=knod,
                    reyn=float(rng.randint(200, 5000)), precision=precision,
                    steps=rng.randint(2, 4), ckpt=rng.randint(1, 3), fp32=rng.random() < 0.5)
    smoother = rng.choice(["blocks", "bf16", "kron", "kron"]) if precision != "fp64" else "blocks"
    family = rng.choice(["cavity", "cavityj", "cavityj", "bfs", "cyl", "channel"])
    if family == "cavityj" and precision != "fp64":
        family = "cavity"  # (as above)
    if family.startswith("cavity"):
        knod = rng.randint(3, 7 if precision == "fp64" else 5)
        return dict(kind=kind, mesh="%s%d" % (family, _log(rng, 8, 256)), knod=knod, reyn=float(rng.randint(100, 5000)),
                    precision=precision, smoother=smoother, rk=rng.choice([2, 4, 4]), adv=rng.choice([1, 1, 2]),
                    steps=rng.randint(1, 4))
    if family == "bfs":
        return dict(kind=kind, mesh="bfs%d" % rng.randint(4, 24), knod=rng.randint(3, 6), reyn=float(rng.randint(100, 600)),
                    precision=precision, smoother=smoother, rk=4, adv=rng.choice([1, 1, 2]), steps=rng.randint(2, 6))
    if family == "channel":
        nr = _log(rng, 16, 64)
        return dict(kind=kind, mesh="channel%dx%d" % (nr, 2 * nr), knod=rng.randint(3, 5), reyn=100.0,
                    precision=precision, smoother=smoother, rk=4, adv=1, steps=rng.randint(2, 10))
    nr = _log(rng, 24, 256)
    return dict(kind=kind, mesh="cyl%dx%d" % (nr, rng.choice([nr + 1, 2 * nr, 2 * nr + 3])), knod=rng.randint(4, 6),
                reyn=100.0, precision=precision, smoother=smoother, rk=4, adv=1, steps=rng.randint(1, 4))


# ------------------------------------------------------------------------------ preparation
def _split(mesh):
    family = mesh.rstrip("0123456789x")
    return family, [int(v) for v in mesh[len(family):].split("x")]


def _start_time(case):
    """Early in the pulsatile inflow's cycle, as the runs of the step and of the cylinder begin: later the inflow
    dominates the Poisson right-hand side, and with it the norm that the solver's tolerance is relative to."""
    return {"bfs": 0.1, "channel": 0.0005, "cyl": 0.0005}.get(_split(case["mesh"])[0], 0.0)


def _dt(case, mesh):
    family, size = _split(case["mesh"])
    if family in ("cavity", "cavityj"):
        return cavity_dt(size[0], case["knod"], reyn=case["reyn"], jitter=0.1 if family == "cavityj" else 0.0)
    speed = {"bfs": 1.5, "annulus": 2.5}.get(family, 2.0)
    return min(meshgen.cfl_dt(mesh, case["knod"], speed), meshgen.viscous_dt(mesh, case["knod"], case["reyn"]))


def _mesh(case):
    family, size = _split(case["mesh"])
    if family == "cavity":
        return meshgen.cavity(size[0])
    if family == "cavityj":
        return meshgen.cavity(size[0], jitter=0.1, seed=5)
    if family == "bfs":
        return meshgen.backward_facing_step(h=1.0 / size[0], x_in=-5.0, x_out=30.0)
    if family == "channel":
        return meshgen.cylinder_channel(*size)
    return meshgen.cylinder_ogrid(size[0], size[1], r1=20.0 if family == "cyl" else 3.0,
                                  stretch=1.02 if family == "cyl" else 1.05)


def _solver(case):
    """A set-up solver of the case, from an input file and its mesh as a user has them on disk."""
    mesh = _mesh(case)
    ptype = {"cavity": 1, "cavityj": 1, "bfs": 2}.get(_split(case["mesh"])[0], 3)
    s = HO_2D()
    with tempfile.TemporaryDirectory() as d:
        meshgen.write_msh(mesh, os.path.join(d, "mesh.msh"))
        path = os.path.join(d, "input.dat")
        meshgen.write_input_dat(path, "mesh.msh", case["knod"], case["reyn"], _dt(case, mesh), 1, ptype,
                                time_integration=case.get("rk", 4), advection_type=case.get("adv", 1))
        s.read_input_file(path)
        s.set_precision(PRECISION[case["precision"]])
        if "smoother" in case:
            s.set_smoother(SMOOTHER[case["smoother"]])
        if case["kind"] == "gradient":
            s.set_poisson_tolerance(1e-13, 2000)  # as the differentiation case does
        s.setup()
    if case["kind"] == "gradient":
        s.set_adjoint_storage(case["fp32"])
    return s


_kept = {}


def _kept_solver(case):
    """The program's one solver of this mesh and its solution points: set up once, given new fields after that."""
    key = repr(sorted((k, v) for k, v in case.items() if k not in ("name", "steps", "ckpt")))
    if key not in _kept:
        while len(_kept) >= 24:
            _kept.pop(next(iter(_kept)))[0].close()
        s = _solver(case)
        if case["kind"] == "steps" and _split(case["mesh"])[0].startswith("cavity"):
            # the regularised lid, u(x) = 16 x^2 (1 - x)^2
            b = s.get_boundary_points()
            s.set_boundary(capi.BC_PARL_VEL, np.where(b[..., 1] > 1.0 - 1e-9, -_lid(b[..., 0]), 0.0))
        _kept[key] = (s, s.getsolnpts_d())
    return _kept[key]


def _lid(x):
    return 16.0 * (x * (1.0 - x)) ** 2


def _streamfunction(case, seed):
    """psi(x, y) of a flow in mid-run, which meets the walls without slip: the mean flow of the case's
    boundaries and seeded eddies of both signs, each with psi' = 0 on a no-slip wall."""
    family, _ = _split(case["mesh"])
    rng = np.random.Generator(np.random.PCG64(seed))
    flow = 2.0 * abs(math.sin(math.pi * _start_time(case) / 40.0))  # inflow speed of problem types 2 and 3
    if family in ("cavity", "cavityj"):
        m = np.arange(1, 5)
        c = 0.05 * rng.standard_normal((4, 4)) / (m[:, None] ** 2 + m[None, :] ** 2)

        def psi(x, y):
            sx, sy = ([torch.sin(math.pi * k * z) for k in m] for z in (x, y))
            eddies = sum(sx[i] * sum(c[i, j] * sy[j] for j in range(4)) for i in range(4))
            return 16.0 * x * (1 - x) * y * (1 - y) * eddies - 16.0 * (x * (1 - x)) ** 2 * y ** 2 * (1 - y)
        return psi
    centres = []
    for _ in range(6):
        if family == "bfs":
            centres.append((rng.uniform(2.0, 12.0), rng.uniform(-0.6, 0.6), rng.uniform(0.2, 0.5), rng.normal(0.0, 0.05)))
        else:
            a, d = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(1.0, 2.5)
            centres.append((d * math.cos(a), d * math.sin(a), rng.uniform(0.4, 0.9), rng.normal(0.0, 2.0)))

    def eddies(x, y):
        return sum(a * torch.exp(-((x - cx) ** 2 + (y - cy) ** 2) / r ** 2) for cx, cy, r, a in centres)

    if family == "bfs":
        def psi(x, y):
            s = torch.clamp(x / 6.0, 0.0, 1.0)
            floor = -s * s * s * (10.0 - 15.0 * s + 6.0 * s * s)  # the stream fills the step over six heights
            e = torch.clamp((y - floor) / (1.0 - floor), min=0.0)
            return flow * e * e * (3.0 - 2.0 * e) + ((1.0 - y) * (1.0 + y)) ** 2 * eddies(x, y)
        return psi

    def psi(x, y):
        near = 1.0 - torch.exp(-((torch.hypot(x, y) - 0.5) / 0.5) ** 2)
        return near * (flow * y + eddies(x, y))
    return psi


def _vorticity(case, xy, seed):
    """The start of a pass: the sine spectrum for the gradients, as in the differentiation case, else the
    vorticity -lap psi of _streamfunction, by fourth-order differences."""
    if case["kind"] == "gradient":
        return meshgen.sine_spectrum(xy, seed=seed)
    psi, h = _streamfunction(case, seed), 1e-3
    p = torch.from_numpy(xy).to(DEVICE)
    x, y = p[..., 0].contiguous(), p[..., 1].contiguous()
    w = 5.0 * psi(x, y)  # 2 x 30 / 12
    for d, c in ((h, -16.0), (2.0 * h, 1.0)):
        w = w + c / 12.0 * (psi(x + d, y) + psi(x - d, y) + psi(x, y + d) + psi(x, y - d))
    return (w / h ** 2).cpu().numpy()


def prepare(case, seed):
    if case["kind"] == "hybrid":
        return _prepare_hybrid(case, seed)
    s, xy = _kept_solver(case)
    state = {"case": case, "solver": s, "t0": _start_time(case)}
    if case["kind"] == "operator":
        g = torch.Generator(device="cuda").manual_seed(seed)
        state["x"] = torch.randn(xy.shape[:-1], generator=g, device="cuda", dtype=torch.float64)
        state["y"] = torch.empty_like(state["x"])
        return state
    state["w0"] = _vorticity(case, xy, seed)
    if case["kind"] == "gradient":
        # lid of the differentiation case: u(x) = 1 + sum a_m sin(m pi x); the target from another seed
        lid = s.get_boundary_points()[..., 1] > 1.0 - 1e-9
        u = meshgen.lid_velocity(s.get_boundary_points()[..., 0], meshgen.lid_coefficients(seed=seed + 41))
        state["pv"] = torch.from_numpy(np.where(lid, -u, 0.0))
        state["w0"] = torch.from_numpy(state["w0"])
        state["target"] = torch.from_numpy(meshgen.sine_spectrum(xy, seed=seed + 42))
    return state


def _prepare_hybrid(case, seed):
    """The arrays an outer vortex-method driver hands over, and the solver it has set up with them."""
    _, (nr, nt) = _split(case["mesh"])
    mesh = _mesh(case)
    s = HO_2D()
    s.set_defaults()
    s.enable_hybrid()
    s.set_elemorder(case["knod"])
    outer = np.concatenate([mesh.boundaries["inlet"], mesh.boundaries["outlet"]])
    s.load_mesh_arrays_d(1, mesh.xy, mesh.quads, mesh.boundaries["object"], outer)
    s.load_inout_arrays_d()
    s.process_mesh_input()
    rng = np.random.Generator(np.random.PCG64(seed))
    xy, pts = s.getsolnpts_d(), s.getopenpts_d()
    z = pts[..., 0] + 1j * pts[..., 1]
    w = (1.0 - 0.25 / z ** 2) + 0.05 * sum(rng.normal() / z ** k for k in range(1, 5))  # potential flow, disturbed
    vel = np.stack([w.real, -w.imag], -1)
    r = np.hypot(xy[..., 0], xy[..., 1])
    target = 0.5 * np.exp(-((xy[..., 0] - rng.uniform(1.0, 2.0)) ** 2 + (xy[..., 1] - rng.normal(0.0, 0.5)) ** 2) / 0.3)
    return {"case": case, "solver": s, "dt": _dt(case, mesh), "vel": vel, "openvort": np.zeros(pts.shape[:-1]),
            "target": target, "weights": np.clip((r - 2.0) / 1.0, 0.0, 1.0) ** 2}


# ------------------------------------------------------------------------------ one pass
def run(state):
    case, s = state["case"], state["solver"]
    if case["kind"] == "steps":
        s.set_time(state["t0"])
        s.set_vorticity(state["w0"])
        s.solve_advection_diffusion(case["steps"])
        return {"vorticity": s.get_vorticity()}
    if case["kind"] == "gradient":
        s.set_time(state["t0"])
        w0, pv = state["w0"].clone().requires_grad_(), state["pv"].clone().requires_grad_()
        w1 = rollout(s, w0, pv, case["steps"], case["ckpt"])
        (0.5 * ((w1 - state["target"]) ** 2).sum()).backward()
        return {"vorticity": w1.detach(), "grad_vorticity": w0.grad, "grad_wall": pv.grad}
    if case["kind"] == "hybrid":
        s.setsolnvort_d(state["target"])
        s.setopenvels_d(state["vel"])
        s.setopenvort_d(state["openvort"])
        s.setptogweights_d(state["weights"])
        s.solveto_d(case["steps"] * state["dt"], case["steps"], case["rk"], case["reyn"])
        return {"vorticity": s.getallvorts_d()}
    x, y = state["x"], state["y"]
    torch.cuda.current_stream().synchronize()  # the entry point wants x complete; it returns with y complete
    code = s._lib.ho2d_apply_poisson_noalloc(s._h, x.numel(), x.data_ptr(), y.data_ptr())
    if code:
        raise RuntimeError("ho2d_apply_poisson_noalloc: %d" % code)
    return {"y": y}


def _elements(case):
    family, size = _split(case["mesh"])
    if family in ("cavity", "cavityj"):
        return size[0] ** 2
    if family == "bfs":
        return 5 * size[0] * size[0] + 30 * size[0] * 2 * size[0]
    return size[0] * size[1]


def work(case):
    """Per stage: the vorticity in and the stage value out, the streamfunction out, eight metric and
    operator coefficients a point, and the contractions of the residual, the velocity and one application
    of the Poisson operator (a solve applies it a number of times that depends on the method)."""
    k, n = case["knod"], _elements(case)
    dof = n * k * k
    if case["kind"] == "operator":
        return {"bytes": 8.0 * (5 * dof + 16 * n * k), "flops": dof * (16.0 * k + 20.0)}
    wide = 4 if case["precision"] == "mixed" else 8
    stages = {1: 1, 2: 2, 4: 4}[case.get("rk", 4)] * case["steps"]
    sweeps = 4 if case["kind"] == "gradient" else 1  # forward, recomputation, and the transpose twice as heavy
    return {"bytes": sweeps * stages * dof * (3.0 * 8 + 8.0 * wide) + 16.0 * dof,
            "flops": sweeps * stages * dof * 3 * (16.0 * k + 20.0)}


# ------------------------------------------------------------------------------ 64-bit answers
class _Cavity:
    """The discretisation on an n x n cavity in torch, 64 bits: fields [row][column][j][i], method-2 flux
    reconstruction, the Poisson problem by a block-tridiagonal factorisation over the rows of elements."""

    def __init__(self, case):
        family, (n,) = _split(case["mesh"])
        mesh = _mesh(case)
        K = self.K = case["knod"]
        self.n, self.re_inv, self.dt = n, 1.0 / case["reyn"], _dt(case, mesh)
        self.rk, self.adv = case.get("rk", 4), case.get("adv", 1)
        x, wq = np.polynomial.legendre.leggauss(K)
        P = lambda m, t: np.polynomial.legendre.legval(t, [0.0] * m + [1.0])  # noqa: E731
        c = np.linalg.inv(np.vander(x, increasing=True))  # Lagrange coefficients [power][k]
        van = lambda t: np.vander(np.atleast_1d(t), K, increasing=True)  # noqa: E731
        dvan = lambda t: np.stack([m * np.atleast_1d(t) ** max(m - 1, 0) for m in range(K)], 1)  # noqa: E731
        ends = np.array([-1.0, 1.0])
        s, cd = 0.5 * (-1.0) ** K, 0.5 * K * (-1.0) ** K
        # corrections and their derivatives: Radau polynomials of the left and the right end
        R = np.stack([s * (P(K, x) - P(K - 1, x)), s * (P(K, -x) - P(K - 1, -x))], 1)
        gR = np.stack([cd * (P(K, x) + P(K - 1, x)) / (1 + x), -cd * (P(K, -x) + P(K - 1, -x)) / (1 - x)], 1)
        dev = DEVICE
        t = lambda a: torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.t = t
        self.end, self.dend = t((van(ends) @ c).T), t((dvan(ends) @ c).T)  # [k][end]
        self.D, self.R, self.gR = t((dvan(x) @ c).T), t(R), t(gR)          # D[m][i] = l_m'(x_i)
        self.gp = [-0.5 * K * (K + 1.0), 0.5 * K * (K + 1.0)]
        X = mesh.xy.reshape(n + 1, n + 1, 2)
        corner = t(np.stack([np.stack([X[:-1, :-1], X[:-1, 1:]], 2), np.stack([X[1:, :-1], X[1:, 1:]], 2)], 2))
        lin = lambda v: t(np.stack([(1 - v) / 2, (1 + v) / 2]))  # noqa: E731  [node][point]
        dl = t(np.array([-0.5, 0.5]))

        def jac(px, py):  # derivatives along xi and eta at (px, py): [..][len py][len px][x, y]
            a = torch.einsum("yxqpc,p,qj->yxjc", corner, dl, lin(py)).unsqueeze(3).expand(-1, -1, -1, len(px), -1)
            b = torch.einsum("yxqpc,q,pi->yxic", corner, dl, lin(px)).unsqueeze(2).expand(-1, -1, len(py), -1, -1)
            return a, b

        a, b = jac(x, x)
        self.xxi, self.yxi, self.xet, self.yet = a[..., 0], a[..., 1], b[..., 0], b[..., 1]
        self.J = self.xxi * self.yet - self.xet * self.yxi
        fA, fB, fJ = [], [], []
        for f in range(4):
            e = ends[f & 1:(f & 1) + 1]
            a, b = jac(e, x) if f < 2 else jac(x, e)
            a, b = a.reshape(n, n, K, 2), b.reshape(n, n, K, 2)
            fJ.append(a[..., 0] * b[..., 1] - b[..., 0] * a[..., 1])
            fA.append(((b if f < 2 else a) ** 2).sum(-1))
            fB.append((a * b).sum(-1))
        self.fA, self.fB, self.fJ = (torch.stack(v, 2) for v in (fA, fB, fJ))  # [n][n][face][k]
        self.fn = self.fA.sqrt()
        inner = torch.ones(n, n, 4, 1, dtype=torch.bool, device=dev)
        inner[:, 0, 0] = inner[:, -1, 1] = inner[0, :, 2] = inner[-1, :, 3] = False
        self.inner = inner
        self.sgn = t([-1.0, 1.0, -1.0, 1.0]).reshape(4, 1)
        self.w = t(wq)
        self.neu = None
        self.lid = torch.zeros(n, n, 4, K, dtype=torch.float64, device=dev)
        xs = torch.einsum("xp,pi->xi", self.t(X[-1, :, 0]).unfold(0, 2, 1), lin(x))
        self.lid[-1, :, 3] = -_lid(xs)

    def faces(self, a, b):
        """Traces: a at the W and E ends of its rows, b at the S and N ends of its columns."""
        we, sn = a @ self.end, torch.einsum("yxji,je->yxie", b, self.end)
        return torch.stack([we[..., 0], we[..., 1], sn[..., 0], sn[..., 1]], 2)

    def dfaces(self, f):
        we, sn = f @ self.dend, torch.einsum("yxji,je->yxie", f, self.dend)
        return torch.stack([we[..., 0], we[..., 1], sn[..., 0], sn[..., 1]], 2)

    @staticmethod
    def other(v):
        """The neighbour's value at each face (the domain's edge gets its opposite side's, masked by the caller)."""
        return torch.stack([v[:, :, 1].roll(1, 1), v[:, :, 0].roll(-1, 1), v[:, :, 3].roll(1, 0), v[:, :, 2].roll(-1, 0)], 2)

    def ddx(self, f):
        return f @ self.D

    def ddy(self, f):
        return torch.einsum("yxdi,dj->yxji", f, self.D)

    def lift(self, c, w, z):
        """Correction of the jumps c[face] at the W and E ends (rows) or S and N ends (columns)."""
        if w == 0:
            return c[:, :, 0].unsqueeze(3) * z[:, 0] + c[:, :, 1].unsqueeze(3) * z[:, 1]
        return c[:, :, 2].unsqueeze(2) * z[:, 0].unsqueeze(1) + c[:, :, 3].unsqueeze(2) * z[:, 1].unsqueeze(1)

    def common(self, v, g, neumann=None):
        """Common values and normal fluxes of method 2; on the walls a zero value or, with `neumann`, the
        normal derivative it gives."""
        gp = self.t(self.gp * 2).reshape(4, 1)
        com = torch.where(self.inner, 0.5 * (v + self.other(v)), torch.zeros_like(v))
        if neumann is not None:
            cg = neumann * self.fn
            rhs = self.fJ * cg - self.fA * (g - v * gp)
            if self.neu is None:
                m = -self.fB.unsqueeze(-1) * self.D.T + torch.diag_embed(self.fA * gp)
                self.neu = torch.linalg.inv(m)
            com = torch.where(self.inner, com, (self.neu @ rhs.unsqueeze(-1)).squeeze(-1))
        flux = ((g + (com - v) * gp) * self.fA - (com @ self.D) * self.fB) / self.fJ
        mean = 0.5 * (flux + self.other(flux))
        return com, torch.where(self.inner, mean, flux if neumann is None else cg)

    def gradient(self, f, com, v):
        """Contravariant gradient f~, g~ (times the Jacobian)."""
        dx, de = self.ddx(f) + self.lift(com - v, 0, self.gR), self.ddy(f) + self.lift(com - v, 1, self.gR)
        cross = self.xxi * self.xet + self.yxi * self.yet
        return ((dx * (self.xet ** 2 + self.yet ** 2) - de * cross) / self.J,
                (de * (self.xxi ** 2 + self.yxi ** 2) - dx * cross) / self.J)

    def laplacian(self, f, neumann=None):
        v, g = self.faces(f, f), self.dfaces(f)
        com, cg = self.common(v, g, neumann)
        a, b = self.gradient(f, com, v)
        jump = cg - self.faces(a, b)
        return self.ddx(a) + self.ddy(b) + self.lift(jump, 0, self.gR) + self.lift(jump, 1, self.gR), com

    def factor(self):
        """Block-tridiagonal factors of the Poisson operator, probed with five colours of elements."""
        n, K2 = self.n, self.K ** 2
        m = n * K2
        jj, ii = torch.meshgrid(torch.arange(n), torch.arange(n), indexing="ij")
        colour = ((ii + 2 * jj) % 5).to(self.J.device)
        diag = torch.zeros(n, n, K2, n, K2, dtype=torch.float64, device=self.J.device)  # [row][el, dof][el, dof]
        low = torch.zeros(n, n, K2, K2, dtype=torch.float64, device=self.J.device)
        up = torch.zeros_like(low)
        col = torch.arange(n, device=self.J.device)
        for c in range(5):
            for q in range(K2):
                x = torch.zeros(n, n, K2, dtype=torch.float64, device=self.J.device)
                x[..., q] = (colour == c).double()
                y = self.laplacian(x.reshape(n, n, self.K, self.K))[0].reshape(n, n, K2)
                for dj, di in ((0, 0), (0, 1), (0, -1), (1, 0), (-1, 0)):
                    # rows of the elements whose neighbour at (dj, di) has this colour
                    src = ((ii + di) + 2 * (jj + dj)).to(self.J.device) % 5 == c
                    ok = src & ((ii + di >= 0) & (ii + di < n) & (jj + dj >= 0) & (jj + dj < n)).to(self.J.device)
                    r, e = torch.nonzero(ok, as_tuple=True)
                    if dj == 0:
                        diag[r, e, :, col[e] + di, q] = y[r, e]
                    elif dj < 0:
                        low[r, e, :, q] = y[r, e]
                    else:
                        up[r, e, :, q] = y[r, e]
        self.low, self.up, self.lu = low, up, []
        for j in range(n):
            d = diag[j].reshape(m, m)
            if j:
                # low_j S^-1 up_{j-1}, both block diagonal over the elements of a row
                w = torch.linalg.lu_solve(*self.lu[-1], torch.block_diag(*up[j - 1]))
                d = d - torch.einsum("epq,eqc->epc", low[j], w.reshape(n, K2, m)).reshape(m, m)
            self.lu.append(torch.linalg.lu_factor(d))

    def tri(self, b, transpose=False):
        n, K2 = self.n, self.K ** 2
        b = b.reshape(n, n, K2)
        lo, up = (self.up.transpose(-1, -2), self.low.transpose(-1, -2)) if transpose else (self.low, self.up)
        # transposed: row j couples to j-1 through up[j-1]^T and to j+1 through low[j+1]^T
        solve = lambda j, r: torch.linalg.lu_solve(*self.lu[j], r.reshape(-1, 1), adjoint=transpose).reshape(n, K2)  # noqa: E731
        at = (lambda j: (j - 1, j + 1)) if transpose else (lambda j: (j, j))
        z = [None] * n
        for j in range(n):
            r = b[j]
            if j:
                r = r - torch.einsum("epq,eq->ep", lo[at(j)[0]], z[j - 1])
            z[j] = solve(j, r)
        for j in range(n - 2, -1, -1):
            z[j] = z[j] - solve(j, torch.einsum("epq,eq->ep", up[at(j)[1]], z[j + 1]))
        return torch.stack(z).reshape(n, n, self.K, self.K)

    def poisson(self, rhs):
        return _Solve.apply(rhs, self)

    def stage(self, w):
        psi = self.poisson(-w * self.J)
        v, g = self.faces(psi, psi), self.dfaces(psi)
        com, cg = self.common(v, g)
        a, b = self.gradient(psi, com, v)
        jump = cg - self.faces(a, b)
        tx, ty = a + self.lift(jump, 0, self.R), b + self.lift(jump, 1, self.R)
        us = (tx * self.yxi + ty * self.yet) / self.J
        vs = -(tx * self.xxi + ty * self.xet) / self.J
        slip = cg / self.fn + self.sgn * self.lid
        lap, _ = self.laplacian(w, slip / (self.dt * self.re_inv))
        diff = lap * self.re_inv / self.J
        ux, uy = us * self.yet - vs * self.xet, -us * self.yxi + vs * self.xxi
        uf, wf = self.faces(ux, uy), self.faces(w, w)
        zero = torch.zeros_like(uf)
        if self.adv == 1:
            fx, fy = ux * w, uy * w
            own = torch.where(self.inner, uf * wf, zero)
            far, dw = self.other(own), wf - self.other(wf)
            big = dw.abs() > 1e-4
            speed = torch.where(big, (own - far) / torch.where(big, dw, torch.ones_like(dw)), zero)
            up = 0.5 * (own + far) + torch.where(big, 0.5 * self.sgn * speed.abs() * dw, zero)
        else:
            cv = torch.where(self.inner, 0.5 * (uf + self.other(uf)), zero)
            ux, uy = ux + self.lift(cv - uf, 0, self.R), uy + self.lift(cv - uf, 1, self.R)
            fx, fy = ux * w, uy * w
            side = self.sgn > 0
            up = cv * torch.where((cv > 0) == side, wf, self.other(wf))
        up = torch.where(self.inner, up, zero)
        jump = up - self.faces(fx, fy)
        div = self.ddx(fx) + self.ddy(fy) + self.lift(jump, 0, self.gR) + self.lift(jump, 1, self.gR)
        return self.dt * (diff - div / self.J)

    def step(self, w):
        if self.rk == 1:
            return w + self.stage(w)
        k1 = self.stage(w)
        if self.rk == 2:
            return w + 0.5 * (k1 + self.stage(w + k1))
        k2 = self.stage(w + 0.5 * k1)
        k3 = self.stage(w + 0.5 * k2)
        return w + (k1 + 2.0 * k2 + 2.0 * k3 + self.stage(w + k3)) / 6.0


class _Solve(torch.autograd.Function):
    @staticmethod
    def forward(ctx, rhs, cavity):
        ctx.cavity = cavity
        psi = cavity.tri(rhs)
        return psi + cavity.tri(rhs - cavity.laplacian(psi)[0])  # one step of refinement

    @staticmethod
    def backward(ctx, g):
        return ctx.cavity.tri(g.contiguous(), transpose=True), None


def exact(case, seed):
    """What run() returns, in 64 bits from the discretisation written out in torch above. Cavities only, of
    a size whose factorisation takes a few seconds; the other meshes and the coupled operation have none."""
    family, size = _split(case["mesh"])
    if family not in ("cavity", "cavityj"):
        return None
    n, K = size[0], case["knod"]
    if case["kind"] != "operator" and n * K * K > 2400:
        return None
    c = _Cavity(case)
    shape = (n * n, K, K)
    state = prepare(case, seed)
    if case["kind"] == "operator":
        with torch.no_grad():
            return {"y": c.laplacian(state["x"].reshape(n, n, K, K))[0].reshape(shape)}
    with torch.no_grad():
        c.factor()
    w0 = c.t(np.asarray(state["w0"])).reshape(n, n, K, K)
    if case["kind"] == "steps":
        with torch.no_grad():
            w = w0
            for _ in range(case["steps"]):
                w = c.step(w)
        return {"vorticity": w.reshape(shape)}
    # the wall velocity [edge][k] in the mesh file's edge order: bottom, right, top, left (each counter-clockwise)
    pv = state["pv"].to(w0.device).clone().requires_grad_()
    w0.requires_grad_()
    order = _wall_order(case, state["solver"], c)
    c.lid = torch.zeros(n * n * 4 * K, dtype=torch.float64, device=w0.device).index_put(
        (order,), pv.reshape(-1)).reshape(n, n, 4, K)
    w = w0
    for _ in range(case["steps"]):
        w = c.step(w)
    target = c.t(state["target"].numpy()).reshape(w.shape)
    (0.5 * ((w - target) ** 2).sum()).backward()
    return {"vorticity": w.detach().reshape(shape), "grad_vorticity": w0.grad.reshape(shape), "grad_wall": pv.grad}


def _wall_order(case, solver, c):
    """Where each wall point [edge][k] of the boundary arrays lies in a field [row][column][face][k]."""
    n, K = c.n, c.K
    p = solver.get_boundary_points().reshape(-1, 2)
    X = _mesh(case).xy.reshape(n + 1, n + 1, 2)
    g = 0.5 * (1.0 + np.polynomial.legendre.leggauss(K)[0])
    where = {}
    for i in range(n):
        for k in range(K):
            for face, el, a, b in ((2, i, X[0, i], X[0, i + 1]), (3, (n - 1) * n + i, X[n, i], X[n, i + 1]),
                                   (0, i * n, X[i, 0], X[i + 1, 0]), (1, i * n + n - 1, X[i, n], X[i + 1, n])):
                q = a + g[k] * (b - a)
                where[(round(q[0], 9), round(q[1], 9))] = (el * 4 + face) * K + k
    return torch.tensor([where[(round(x, 9), round(y, 9))] for x, y in p], device=c.J.device)
