"""Workloads of the residual / time-integration path, called as a user's program calls them.

A case is one of five ways to use the package on one of four flows:

* kinds: "residual" (one derivative of a host state), "step" (one Advance call from host state to host
  state, what a teal program's own loop does), "run" (a resident run up to an output point),
  "batch" (several meshes advanced in one arena); "run" and "batch" take explicit or implicit methods;
* flows: "vortex" (isentropic vortex, periodic), "tgv" (Navier-Stokes Taylor-Green vortex, periodic),
  "channel" (a wavy stream with a density bump between far fields and a wall), "ramp" (compression
  ramp on a jittered mesh of tetrahedra, prisms, hexahedra and pyramids, far field and slip walls).

The states depend on the seed: phases of the periodic flows, Mach number, angle and a smooth
perturbation of the free streams. `exact` restates the scheme in plain 64-bit torch on the mesh's
arrays (the mesh is an input, not a result).
"""

import functools
import math

import numpy as np
import torch

import teal_b200 as tb
from teal_b200 import meshes

GAMMA, PRANDTL, NEWTON = 1.4, 0.71, (0.1, 0.3, 30)


def listed():
    box = {"ny": 0, "nz": 0, "limiter": "minmod", "precision": "fp64", "method": "lserk", "steps": 1, "cfl": 0.99}

    def case(name, kind, flow, nx, **more):
        return {**box, "name": name, "kind": kind, "flow": flow, "nx": nx, **more}

    return [
        # the smallest call: one residual of a coarse mesh, as a host code couples to the flow solver
        case("residual_channel_20x12x10", "residual", "channel", 20, ny=12, nz=10, flux="hllc"),
        # a residual of an ordinary odd-sized viscous mesh
        case("residual_tgv_61x47x53", "residual", "tgv", 61, ny=47, nz=53, flux="roe", limiter="venkatakrishnan"),
        # the isentropic vortex of the accuracy studies: thousands of short steps, launch-bound
        case("vortex_64x64x4_50_steps", "run", "vortex", 64, ny=64, nz=4, flux="hllc", steps=50, cfl=0.5),
        # teal's own time loop with the device Advance: host state in, host state out, every step
        case("tgv_48_host_step", "step", "tgv", 48, ny=48, nz=48, flux="roe", limiter="venkatakrishnan"),
        # the Taylor-Green vortex at an ordinary and at the headline size, between two outputs
        case("tgv_64_10_steps", "run", "tgv", 64, ny=64, nz=64, flux="roe", limiter="venkatakrishnan", steps=10),
        case("tgv_128_20_steps", "run", "tgv", 128, ny=128, nz=128, flux="roe", limiter="venkatakrishnan", steps=20),
        # the same flow with fluxes in 32 bits
        case("tgv_96_fp32_flux_20_steps", "run", "tgv", 96, ny=96, nz=96, flux="roe", limiter="venkatakrishnan",
             precision="fp32", steps=20),
        # supersonic ramp on the unstructured mesh, explicit
        case("ramp_48_20_steps", "run", "ramp", 48, flux="ausmd", steps=20),
        # parameter study: meshes of uneven size advanced together, 32-bit fluxes
        case("ramp_batch_10_fp32_flux", "batch", "ramp", 24, flux="ausmd", precision="fp32", steps=10, count=10),
        # steady solves by implicit Euler (Newton-GMRES): one mesh, viscous, and a batch with 32-bit matvecs
        case("ramp_20_implicit", "run", "ramp", 20, flux="hllc", limiter="venkatakrishnan",
             method="implicit euler", steps=2, cfl=30.0),
        case("channel_80x64x24_implicit_ns", "run", "channel", 80, ny=64, nz=24, flux="roe",
             limiter="venkatakrishnan", viscosity=1e-3, method="implicit euler", steps=2, cfl=20.0),
        case("ramp_batch_6_implicit_fp32_matvec", "batch", "ramp", 24, flux="hllc", limiter="venkatakrishnan",
             precision="fp32", method="implicit euler", steps=2, cfl=10.0, count=6),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    c = {"limiter": rng.choice(["minmod", "venkatakrishnan"]), "precision": rng.choice(["fp64", "fp64", "fp32"]),
         "flux": rng.choice(["roe", "hllc", "ausmd"]), "method": "lserk", "steps": rng.randint(2, 16), "cfl": 0.9,
         "kind": rng.choice(["residual", "step", "run", "run", "batch", "run", "batch"])}
    c["flow"] = "ramp" if c["kind"] == "batch" else rng.choice(["vortex", "tgv", "channel", "ramp"])
    if c["flow"] == "ramp":
        n = size(9, 40)
        c.update(nx=n, ny=0, nz=0)
    else:
        n = size(14, 100)
        c.update(nx=n, ny=max(6, int(n * rng.uniform(0.6, 1.1))), nz=max(4, int(n * rng.uniform(0.1, 1.0))))
    if c["kind"] == "batch":
        c.update(count=rng.randint(2, 8), nx=min(n, 22))
    if c["kind"] in ("run", "batch") and c["flow"] in ("ramp", "channel") and rng.random() < 0.5:
        c.update(method="implicit euler", steps=rng.randint(1, 3), cfl=10.0, limiter="venkatakrishnan", flux="hllc",
                 nx=min(c["nx"], 64 if c["flow"] == "channel" else 24))
    if c["flow"] == "channel" and rng.random() < 0.5:
        c["viscosity"] = 1e-3
    if c["kind"] in ("residual", "step"):
        c["steps"] = 1
    return c


# ---- what a program has in hand ------------------------------------------------------------------


@functools.lru_cache(maxsize=64)
def _mesh(flow, nx, ny, nz, variant=0):
    """Host mesh (a program builds it once and starts many solves on it)."""
    if flow == "ramp":
        return tb.Mesh.from_cells(meshes.ramp_mesh(n=(nx, nx, nx), seed=variant))
    hi = {"vortex": (10.0, 10.0, 10.0 * nz / nx), "tgv": (2 * math.pi,) * 3, "channel": (nx / ny, 1.0, nz / ny)}[flow]
    return tb.Mesh.create((0, 0, 0), hi, (nx, ny, nz), (0, 0, 1) if flow == "channel" else (1, 1, 1))


def _sizes(case):
    """Grid sizes of the case's meshes: one, or uneven sizes up to nx for a batch."""
    if case["kind"] != "batch":
        return [(case["nx"], case["ny"], case["nz"], 0)]
    k = case["count"]
    return [(max(8, int(round(8 * (case["nx"] / 8) ** (i / max(1, k - 1))))), 0, 0, i) for i in range(k)]


def _state(flow, x, rng):
    """Initial primitive state at the cell centres x and the free stream (None for periodic flows)."""
    out = np.zeros((x.shape[0], 5))
    if flow == "vortex":
        at, beta = rng.uniform(3.5, 6.5, 2), 5.0
        d = (x[:, :2] - at + 5.0) % 10.0 - 5.0
        r2 = (d**2).sum(axis=1)
        out[:, 0] = (1 - (GAMMA - 1) * beta**2 / (8 * GAMMA * np.pi**2) * np.exp(1 - r2)) ** (1 / (GAMMA - 1))
        e = beta / (2 * np.pi) * np.exp((1 - r2) / 2)
        out[:, 1], out[:, 2], out[:, 4] = 1 - e * d[:, 1], 1 + e * d[:, 0], out[:, 0] ** GAMMA
        return out, None
    if flow == "tgv":
        a, b, c = (x + rng.uniform(0, 2 * np.pi, 3)).T
        p0 = 1 / (GAMMA * 0.1**2)
        out[:, 1], out[:, 2] = np.sin(a) * np.cos(b) * np.cos(c), -np.cos(a) * np.sin(b) * np.cos(c)
        out[:, 4] = p0 + (np.cos(2 * a) + np.cos(2 * b)) * (np.cos(2 * c) + 2) / 16
        out[:, 0] = out[:, 4] / p0
        return out, None
    mach, angle = (rng.uniform(1.8, 2.6), 0.0) if flow == "ramp" else (rng.uniform(0.4, 0.7), rng.uniform(0, 0.1))
    free = np.array([1.0, mach * math.cos(angle), mach * math.sin(angle), 0.0, 1 / GAMMA])
    # a flow under way: nowhere uniform, with a density bump
    wave = np.sin(x @ rng.uniform(2, 5, (3, 5)) + rng.uniform(0, 2 * np.pi, 5))
    out[:] = free * (1 + 0.02 * wave)
    out[:, 3] += 0.02 * wave[:, 3]
    r2 = ((x[:, :2] - x[:, :2].mean(axis=0) + rng.uniform(-0.1, 0.1, 2)) ** 2).sum(axis=1) / 0.02
    out[:, 0] *= 1 + 0.2 * np.exp(-r2)
    return out, free


def _viscous(case):
    return case["flow"] == "tgv" or "viscosity" in case


def _problem(case, size, rng):
    mesh = _mesh(case["flow"], *size)
    eqns = (tb.Equations.navierstokes if _viscous(case) else tb.Equations.euler)(mesh)
    eqns.set_convective_flux(case["flux"])
    eqns.set_limiter(case["limiter"], 1.0)
    if _viscous(case):
        eqns.set_property("dynamic viscosity", case.get("viscosity", 1 / 1600))
    state, free = _state(case["flow"], mesh.cell_center[: mesh.num_inner_cells], rng)
    for side, (kind, context) in _boundaries(case, free).items():
        eqns.set_boundary_condition(side, kind, context)
    eqns.primitive[: mesh.num_inner_cells] = state
    return eqns


def _boundaries(case, free):
    """Boundary kinds by side: far field around, a wall below."""
    if free is None:
        return {}
    far, slip = ("farfield", free), ("slipwall", None)
    if case["flow"] == "ramp":
        return {"left": far, "right": far, "top": far, "bottom": slip, "back": slip, "front": slip}
    return {"left": far, "right": far, "top": far, "bottom": ("adiabatic wall", None) if _viscous(case) else slip}


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    precision = tb.TG_PRECISION_FP32_FLUX if case["precision"] == "fp32" else tb.TG_PRECISION_FP64
    method = tb.TG_ADVANCE_LSERK if case["method"] == "lserk" else tb.TG_ADVANCE_IMPLICIT_EULER
    context = (3, 3) if case["method"] == "lserk" else NEWTON
    problems = [_problem(case, size, rng) for size in _sizes(case)]
    state = {"case": case, "args": (method, case["cfl"]), "context": context}
    state["device"] = tb.Batch(problems, precision) if case["kind"] == "batch" else problems[0].context(precision)
    state["problems"], state["in"], state["out"] = problems, [], []
    for p in problems:
        state["in"].append(_pinned(p.primitive.shape))
        state["in"][-1][:] = p.primitive
        state["out"].append(_pinned(p.primitive.shape))
    return state


def run(state):
    case, device, (method, cfl) = state["case"], state["device"], state["args"]
    if case["kind"] == "residual":
        return device.derivative(state["in"][0])
    if case["kind"] == "step":
        time, step, residual = device.advance_host(method, cfl, 0.0, state["in"][0], state["out"][0],
                                                   context=state["context"])
        return {"primitive": state["out"][0], "time": time, "step": step, "residual": residual}
    if case["kind"] == "run":
        device.set_primitive(state["in"][0])
        time, steps, residual = device.run(method, cfl, case["steps"], context=state["context"])
        device.get_primitive(state["out"][0])
        return {"primitive": state["out"][0], "time": time, "steps": steps, "residual": residual}
    for i, primitive in enumerate(state["in"]):
        device.set_primitive(i, primitive)
    time, steps, residual = device.run(method, cfl, case["steps"], context=state["context"])
    for i, out in enumerate(state["out"]):
        device.get_primitive(i, out)
    return {"primitive": state["out"], "time": time, "steps": steps, "residual": residual}


def work(case):
    """Bytes and operations of the residuals and vector updates a pass cannot do without: per residual the
    state, gradients and geometry once and the new state, 4-byte geometry and gradients with 32-bit
    fluxes; an implicit step is counted as one Newton iteration with three Krylov vectors."""
    nbytes = flops = 0
    g = 4 if case["precision"] == "fp32" else 8
    for nx, ny, nz, _ in _sizes(case):
        cells, faces = (4.7 * nx**3, 10.0 * nx**3) if case["flow"] == "ramp" else (nx * ny * nz, 3.0 * nx * ny * nz)
        residual = (168 + 30 * g) * cells + (8 + 22 * g) * faces
        if _viscous(case):
            residual += (10 * g + 8) * cells + 4 * g * faces
        operations = 400 * cells + (500 if _viscous(case) else 300) * faces
        count = {"residual": 1, "step": 3}.get(case["kind"], case["steps"] * (3 if case["method"] == "lserk" else 5))
        vectors = 40 * cells * case["steps"] * 30 if case["method"] != "lserk" else 0
        nbytes += count * residual + 80 * cells + vectors
        flops += count * operations
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    """Relative 2-norm, about four times what the package's own exact-arithmetic form and `exact` differ by."""
    if case["method"] != "lserk":
        # The finite-difference Jacobian (perturbation 1e-6, or 3e-4 with 32-bit fluxes) amplifies rounding to
        # 2e-7, and a Krylov tolerance of 0.3 lets rounding decide now and then whether one more vector is
        # taken (1e-3 in the residual seen); 32-bit matvecs move the iterate by 5e-3.
        return {"rel": 2e-2} if case["precision"] == "fp32" else {"rel": 4e-3}
    if case["precision"] == "fp32":
        # at low Mach number the residual is a small difference of pressures (1e-2 off with hllc and ausmd)
        if case["flow"] == "tgv":
            return {"rel": 3e-2} if case["kind"] == "residual" else {"rel": 5e-4}
        return {"rel": 4e-5}
    return {"rel": 1e-10}  # the low-Mach residual's cancellation: 9e-12 at 61 x 47 x 53


# ---- the same in plain 64-bit torch ---------------------------------------------------------------


def exact(case, seed):
    if case["method"] != "lserk" and case["precision"] == "fp32":
        return None  # the loose Newton iteration stops at another iterate, no rounding of this one
    rng = np.random.default_rng(seed)
    out = []
    for size in _sizes(case):
        flow = _Flow(case, _mesh(case["flow"], *size), rng)
        if case["kind"] == "residual":
            return flow.derivative(flow.q).cpu().numpy()
        time = step = 0.0
        for _ in range(case["steps"]):
            step, residual = (flow.lserk if case["method"] == "lserk" else flow.implicit)(case["cfl"])
            time += step
        out.append((flow.rows(), time, case["steps"], residual))
    if case["kind"] == "step":
        return {"primitive": out[0][0], "time": out[0][1], "step": step, "residual": out[0][3]}
    if case["kind"] == "run":
        return dict(zip(("primitive", "time", "steps", "residual"), out[0]))
    rows, time, steps, residual = zip(*out)
    return {"primitive": list(rows), "time": np.array(time), "steps": np.array(steps, np.int32),
            "residual": np.array(residual)}


def _conserved(q):
    kinetic = 0.5 * q[:, 0] * (q[:, 1:4] ** 2).sum(1)
    return torch.cat([q[:, :1], q[:, :1] * q[:, 1:4], (q[:, 4] / (GAMMA - 1) + kinetic)[:, None]], 1)


def _primitive(u):
    rho = u[:, 0].clamp(min=1e-8)
    vel = u[:, 1:4] / rho[:, None]
    p = ((GAMMA - 1) * (u[:, 4] - 0.5 * (u[:, 1:4] * vel).sum(1))).clamp(min=1e-8)
    return torch.cat([rho[:, None], vel, p[:, None]], 1)


def _physical(w, u):
    f = u * w[:, 1:2]
    f[:, 1] += w[:, 4]
    f[:, 4] += w[:, 4] * w[:, 1]
    return f


def _roe_average(a, b):
    ha, hb = ((_conserved(w)[:, 4] + w[:, 4]) / w[:, 0] for w in (a, b))
    sa, sb = a[:, 0].sqrt(), b[:, 0].sqrt()
    vel = (sa[:, None] * a[:, 1:4] + sb[:, None] * b[:, 1:4]) / (sa + sb)[:, None]
    h = (sa * ha + sb * hb) / (sa + sb)
    return vel, h, ((GAMMA - 1) * (h - 0.5 * (vel**2).sum(1))).sqrt()


def _sound(w):
    return (GAMMA * w[:, 4] / w[:, 0]).sqrt()


def _roe(a, b):
    """Roe's flux with the Harten-Hyman entropy fix, states in the face frame."""
    v, h, c = _roe_average(a, b)
    ca, cb = _sound(a), _sound(b)
    eig = []
    for s in (-1, 0, 1):
        lam = v[:, 0] + s * c
        delta = torch.maximum(lam - (a[:, 1] + s * ca), b[:, 1] + s * cb - lam).clamp(min=0)
        eig.append(torch.where(lam.abs() < delta, delta, lam.abs()))
    ua, ub = _conserved(a), _conserved(b)
    j = ub - ua
    w2, w3 = j[:, 2] - v[:, 1] * j[:, 0], j[:, 3] - v[:, 2] * j[:, 0]
    w1 = (GAMMA - 1) / c**2 * (j[:, 0] * (h - v[:, 0] ** 2) + v[:, 0] * j[:, 1] - j[:, 4] + w2 * v[:, 1] + w3 * v[:, 2])
    w0 = (j[:, 0] * (v[:, 0] + c) - j[:, 1] - c * w1) / (2 * c)
    w4 = j[:, 0] - w0 - w1
    w0, w1, w2, w3, w4 = w0 * eig[0], w1 * eig[1], w2 * eig[1], w3 * eig[1], w4 * eig[2]
    d = torch.stack([
        w0 + w1 + w4,
        (v[:, 0] - c) * w0 + v[:, 0] * w1 + (v[:, 0] + c) * w4,
        v[:, 1] * (w0 + w1 + w4) + w2,
        v[:, 2] * (w0 + w1 + w4) + w3,
        (h - v[:, 0] * c) * w0 + 0.5 * (v**2).sum(1) * w1 + v[:, 1] * w2 + v[:, 2] * w3 + (h + v[:, 0] * c) * w4], 1)
    return 0.5 * (_physical(a, ua) + _physical(b, ub) - d)


def _hllc(a, b):
    v, _, c = _roe_average(a, b)
    sa, sb = torch.minimum(a[:, 1] - _sound(a), v[:, 0] - c), torch.maximum(b[:, 1] + _sound(b), v[:, 0] + c)
    ma, mb = a[:, 0] * (sa - a[:, 1]), b[:, 0] * (sb - b[:, 1])
    s = (b[:, 4] - a[:, 4] + ma * a[:, 1] - mb * b[:, 1]) / (ma - mb)
    flux = []
    for w, sk, mk in ((a, sa, ma), (b, sb, mb)):
        u = _conserved(w)
        rho = mk / (sk - s)
        star = torch.stack([rho, rho * s, rho * w[:, 2], rho * w[:, 3],
                            rho * (u[:, 4] / w[:, 0] + (s - w[:, 1]) * (s + w[:, 4] / mk))], 1)
        f = _physical(w, u)
        flux += [f, f + sk[:, None] * (star - u)]
    fa, ga, fb, gb = flux
    out = torch.where((s >= 0)[:, None], ga, gb)
    out = torch.where((sb <= 0)[:, None], fb, out)
    return torch.where((sa >= 0)[:, None], fa, out)


def _ausmd(a, b):
    c = torch.maximum(_sound(a), _sound(b))
    ta, tb_ = a[:, 4] / a[:, 0], b[:, 4] / b[:, 0]
    speed, pressure = [], []
    for w, t, s in ((a, ta, 1), (b, tb_, -1)):
        un, alpha = w[:, 1], 2 * t / (ta + tb_)
        half = (un + s * un.abs()) / 2
        sub = un.abs() <= c
        speed.append(torch.where(sub, s * alpha * (un + s * c) ** 2 / (4 * c) + (1 - alpha) * half, half))
        pressure.append(torch.where(sub, w[:, 4] * (un + s * c) ** 2 / (4 * c * c) * (2 - s * un / c), w[:, 4] * half / un))
    mass = (speed[0] * a[:, 0] + speed[1] * b[:, 0])[:, None]
    pa, pb = (torch.cat([torch.ones_like(w[:, :1]), w[:, 1:4], ((_conserved(w)[:, 4] + w[:, 4]) / w[:, 0])[:, None]], 1)
              for w in (a, b))
    f = 0.5 * (mass * (pa + pb) - mass.abs() * (pb - pa))
    f[:, 1] += pressure[0] + pressure[1]
    return f


class _Flow:
    """The scheme on one mesh: least-squares gradients, limiter, fluxes, boundary ghosts, steps."""

    def __init__(self, case, mesh, rng):
        self.device = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = self._tensor
        s = mesh.struct
        self.case, self.viscous, self.mu = case, _viscous(case), case.get("viscosity", 1 / 1600)
        self.C, self.N, self.inner, self.bound = s.num_inner_cells, s.off_boundary_cells, s.num_inner_faces, s.off_boundary_faces
        cells = np.array(mesh.array("faces.cell_idx"), np.int64)
        owner = np.full(mesh.num_cells - self.N, -1, np.int64)
        if len(owner):  # periodic ghosts take their owners' states, exchanged by tag
            tags, recv = mesh.array("neighbors.tag"), mesh.array("neighbors.recv_off")
            send, idx, used = mesh.array("neighbors.send.off"), mesh.array("neighbors.send.idx"), set()
            for k in range(len(tags)):
                m = next(j for j in range(len(tags)) if j not in used and tags[j, 1] == tags[k, 0])
                used.add(m)
                owner[recv[k] - self.N: recv[k + 1] - self.N] = idx[send[m]: send[m + 1]]
            ghost = cells[:, 1] >= self.N
            cells[ghost, 1] = owner[cells[ghost, 1] - self.N]
        self.owner = t(owner)
        self.l, self.r = t(cells[:, 0]), t(cells[:, 1])
        self.area, self.basis = t(mesh.array("faces.area")), t(mesh.array("faces.basis"))
        self.weight, self.offset = t(mesh.array("faces.weight")), t(mesh.array("faces.offset"))
        self.volume, self.projection = t(mesh.cell_volume[: self.C]), t(mesh.array("cells.projection")[: self.C])
        self.total = mesh.sum_volume
        self.correction = t(mesh.array("faces.correction")) if self.viscous else None
        state, self.free = _state(case["flow"], mesh.cell_center[: self.C], rng)
        sides = _boundaries(case, self.free)
        first, off = s.num_inner_entities, mesh.array("entities.face_off")
        self.sides = [(sides[mesh.entities[i][0]][0], int(off[i]), int(off[i + 1]))
                      for i in range(first, s.off_boundary_entities)]
        self.q = torch.zeros((self.N, 5), dtype=torch.float64, device=self.device)
        self.q[: self.C] = t(state)

    def _tensor(self, a):
        return torch.from_numpy(np.array(a)).to(self.device)

    def rows(self):
        return torch.cat([self.q, self.q[self.owner]]).cpu().numpy()

    def _to_cells(self, left, right):
        """Sum of face values over each cell: `left` to the left cells, `right` to the inner faces' right ones."""
        out = torch.zeros((self.C, *left.shape[1:]), dtype=torch.float64, device=self.device)
        out.index_add_(0, self.l, left)
        return out.index_add_(0, self.r[: self.inner], right)

    def _ghosts(self, q):
        for kind, beg, end in self.sides:
            w, n, rows = q[self.l[beg:end]], self.basis[beg:end, 0], self.r[beg:end]
            if kind == "slipwall":
                w[:, 1:4] -= 2 * (w[:, 1:4] * n).sum(1, keepdim=True) * n
            elif kind == "adiabatic wall":
                w[:, 1:4] *= -1
            else:
                w = self._farfield(w, beg, end)
            q[rows] = w

    def _farfield(self, w, beg, end):
        """Characteristic far field: the free stream's waves where they enter, the cell's where they leave."""
        b = self.basis[beg:end]
        inside = self._local(w, b)
        outside = self._local(self._tensor(self.free).expand_as(w).contiguous(), b)
        c2, g1 = GAMMA * inside[:, 4] / inside[:, 0], GAMMA - 1
        c, (x, y, z) = c2.sqrt(), inside[:, 1:4].T
        h, o, i = 0.5 * (inside[:, 1:4] ** 2).sum(1) + c2 / g1, torch.zeros_like(x), torch.ones_like(x)
        left = torch.stack([
            torch.stack([h + c / g1 * (x - c), -(x + c / g1), -y, -z, i], 1),
            torch.stack([-2 * h + 4 / g1 * c2, 2 * x, 2 * y, 2 * z, -2 * i], 1),
            torch.stack([-2 * y * c2 / g1, o, 2 * c2 / g1, o, o], 1),
            torch.stack([-2 * z * c2 / g1, o, o, 2 * c2 / g1, o], 1),
            torch.stack([h - c / g1 * (x + c), -x + c / g1, -y, -z, i], 1)], 1) * (g1 / (2 * c2))[:, None, None]
        right = torch.stack([
            torch.stack([i, i, o, o, i], 1), torch.stack([x - c, x, o, o, x + c], 1),
            torch.stack([y, y, i, o, y], 1), torch.stack([z, z, o, i, z], 1),
            torch.stack([h - x * c, 0.5 * (inside[:, 1:4] ** 2).sum(1), y, z, h + x * c], 1)], 1)
        a, g = ((left @ _conserved(k)[:, :, None])[:, :, 0] for k in (inside, outside))
        un, cg = outside[:, 1], _sound(outside)
        leaves = torch.stack([un - cg, un, un, un, un + cg], 1) > 0
        u = (right @ torch.where(leaves, a, g)[:, :, None])[:, :, 0]
        out = _primitive(u)
        out[:, 1:4] = (b.transpose(1, 2) @ out[:, 1:4, None])[:, :, 0]
        return out

    @staticmethod
    def _local(w, basis):
        return torch.cat([w[:, :1], (basis @ w[:, 1:4, None])[:, :, 0], w[:, 4:]], 1)

    def derivative(self, q):
        self._ghosts(q)
        inner, l, r = self.inner, self.l, self.r
        ri, li = r[:inner], l[:inner]
        jump = (q[r] - q[l])[:, :, None]
        grad = self._to_cells(jump * self.weight[:, None, 0], -jump[:inner] * self.weight[:inner, None, 1])
        del jump
        psi = self._limiter(q, grad)
        limited = psi[:, :, None] * grad
        a, b = q[l], q[r]
        a = a + (limited[l] * self.offset[:, None, 0]).sum(2)
        two = torch.ones_like(r, dtype=torch.bool)
        two[inner: self.bound] = False
        at = torch.where(two, r, 0)
        b = b + (limited[at] * self.offset[:, None, 1]).sum(2) * two[:, None]
        f = {"roe": _roe, "hllc": _hllc, "ausmd": _ausmd}[self.case["flux"]](self._local(a, self.basis), self._local(b, self.basis))
        f[:, 1:4] = (self.basis.transpose(1, 2) @ f[:, 1:4, None])[:, :, 0]
        del a, b, limited
        if self.viscous:
            f -= self._viscous_flux(q, grad, at, two)
        f *= self.area[:, None]
        return -self._to_cells(f, -f[:inner]) / self.volume[:, None]

    def _limiter(self, q, grad):
        l, r, n = self.l, self.r, self.inner
        hi, lo = q[: self.C].clone(), q[: self.C].clone()
        for index, value in ((l, q[r]), (r[:n], q[l[:n]])):
            at = index[:, None].expand_as(value)
            hi.scatter_reduce_(0, at, value, "amax")
            lo.scatter_reduce_(0, at, value, "amin")
        hi, lo = hi - q[: self.C], lo - q[: self.C]
        eps = self.volume[:, None]
        psi = torch.ones_like(hi)
        for index, side, faces in ((l, 0, slice(None)), (r[:n], 1, slice(0, n))):
            d2 = (grad[index] * self.offset[faces, None, side]).sum(2)
            d1 = torch.where(d2 > 0, hi[index], lo[index])
            if self.case["limiter"] == "minmod":
                value = (d1 / d2).clamp(max=1)
            else:
                value = ((d1**2 + eps[index]) * d2 + 2 * d2**2 * d1) / (d1**2 + 2 * d2**2 + d1 * d2 + eps[index]) / d2
            value = torch.where(d2.abs() <= 1e-8, 1.0, value)
            psi.scatter_reduce_(0, index[:, None].expand_as(value), value, "amin")
        return psi

    def _viscous_flux(self, q, grad, at, two):
        a, b, unit = q[self.l], q[self.r], self.correction[:, None, :3]
        g = grad[self.l]
        g = torch.where(two[:, None, None], 0.5 * (g + grad[at]), g)
        g = g - ((g * unit).sum(2) - (b - a) / self.correction[:, 3:])[:, :, None] * unit
        m, du = 0.5 * (a + b), g[:, 1:4]
        tau = self.mu * (du + du.transpose(1, 2))
        tau -= 2 / 3 * self.mu * (du[:, 0, 0] + du[:, 1, 1] + du[:, 2, 2])[:, None, None] * torch.eye(3, dtype=torch.float64, device=self.device)
        heat = -self.mu * GAMMA / ((GAMMA - 1) * PRANDTL) * ((m[:, :1] * g[:, 4] - m[:, 4:] * g[:, 0]) / m[:, :1] ** 2)
        theta = (tau @ m[:, 1:4, None])[:, :, 0] - heat
        n = self.basis[:, 0]
        return torch.cat([torch.zeros_like(m[:, :1]), (tau @ n[:, :, None])[:, :, 0], (theta * n).sum(1, keepdim=True)], 1)

    def timestep(self):
        q = self.q[: self.C]
        speed = ((q[:, 1:4].abs() + _sound(q)[:, None]) * self.projection).sum(1)
        if self.viscous:
            lam = torch.maximum(4 * self.mu / (3 * q[:, 0]), GAMMA * self.mu / (q[:, 0] * PRANDTL))
            speed = speed + 4 * lam * (self.projection**2).sum(1) / self.volume
        return float((self.volume / speed).min())

    def _residual(self, d):
        return ((self.volume[:, None] * d**2).sum(0) / self.total).sqrt().cpu().numpy()

    def lserk(self, cfl):
        step, u0 = cfl * self.timestep(), _conserved(self.q[: self.C])
        for alpha in (0.2884, 0.5010, 1.0):
            d = self.derivative(self.q)
            self.q[: self.C] = _primitive(u0 + d * (alpha * step))
        return step, self._residual(d)

    def implicit(self, cfl):
        """Implicit Euler by Newton-GMRES with finite-difference products."""
        step, u0 = cfl * self.timestep(), _conserved(self.q[: self.C])
        u, d = u0.clone(), self.derivative(self.q)
        r = -d * step
        norm = float(r.norm())
        target, q1 = NEWTON[0] * norm, torch.zeros_like(self.q)
        while norm > target:
            scale = 1e-6 * max(1.0, float(u.norm())) / max(1.0, norm)

            def product(v):
                eps = scale / float(v.norm())
                q1[: self.C] = _primitive(u + eps * v)
                return v - step * (self.derivative(q1) - d) / eps

            u = u + self._gmres(product, r, norm)
            self.q[: self.C] = _primitive(u)
            d = self.derivative(self.q)
            r = u - u0 - step * d
            norm = float(r.norm())
        return step, self._residual(d)

    @staticmethod
    def _gmres(product, r, norm):
        basis, n = [-r / norm], NEWTON[2]
        h, rhs, rotations = np.zeros((n + 1, n)), np.zeros(n + 1), []
        rhs[0] = norm
        for k in range(n):
            w = product(basis[k])
            for i in range(k + 1):
                h[i, k] = float((basis[i] * w).sum())
                w = w - h[i, k] * basis[i]
            h[k + 1, k] = float(w.norm())
            basis.append(w / h[k + 1, k])
            for i, (c, s) in enumerate(rotations):
                h[i, k], h[i + 1, k] = c * h[i, k] + s * h[i + 1, k], -s * h[i, k] + c * h[i + 1, k]
            rot = math.hypot(h[k, k], h[k + 1, k])
            rotations.append((h[k, k] / rot, h[k + 1, k] / rot))
            h[k, k] = rot
            rhs[k + 1], rhs[k] = -rotations[k][1] * rhs[k], rotations[k][0] * rhs[k]
            if abs(rhs[k + 1]) < NEWTON[1] * norm:
                break
        y = np.linalg.solve(np.triu(h[: k + 1, : k + 1]), rhs[: k + 1])
        return sum(float(c) * v for c, v in zip(y, basis))
