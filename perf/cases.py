"""The workloads this engine is timed on, through its public entry points.

``listed()`` names them, ``draw(rng)`` gives one more of the same ranges,
``prepare(case, seed)`` builds what a user's program holds before the call
(a finalized ``Solver``, an ``Ensemble``, a ``ChannelProblem`` with its
parameters), ``run(state)`` is one call and ``work(case)`` its unavoidable
bytes and operations.  ``exact(case, seed)`` computes the same outputs with a
plain two-lattice FP64 step in torch that shares no code with the engine.

Flow kinds (all through ``Solver.evolve``):
  rows    gravity-driven channel, solid rows at both y ends, periodic faces
  half    half channel: wall on 1Y, symmetric Y1, gravity along x
  cavity  box of walls with a Zou-He velocity lid on Y1
  duct    Zou-He velocity inlet on 1X, density outlet on X1, walls, cylinder
  porous  channel through non-overlapping spheres, porosity 0.6
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "jyu-lb_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from jyulb.adjoint import ChannelProblem  # noqa: E402
from jyulb.defs import (BGK, FIXED_DEN, FIXED_VEL, FP16, FP32, FP64, FP64_FAST, PERIODIC,  # noqa: E402
                        REGULARIZATION, SYMMETRIC, TRT, WALL)
from jyulb.ensemble import Domain, Ensemble  # noqa: E402
from jyulb.isothermal import Solver  # noqa: E402

SCHEME = {"bgk": BGK, "trt": TRT, "reg": REGULARIZATION}
PRECISION = {"fp64": FP64, "fp64_fast": FP64_FAST, "fp32": FP32, "fp16": FP16}
POP_BYTES = {"fp64": 8, "fp64_fast": 8, "fp32": 4, "fp16": 2}


def _flow(name, kind, shape, scheme, precision, steps, tau, magic=0.0):
    return {"name": name, "kind": kind, "nx": shape[0], "ny": shape[1], "nz": shape[2], "scheme": scheme,
            "precision": precision, "steps": steps, "tau": tau, "magic": magic}


def listed():
    return [
        # the reference's example channel: a lattice far smaller than the GPU,
        # advanced 500 steps per call as its scripts do; launches and latency
        _flow("channel_4x34x4_fp64", "rows", (4, 34, 4), "bgk", "fp64", 500, 0.8),
        # an ordinary flow around an obstacle at the default precision, sizes
        # that divide by nothing
        _flow("duct_100x61x47_fp64", "duct", (100, 61, 47), "trt", "fp64", 100, 0.6),
        # the 256^3 cavity at the default precision (the reference's numbers)
        _flow("cavity_256_fp64", "cavity", (256, 256, 256), "trt", "fp64", 20, 0.56, 0.25),
        # the opt-in fast FP64 form on a medium cavity
        _flow("cavity_128_fp64fast", "cavity", (128, 128, 128), "trt", "fp64_fast", 100, 0.56, 0.25),
        # the headline configuration: FP32 shifted populations, long calls
        _flow("cavity_256_fp32", "cavity", (256, 256, 256), "trt", "fp32", 200, 0.56, 0.25),
        # the same read out after every step (time series, coupling)
        _flow("cavity_256_fp32_each", "cavity", (256, 256, 256), "trt", "fp32", 1, 0.56, 0.25),
        # half the memory per site: FP16 storage
        _flow("cavity_256_fp16", "cavity", (256, 256, 256), "trt", "fp16", 200, 0.56, 0.25),
        # a medium lattice about the size of the L2, ragged in every direction
        _flow("duct_200x90x75_fp32", "duct", (200, 90, 75), "reg", "fp32", 200, 0.6),
        # flow through a porous medium, the largest lattice
        _flow("porous_384x256x256_fp32", "porous", (384, 256, 256), "reg", "fp32", 100, 0.7),
        # a medium porous sample in FP16 storage
        _flow("porous_192x128x128_fp16", "porous", (192, 128, 128), "reg", "fp16", 100, 0.7),
        # a parameter study: many channels of uneven size in one launch
        {"name": "ensemble_32", "kind": "ensemble", "domains": 32, "scale": 1.0, "steps": 1000, "scheme": "bgk"},
        # gradients of a velocity loss through the time loop (forward and
        # reverse), checkpoints every 50 steps
        {"name": "adjoint_256x64x64", "kind": "adjoint", "nx": 256, "ny": 64, "nz": 64, "scheme": "trt",
         "precision": "fp32", "steps": 200, "every": 50, "tau": 0.58, "magic": 0.25},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    pick = rng.random()
    if pick < 0.12:
        return {"kind": "ensemble", "domains": rng.randint(3, 32), "scale": round(rng.uniform(0.3, 1.0), 3),
                "steps": _log_int(rng, 50, 500), "scheme": rng.choice(["bgk", "trt", "reg"])}
    if pick < 0.27:
        return {"kind": "adjoint", "nx": rng.randint(40, 256), "ny": rng.randint(12, 64), "nz": rng.randint(12, 64),
                "scheme": rng.choice(["trt", "bgk", "reg"]), "precision": rng.choice(["fp32", "fp32", "fp64"]),
                "steps": rng.randint(40, 150), "every": rng.randint(10, 50), "tau": round(rng.uniform(0.56, 0.9), 3),
                "magic": 0.25}
    kind = rng.choice(["rows", "half", "cavity", "duct", "porous"])
    precision = rng.choice(["fp64", "fp64", "fp64_fast", "fp32", "fp32", "fp16"])
    lo = 100_000 if kind == "porous" else 600
    n = _log_int(rng, lo, 6_000_000)
    # uneven aspect ratios around the cube root
    a, b = math.exp(rng.uniform(-0.7, 0.7)), math.exp(rng.uniform(-0.7, 0.7))
    s = n ** (1.0 / 3.0)
    least = 40 if kind == "porous" else 5
    shape = [max(least, int(round(v))) for v in (s * a, s * b, s / (a * b))]
    if rng.random() < 0.3:  # lines of a length the kernels tile evenly
        shape[2] = max(32, (shape[2] + 31) // 64 * 64)
    sites = shape[0] * shape[1] * shape[2]
    cost = {"fp64": 8.0, "fp64_fast": 5.0}.get(precision, 1.0)
    steps = max(1, min(_log_int(rng, 1, 500), int(1.5e9 / (cost * sites))))
    c = _flow("", kind, shape, rng.choice(["bgk", "trt", "reg"]), precision, steps,
              round(rng.uniform(0.56, 0.95), 3), rng.choice([0.0, 0.25]))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _spheres(shape, rng, r=8, porosity=0.6):
    """Solid mask of non-overlapping spheres: a lattice of spacing 2r+1 with a
    jitter of half a site, filled in random order down to the porosity;
    periodic in x and z, whole spheres between the y walls."""
    nx, ny, nz = shape
    sp = 2 * r + 1
    axes = [np.arange(max(1, n // sp)) * sp + sp / 2.0 for n in shape]
    c = np.stack(np.meshgrid(*axes, indexing="ij"), -1).reshape(-1, 3)
    c = (c + rng.uniform(-0.5, 0.5, c.shape))[rng.permutation(len(c))]
    solid = np.zeros(shape, bool)
    off = np.arange(-r - 1, r + 2)
    left = (1.0 - porosity) * solid.size
    for x, y, z in c:
        bx, by, bz = int(x), int(y), int(z)
        inside = ((bx + off - x) ** 2)[:, None, None] + ((by + off - y) ** 2)[:, None] + (bz + off - z) ** 2 <= r * r
        i, j, k = (off[v] for v in np.nonzero(inside))
        j = by + j
        ok = (j >= 0) & (j < ny)
        i, j, k = (bx + i[ok]) % nx, j[ok], (bz + k[ok]) % nz
        solid[i, j, k] = True
        left -= len(i)
        if left <= 0:
            break
    return solid


def _swirl(n, rng, modes=3):
    x = (np.arange(n) + 0.5) / n
    return sum(rng.uniform(-1, 1) * np.cos(2 * math.pi * m * x + rng.uniform(0, 6.28)) for m in range(1, modes + 1))


def _flow_inputs(case, seed):
    """phase, den, vel (interior), bc, g, kvisc of a flow case."""
    rng = np.random.default_rng([int(seed), case["nx"], case["ny"], case["nz"]])
    shape = nx, ny, nz = case["nx"], case["ny"], case["nz"]
    kind = case["kind"]
    phase = np.ones(shape, np.uint8)
    g = np.zeros(3)
    if kind == "rows":
        phase[:, 0, :] = phase[:, -1, :] = 0
        bc = [PERIODIC] * 6
        g[0] = 1e-6 * rng.uniform(0.8, 1.2)
    elif kind == "half":
        bc = [PERIODIC, PERIODIC, WALL, SYMMETRIC, PERIODIC, PERIODIC]
        g[0] = 1e-5 * rng.uniform(0.8, 1.2)
    elif kind == "cavity":
        bc = [WALL, WALL, WALL, FIXED_VEL, WALL, WALL]
    elif kind == "duct":
        bc = [FIXED_VEL, FIXED_DEN, WALL, WALL, WALL, WALL]
        x, y = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
        r = max(1.0, min(8.0, ny / 6.0))
        cx, cy = nx / 3.0 + rng.uniform(-1, 1), ny / 2.0 + rng.uniform(-1, 1)
        phase[(x - cx) ** 2 + (y - cy) ** 2 <= r * r] = 0
        phase[0] = phase[-1] = 1
    else:
        phase[_spheres(shape, rng)] = 0
        bc = [PERIODIC, PERIODIC, WALL, WALL, PERIODIC, PERIODIC]
        g[0] = 5e-6 * rng.uniform(0.8, 1.2)
    # a smooth flow to start from, as after an earlier run
    sx, sy, sz = (_swirl(n, rng) for n in shape)
    den = 1.0 + 1e-4 * sx[:, None, None] * (sy[:, None] * sz)
    vel = np.empty(shape + (3,))
    for d in range(3):
        sx, sy, sz = (_swirl(n, rng) for n in shape)
        np.multiply(2e-3 * sx[:, None, None], sy[:, None] * sz, out=vel[..., d])
    vel[phase == 0] = 0.0
    if kind == "cavity":
        vel[:, -1, :, 0] = 0.05 * rng.uniform(0.9, 1.1)
        vel[:, -1, :, 1] = 0.0
        vel[:, -1, :, 2] = 0.01 * rng.uniform(-1, 1)
    elif kind == "duct":
        yy, zz = (np.arange(ny) + 0.5) / ny, (np.arange(nz) + 0.5) / nz
        vel[0] = 0.0
        vel[0, :, :, 0] = 0.04 * rng.uniform(0.9, 1.1) * 16.0 * np.outer(yy * (1 - yy), zz * (1 - zz))
        vel[-1] = 0.0
        den[-1] = 1.0
    return phase, den, vel, bc, g, (case["tau"] - 0.5) / 3.0


def _ensemble_inputs(case, seed):
    rng = np.random.default_rng([int(seed), case["domains"]])
    s = case["scale"]
    doms = []
    for d in range(case["domains"]):
        # sizes belong to the case, values to the seed
        szr = np.random.default_rng([case["domains"], d])
        shape = (max(4, int(szr.integers(32, 257) * s)), max(4, int(szr.integers(16, 129) * s)),
                 max(2, int(szr.integers(8, 65) * s)))
        phase = np.ones(shape, np.uint8)
        phase[:, 0, :] = phase[:, -1, :] = 0
        tau, gx, uw = rng.uniform(0.55, 1.5), rng.uniform(1e-7, 1e-5), rng.uniform(0.01, 0.05)
        vel = None
        if d % 2 == 1:
            vel = np.zeros(shape + (3,))
            vel[:, -1, :, 0] = uw
        doms.append((phase, vel, (tau - 0.5) / 3.0, [gx, 0.0, 0.0]))
    return doms


def _adjoint_inputs(case, seed):
    rng = np.random.default_rng([int(seed), case["nx"], case["ny"], case["nz"]])
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    x, y = np.meshgrid(np.arange(nx), np.arange(ny), indexing="ij")
    phase = np.ones((nx, ny, nz), np.uint8)
    r = min(8.0, ny / 6.0)
    phase[(x - nx / 4.0) ** 2 + (y - ny / 2.0 - 0.3) ** 2 <= r * r] = 0
    yy, zz = (np.arange(ny) + 0.5) / ny, (np.arange(nz) + 0.5) / nz
    prof = 16.0 * np.outer(yy * (1 - yy), zz * (1 - zz))
    uin = 0.035 * prof * (1 + 0.1 * rng.standard_normal((ny, nz)))
    target = np.zeros((ny, nz, 3))
    target[..., 0] = 0.04 * prof * rng.uniform(0.9, 1.1)
    g = np.array([1e-6 * rng.uniform(0.5, 1.5), 0.0, 0.0])
    # near enough to the inlet for the flow to arrive within the steps
    plane = min(nx * 3 // 4, max(3, case["steps"] // 4))
    return phase, uin, target, g, plane


ADJOINT_BC = [FIXED_VEL, FIXED_DEN, WALL, WALL, WALL, WALL]


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "ensemble":
        doms = [Domain(p, None, v, kv, g) for p, v, kv, g in _ensemble_inputs(case, seed)]
        return {"case": case, "ensemble": Ensemble(doms, SCHEME[case["scheme"]])}
    if case["kind"] == "adjoint":
        phase, uin, target, g, plane = _adjoint_inputs(case, seed)
        p = ChannelProblem(phase, bc=ADJOINT_BC, rlx_scheme=SCHEME[case["scheme"]],
                           precision=PRECISION[case["precision"]], trt_magic=case["magic"], loss_plane=plane,
                           checkpoint_every=case["every"])
        return {"case": case, "problem": p, "args": (case["tau"], g, uin, case["steps"], target)}
    phase, den, vel, bc, g, kvisc = _flow_inputs(case, seed)
    s = Solver.with_iflow(phase, den, vel, SCHEME[case["scheme"]], kvisc, g, np.array(bc, dtype=np.int32),
                          precision=PRECISION[case["precision"]], trt_magic=case["magic"] or None)
    s.finalize_init()
    return {"case": case, "solver": s}


def run(state):
    if "ensemble" in state:
        e = state["ensemble"]
        e.evolve(state["case"]["steps"])
        return [e.moments(d) for d in range(state["case"]["domains"])]
    if "problem" in state:
        loss, u = state["problem"].forward(*state["args"])
        dtau, dg, duin = state["problem"].backward()
        return {"loss": loss, "u": u, "dtau": dtau, "dg": dg, "duin": duin}
    s = state["solver"]
    s.evolve(state["case"]["steps"])
    return {"den": s.get_den(), "vel": s.get_vel()}


# operations of one site update (moments, equilibrium, forcing, relaxation,
# projection), and of its transpose
SITE_FLOPS = 250


def work(case):
    """Per step each population of a fluid site is read once and written once;
    density and velocity come back once per call in FP64."""
    steps = case["steps"]
    if case["kind"] == "ensemble":
        sites = sum(int(np.prod(p.shape)) - 2 * p.shape[0] * p.shape[2] for p, _, _, _ in _ensemble_inputs(case, 0))
        return {"bytes": sites * (152 * steps + 32), "flops": SITE_FLOPS * sites * steps}
    sites = case["nx"] * case["ny"] * case["nz"]
    b = 38 * POP_BYTES[case["precision"]]
    if case["kind"] == "adjoint":
        # forward step, its recomputation in the backward run (all but one of
        # each segment's), and the reverse sweep: state read, adjoint read and
        # written
        again = steps - -(-steps // case["every"])
        return {"bytes": sites * b * (steps + again + 1.5 * steps), "flops": SITE_FLOPS * sites * (3 * steps + again)}
    fluid = {"porous": 0.6, "rows": (case["ny"] - 2) / case["ny"]}.get(case["kind"], 1.0) * sites
    return {"bytes": int(fluid * (b * steps + 32)), "flops": int(SITE_FLOPS * fluid * steps)}


# ---------------------------------------------------------------------------
# the same in 64 bits: a plain pull step on halo-padded arrays
# ---------------------------------------------------------------------------
C = np.array([(-1, -1, 0), (-1, 0, -1), (-1, 0, 0), (-1, 0, 1), (-1, 1, 0), (0, -1, -1), (0, -1, 0), (0, -1, 1),
              (0, 0, -1), (0, 0, 0), (0, 0, 1), (0, 1, -1), (0, 1, 0), (0, 1, 1), (1, -1, 0), (1, 0, -1), (1, 0, 0),
              (1, 0, 1), (1, 1, 0)])
W = [1 / 3 if not c.any() else 1 / 18 if abs(c).sum() == 1 else 1 / 36 for c in C]
INNER = (slice(1, -1),) * 3


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _find(c):
    return next(q for q in range(19) if tuple(C[q]) == tuple(c))


def _faces(bc, shape):
    """(read plane, written plane, axis, mirrored) of the periodic and
    symmetric faces in the order x, y, z that the halo copies run in."""
    out = []
    for face in range(6):
        if bc[face] not in (PERIODIC, SYMMETRIC):
            continue
        ax, high = face // 2, face % 2
        n, per = shape[ax] + 2, bc[face] == PERIODIC
        rd, wr = (n - 2, 0 if per else n - 1) if high else (1, n - 1 if per else 0)
        inner, whole = slice(1, -1), slice(None)
        cover = [[None, inner, inner], [whole, None, inner], [whole, whole, None]][ax]
        r, w = list(cover), list(cover)
        r[ax], w[ax] = rd, wr
        out.append((tuple(r), tuple(w), ax, not per))
    return out


def _pad(x, fill):
    """Halo-padded copy of the interior array x."""
    p = torch.full([n + 2 for n in x.shape[:3]] + list(x.shape[3:]), fill, dtype=x.dtype, device=x.device)
    p[INNER] = x
    return p


def _shifted(p, c):
    """The interior's view of the padded array p at x + c."""
    return p[tuple(slice(1 + int(d), p.shape[a] - 1 + int(d)) for a, d in enumerate(c))]


class _Plain:
    def __init__(self, phase, vel, bc, scheme, kvisc, magic):
        dev = _device()
        self.bc, self.scheme, self.shape = [int(b) for b in bc], scheme, phase.shape
        self.faces = _faces(self.bc, phase.shape)
        ph = _pad(torch.from_numpy(np.ascontiguousarray(phase)).to(dev), 0)
        v = _pad(torch.from_numpy(np.ascontiguousarray(vel)).to(dev), 0.0)
        for r, w, ax, mirror in self.faces:
            ph[w] = ph[r]
            t = v[r].clone()
            if mirror:
                t[..., ax] = -t[..., ax]
            v[w] = t
        self.phase, self.vel = ph, v
        self.fluid = ph[INNER] != 0
        # upstream site solid, and the wall speed along q there
        self.solid = [_shifted(ph, -C[q]) == 0 for q in range(19)]
        wall = v * (ph == 0)[..., None]
        self.lw = [None] * 19
        if bool((wall != 0).any()):
            self.lw = [sum(int(C[q][d]) * _shifted(wall, -C[q])[..., d] for d in range(3)) for q in range(19)]
        tau = 0.5 + 3.0 * kvisc
        self.set_tau(tau, magic)

    def set_tau(self, tau, magic):
        self.we = 1.0 / tau
        self.wo = self.we
        if self.scheme == "trt":
            self.wo = 1.0 / (magic / (tau - 0.5) + 0.5) if magic else 8.0 * (2.0 - self.we) / (8.0 - self.we)

    def start(self, den):
        """Initial populations: equilibrium and the velocity gradients' share."""
        v = self.vel
        ph = self.phase
        grad = []
        for a in range(3):
            t = 0.0
            for q in range(19):
                if C[q][a] != 1:
                    continue
                up, dn = _shifted(ph, C[q]) == 0, _shifted(ph, -C[q]) == 0
                c1, c2, c3 = (torch.tensor([[0.5, 1 / 3], [4 / 3, 1.0]], dtype=v.dtype, device=v.device),
                              torch.tensor([[0.0, 1.0], [-1.0, 0.0]], dtype=v.dtype, device=v.device),
                              torch.tensor([[-0.5, -4 / 3], [-1 / 3, -1.0]], dtype=v.dtype, device=v.device))
                c1, c2, c3 = (x[up.long(), dn.long()] for x in (c1, c2, c3))
                t = t + 6.0 * W[q] * (c1[..., None] * _shifted(v, C[q]) + c2[..., None] * v[INNER] +
                                      c3[..., None] * _shifted(v, -C[q]))
            grad.append(t)
        u = [v[INNER][..., d] for d in range(3)]
        k = (1.0 - self.we) * (-2.0 / (3.0 * self.we)) * den
        h2 = {(a, b): den * u[a] * u[b] + k * 0.5 * (grad[a][..., b] + grad[b][..., a])
              for a in range(3) for b in range(a, 3)}
        f = self.project(den, [den * x for x in u], h2)
        return [torch.where(self.fluid, x, torch.zeros_like(x)) for x in f]

    def project(self, h0, h1, h2):
        tr = (h2[0, 0] + h2[1, 1] + h2[2, 2]) / 3.0
        f = []
        for q in range(19):
            c = [int(x) for x in C[q]]
            t = h0 - 4.5 * tr
            for a in range(3):
                if c[a]:
                    t = t + 3.0 * c[a] * h1[a] + 4.5 * h2[a, a]
                    for b in range(a + 1, 3):
                        if c[b]:
                            t = t + 9.0 * c[a] * c[b] * h2[a, b]
            f.append(W[q] * t)
        return f

    def step(self, f, a, den_bc, vel_bc, rho_prev):
        fp = [_pad(x, 0.0) for x in f]
        for r, w, ax, mirror in self.faces:
            src = [x[r].clone() for x in fp]
            for q in range(19):
                c = C[q].copy()
                if mirror:
                    c[ax] = -c[ax]
                fp[q][w] = src[_find(c)]
        s = []
        for q in range(19):
            back = f[18 - q]
            if self.lw[q] is not None and q != 9:
                back = back + 6.0 * W[q] * rho_prev * self.lw[q]
            s.append(torch.where(self.solid[q], back, _shifted(fp[q], -C[q])))
        del fp
        for face in range(6):
            if self.bc[face] in (FIXED_DEN, FIXED_VEL):
                s = self.zou_he(s, face, den_bc, vel_bc)
        return self.collide(s, a)

    def zou_he(self, s, face, den_bc, vel_bc):
        ax, into = face // 2, -1 if face % 2 else 1
        at = [slice(None)] * 3
        at[ax] = -1 if face % 2 else 0
        at = tuple(at)
        p = [x[at] for x in s]
        total = sum(p[q] for q in range(19) if C[q][ax] == 0) + 2.0 * sum(p[q] for q in range(19) if C[q][ax] == -into)
        v = [vel_bc[at][..., d] for d in range(3)]
        if self.bc[face] == FIXED_VEL:
            rho = total / (1.0 - into * v[ax])
            j = [rho * x for x in v]
        else:
            rho = den_bc[at]
            j = [rho * x for x in v]
            j[ax] = into * (rho - total)
        out = list(s)
        for q in range(19):
            if C[q][ax] != into:
                continue
            side = [d for d in range(3) if d != ax and C[q][d]]
            if not side:
                new = p[18 - q] + into * j[ax] / 3.0
            else:
                d = side[0]
                t = sum(int(C[m][d]) * p[m] for m in range(19) if C[m][ax] == 0 and C[m][d])
                new = p[18 - q] + into * j[ax] / 6.0 - 0.5 * int(C[q][d]) * (t - j[d])
            x = s[q].clone()
            x[at] = new
            out[q] = x
        return out

    def collide(self, s, a):
        we, wo = self.we, self.wo
        rho = sum(s)
        j = [sum(int(C[q][d]) * s[q] for q in range(19) if C[q][d]) for d in range(3)]
        u = [j[d] / rho + 0.5 * a[d] for d in range(3)]
        m = [rho * x for x in u]
        h2 = {}
        for p in range(3):
            for r in range(p, 3):
                h2[p, r] = we * m[p] * u[r] + (1.0 - 0.5 * we) * (a[p] * m[r] + a[r] * m[p])
        if self.scheme == "reg":
            for p, r in h2:
                pi = sum(int(C[q][p] * C[q][r]) * s[q] for q in range(19) if C[q][p] * C[q][r])
                h2[p, r] = h2[p, r] + (1.0 - we) * (pi - (rho / 3.0 if p == r else 0.0))
            f = self.project(rho, [j[d] + rho * a[d] for d in range(3)], h2)
        else:
            f = self.project(we * rho, [wo * m[d] + (1.0 - 0.5 * wo) * a[d] * rho for d in range(3)], h2)
            c3, c4 = 1.0 - 0.5 * (we + wo), 0.5 * (we - wo)
            f = [f[q] + ((1.0 - we) * s[q] if q == 9 else c3 * s[q] - c4 * s[18 - q]) for q in range(19)]
        return [torch.where(self.fluid, x, torch.zeros_like(x)) for x in f], rho, u


def _run_plain(phase, den, vel, bc, g, kvisc, scheme, magic, steps):
    plain = _Plain(phase, vel, bc, scheme, kvisc, magic)
    d = torch.from_numpy(np.ascontiguousarray(den)).to(_device())
    v = torch.from_numpy(np.ascontiguousarray(vel)).to(_device())
    f, rho = plain.start(d), d
    for _ in range(steps):
        f, rho, u = plain.step(f, g, d, v, rho)
    out = torch.where(plain.fluid, rho, d)
    ov = torch.where(plain.fluid[..., None], torch.stack(u, -1), v)
    return out.cpu().numpy(), ov.cpu().numpy()


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "ensemble":
            out = []
            for phase, vel, kvisc, g in _ensemble_inputs(case, seed):
                # every domain's loop is launch-bound here: the smallest few
                # stand for the rest
                if phase.size * case["steps"] > 2e8 or len(out) - out.count(None) >= 3 or case["steps"] > 1000:
                    out.append(None)
                    continue
                v = np.zeros(phase.shape + (3,)) if vel is None else vel
                out.append(_run_plain(phase, np.ones(phase.shape), v, [PERIODIC] * 6, g, kvisc, case["scheme"], 0.0,
                                      case["steps"]))
            return out
        if case["kind"] != "adjoint":
            phase, den, vel, bc, g, kvisc = _flow_inputs(case, seed)
            den, vel = _run_plain(phase, den, vel, bc, g, kvisc, case["scheme"], case["magic"], case["steps"])
            return {"den": den, "vel": vel}
    return _exact_adjoint(case, seed)


def _exact_adjoint(case, seed):
    from torch.utils.checkpoint import checkpoint

    phase, uin, target, g, plane = _adjoint_inputs(case, seed)
    dev = _device()
    zero = np.zeros(phase.shape + (3,))
    plain = _Plain(phase, zero, ADJOINT_BC, case["scheme"], 0.1, case["magic"])
    tau = torch.tensor(case["tau"], dtype=torch.float64, device=dev, requires_grad=True)
    gt = torch.tensor(g, dtype=torch.float64, device=dev, requires_grad=True)
    ut = torch.tensor(uin, dtype=torch.float64, device=dev, requires_grad=True)
    one = torch.ones(phase.shape, dtype=torch.float64, device=dev)
    vel0 = torch.zeros(phase.shape + (3,), dtype=torch.float64, device=dev)

    def one_step(tau_, g_, u_, *f):
        plain.set_tau(tau_, case["magic"])
        vin = vel0.clone()
        vin[0, :, :, 0] = u_
        out, _, u = plain.step(list(f), g_, one, vin, one)
        return tuple(out) + tuple(x[plane] for x in u)

    f = tuple(torch.where(plain.fluid, W[q] * one, 0.0 * one) for q in range(19))
    for _ in range(case["steps"]):
        r = checkpoint(one_step, tau, gt, ut, *f, use_reentrant=False)
        f, up = r[:19], r[19:]
    u = torch.stack(up, -1)
    wet = plain.fluid[plane][..., None]
    diff = torch.where(wet, u - torch.from_numpy(target).to(dev), torch.zeros_like(u))
    loss = (diff ** 2).sum()
    loss.backward()
    uo = torch.where(wet, u, torch.zeros_like(u)).detach()
    return {"loss": float(loss.detach()), "u": uo.cpu().numpy(), "dtau": float(tau.grad), "dg": gt.grad.cpu().numpy(),
            "duin": ut.grad.cpu().numpy()}
