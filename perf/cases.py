"""The work that users of libgmgs have it do, as measurable cases.

Each case is a dict of plain values; `kind` names the public entry point:

  operator   Solver.apply_operator_dev: K x of the finest level, the `@AtX`
             handle of a caller's own Krylov loop (device buffers)
  vcycle     Solver.apply_preconditioner_dev: one V-cycle, the `@Vcycle` handle
  solve      Solver.solve_dev on a handle that keeps its model: a new load case
             on a known part, U left on the device
  gradient   gmgs.autograd.compliance, forward and backward: one step of a
             density optimisation (new densities, new hierarchy, solve, dJ/drho)
  analysis   occupancy in host memory -> Solver -> set_bc -> solve -> stress,
             all results in host memory: a one-shot analysis of a new part

Sizes are those of the repository's benchmark workloads (nelx x nely x nelz of
42x37x64, 84x73x128, 169x147x256, 337x294x512; none is a multiple of the
coarsening factor, so every hierarchy is padded) and, in draw(), everything
between.  Parts are blocks with spherical voids fixed at z = 0 and loaded on
the top face, as in the benchmark workloads.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gmgs-3d_gb300"))
from gmgs import Solver, synthetic  # noqa: E402
from gmgs.autograd import compliance  # noqa: E402

OMEGA = 0.4      # the reference's default Jacobi weight
NU = 0.3
NOMINAL_ITERATIONS = 30   # PCG iterations work() counts (16 to 120 are usual)
EXACT_NODES = 1_000_000   # the largest part exact() solves (plain CG in 64 bits)
EXACT_OPERATOR_NODES = 8_000_000


def _case(name, kind, precision, nelx, nely, nelz, part, voids, levels=0, density=False, ex=1.0, ey=1.0, ez=1.0):
    """`part` seeds the voids' places: one part, of which prepare()'s seed gives load cases and densities."""
    return {"name": name, "kind": kind, "precision": precision, "nelx": nelx, "nely": nely, "nelz": nelz, "part": part,
            "voids": voids, "levels": levels, "density": density, "ex": ex, "ey": ey, "ez": ez}


def listed():
    small, middle, large = (42, 37, 64, 1001, 20), (169, 147, 256, 1002, 40), (337, 294, 512, 1004, 120)
    return [
        # a small part in a caller's Krylov loop: latency and launches
        _case("operator_fp64_42", "operator", "fp64", *small, levels=4),
        # the same on a 19M-DOF part: throughput of the FP64 operator
        _case("operator_fp64_169", "operator", "fp64", *middle),
        # the preconditioner handle in the default precision, voxels that are not cubes (a voxelised mesh)
        _case("vcycle_fp64_84", "vcycle", "fp64", 84, 73, 128, 1003, 30, ex=1.02, ey=0.97, ez=1.0),
        # and in mixed precision on a larger part
        _case("vcycle_mixed_169", "vcycle", "mixed", *middle),
        # the default solve (FP64, the drop-in for the reference) on its smallest demo size
        _case("solve_fp64_42", "solve", "fp64", *small, levels=4),
        # the default solve on an ordinary part, 19M DOFs
        _case("solve_fp64_169", "solve", "fp64", *middle),
        # mixed precision: small parts (launch bound), ordinary ones, the headline size (153M DOFs)
        _case("solve_mixed_42", "solve", "mixed", *small, levels=4),
        _case("solve_mixed_169", "solve", "mixed", *middle),
        _case("solve_mixed_337", "solve", "mixed", *large, levels=6),
        # density optimisation: every step brings new densities, so the hierarchy is part of the pass
        _case("gradient_fp64_42", "gradient", "fp64", 42, 37, 64, 1001, 0, density=True),
        _case("gradient_mixed_84", "gradient", "mixed", 84, 73, 128, 1003, 0, density=True),
        # a new part from host memory to displacement and stress in host memory
        _case("analysis_mixed_169", "analysis", "mixed", *middle, ex=1.01, ey=0.98, ez=1.0),
    ]


# nelz ranges per kind and precision (the block keeps roughly the benchmark's
# 0.65 : 0.57 : 1 proportions, each side drawn around them)
_RANGES = [("operator", "fp64", 40, 256), ("vcycle", "fp64", 48, 160), ("vcycle", "mixed", 64, 256),
           ("solve", "fp64", 48, 176), ("solve", "mixed", 48, 384), ("gradient", "fp64", 40, 72),
           ("gradient", "mixed", 48, 128), ("analysis", "mixed", 64, 256)]


def draw(rng):
    kind, precision, lo, hi = rng.choice(_RANGES)
    nz = round(math.exp(rng.uniform(math.log(lo), math.log(hi))))
    nx = max(24, min(337, round(nz * rng.uniform(0.55, 0.75))))
    ny = max(24, min(294, round(nz * rng.uniform(0.5, 0.65))))
    density = kind == "gradient"
    ex, ey, ez = (round(rng.uniform(0.95, 1.05), 3) for _ in range(3)) if rng.random() < 0.5 else (1.0, 1.0, 1.0)
    c = _case("", kind, precision, nx, ny, nz, part=rng.randrange(1 << 20), voids=0 if density else rng.randint(0, 40),
              density=density, ex=ex, ey=ey, ez=ez)
    del c["name"]
    return c


# --------------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda")


@functools.lru_cache(maxsize=2)
def _voxels(nelx, nely, nelz, voids, part):
    """(y, x, z) int32 voxels, y fastest, as the benchmark workloads make them."""
    return np.asfortranarray(synthetic.sphere_voids(nelx, nely, nelz, voids, part))


def _node_sum(e):
    """Sum of the element values e (z, x, y) around every node."""
    n = torch.zeros([s + 1 for s in e.shape], dtype=e.dtype, device=e.device)
    z, x, y = e.shape
    for k in range(8):
        n[k >> 2:(k >> 2) + z, k >> 1 & 1:(k >> 1 & 1) + x, k & 1:(k & 1) + y] += e
    return n


def _part(case, seed):
    """Voxels, 1-based fixed node ids and loads (id, fx, fy, fz) as numpy, densities or None, the solid mask."""
    rng = np.random.default_rng(seed)
    vox = _voxels(*(case[k] for k in ("nelx", "nely", "nelz", "voids", "part")))
    solid = torch.from_numpy(vox.transpose(2, 1, 0)).to(_device()) == 1               # (z, x, y)
    node = _node_sum(solid.to(torch.uint8)) > 0
    ids = torch.cumsum(node.reshape(-1), 0, dtype=torch.int32).reshape(node.shape)   # compact, y fastest
    fixed = ids[0][node[0]].cpu().numpy()
    top = ids[-1][node[-1]].cpu().numpy()
    loads = np.zeros((len(top), 4))
    loads[:, 0] = top
    loads[:, 1:3] = rng.uniform(-0.2, 0.2, size=(len(top), 2)) / len(top)
    loads[:, 3] = -rng.uniform(0.5, 1.5, size=len(top)) / len(top)
    rho = rng.uniform(0.2, 1.0, size=int(solid.sum())) if case["density"] else None
    return vox, fixed, loads, rho, solid, node


def _field(case, seed, n_node, scale=1.0):
    """A displacement-like vector (3 * n_node, interleaved): smooth in the node order's axes, with 1 % noise."""
    g = torch.Generator(device=_device()).manual_seed(seed)
    nx, ny = case["nelx"] + 1, case["nely"] + 1
    i = torch.arange(n_node, device=_device())
    t = torch.stack([i // ny % nx / nx, i % ny / ny, i / n_node], 1).double()          # (x, y, z)-like coordinates
    a = torch.rand((3, 3), generator=g, device=_device(), dtype=torch.float64) * 4 + 1
    u = torch.sin(t @ a) * t[:, 2:]
    u += 0.01 * (torch.rand((n_node, 3), generator=g, device=_device(), dtype=torch.float64) - 0.5)
    return (u * scale).reshape(-1).contiguous()


def _make_solver(case, vox):
    return Solver(vox, ele_size=(case["ex"], case["ey"], case["ez"]), omega=OMEGA, poisson_ratio=NU,
                  num_levels=case["levels"], precision=case["precision"])


def prepare(case, seed):
    vox, fixed, loads, rho, _, _ = _part(case, seed)
    st = {"kind": case["kind"], "case": case, "fixed": fixed, "loads": loads}
    if case["kind"] == "analysis":
        st["vox"] = vox
        return st
    s = st["solver"] = _make_solver(case, vox)
    s.set_bc(fixed, loads)
    n = s.num_nodes(1)
    if case["kind"] in ("operator", "vcycle"):
        st["x"] = _field(case, seed, n, 1.0 if case["kind"] == "operator" else 1e-3)
        st["y"] = torch.zeros_like(st["x"])
        s.set_tolerance(1e-3, 0)       # the operator handles exist after the first solve: one iteration
        s.solve_dev(None)
    elif case["kind"] == "solve":
        st["u"] = torch.zeros(3 * n, dtype=torch.float64, device=_device())
    elif case["kind"] == "gradient":
        st["rho"] = torch.tensor(rho, device=_device(), requires_grad=True)
    torch.cuda.synchronize()
    return st


def run(state):
    kind = state["kind"]
    if kind == "analysis":
        with _make_solver(state["case"], state["vox"]) as s:
            s.set_bc(state["fixed"], state["loads"])
            u = s.solve()
            nodal, voxel = s.stress()
            return {"u": u, "nodal": nodal, "voxel": voxel, "iterations": s.iterations}
    s = state["solver"]
    if kind == "operator":
        s.apply_operator_dev(state["x"].data_ptr(), state["y"].data_ptr())
        return {"y": state["y"]}
    if kind == "vcycle":
        s.apply_preconditioner_dev(state["x"].data_ptr(), state["y"].data_ptr())
        return {"z": state["y"]}
    if kind == "solve":
        s.solve_dev(state["u"].data_ptr())
        return {"u": state["u"], "iterations": s.iterations}
    rho = state["rho"]
    rho.grad = None
    j = compliance(rho, s)
    j.backward()
    return {"j": j.detach(), "grad": rho.grad}


def work(case):
    """Vectors that one pass reads and writes once each; K x of the interior stencil (27 blocks of 3 x 3)."""
    n = (case["nelx"] + 1) * (case["nely"] + 1) * (case["nelz"] + 1)
    ne = case["nelx"] * case["nely"] * case["nelz"]
    b = 8 if case["precision"] == "fp64" else 4
    kx = 2 * 243
    if case["kind"] == "operator":
        return {"bytes": 2 * 24 * n + ne, "flops": kx * n}
    down_up = 7 * 3 * b            # r, w in and r' out; r, r', w in and z out
    if case["kind"] == "vcycle":
        return {"bytes": 2 * 24 * n + down_up * n * 8 / 7, "flops": (kx + 60) * n * 8 / 7}
    state = (7 + 4) * 3 * b        # x, r, p, q, w of the update; z, p, p, q of the direction
    its = NOMINAL_ITERATIONS
    by = its * (state + down_up * 8 / 7) * n + 48 * n
    fl = its * (2 * kx + (kx + 60) * 8 / 7 + 40) * n
    if case["kind"] == "gradient":
        by += (8 + 8 + 24) * ne
        fl += 2 * 600 * ne
    if case["kind"] == "analysis":
        by += 4 * ne + 24 * n + 48 * n + 24 * ne
        fl += 200 * n
    return {"bytes": by, "flops": fl}


# ---------------------------------------------------------------- 64-bit values
# The finite-element model in plain torch: trilinear box elements, 2 x 2 x 2
# Gauss points, isotropic Hooke's law with E = 1.  Element corner k sits at
# offsets (z, x, y) = (k >> 2, k >> 1 & 1, k & 1); physical y runs against the
# y index.
def _hooke():
    lam, mu = NU / ((1 + NU) * (1 - 2 * NU)), 0.5 / (1 + NU)
    d = np.zeros((6, 6))
    d[:3, :3] = lam
    d[np.arange(3), np.arange(3)] += 2 * mu
    d[np.arange(3, 6), np.arange(3, 6)] = mu
    return d


def _strain(case, z, x, y):
    """B (6 x 24) at the local point (z, x, y) of [0, 1]^3; rows xx yy zz yz zx xy, columns 3 * corner + component."""
    b = np.zeros((6, 24))
    for k in range(8):
        f = [(t if c else 1 - t, 1.0 if c else -1.0) for t, c in ((z, k >> 2), (x, k >> 1 & 1), (y, k & 1))]
        gx = f[0][0] * f[1][1] * f[2][0] / case["ex"]
        gy = -f[0][0] * f[1][0] * f[2][1] / case["ey"]
        gz = f[0][1] * f[1][0] * f[2][0] / case["ez"]
        c = 3 * k
        b[0, c] = b[4, c + 2] = b[5, c + 1] = gx
        b[1, c + 1] = b[3, c + 2] = b[5, c] = gy
        b[2, c + 2] = b[3, c + 1] = b[4, c] = gz
    return b


def _stiffness(case):
    g = 0.5 + np.array([-0.5, 0.5]) / math.sqrt(3.0)
    v = case["ex"] * case["ey"] * case["ez"] / 8
    return sum(v * _strain(case, a, b, c).T @ _hooke() @ _strain(case, a, b, c) for a in g for b in g for c in g)


class _Model:
    """K u on dense fields u (3, z, x, y), with an element scale (0 = void)."""

    def __init__(self, case, scale, fixed):
        self.ke = torch.tensor(_stiffness(case), device=_device())
        self.scale, self.fixed = scale, fixed
        self.diag = torch.zeros((3,) + fixed.shape, dtype=torch.float64, device=_device())
        for k, s in self.corners():
            for c in range(3):
                self.diag[c][s] += self.ke[3 * k + c, 3 * k + c] * scale

    def corners(self):
        z, x, y = self.scale.shape
        return [(k, (slice(k >> 2, (k >> 2) + z), slice(k >> 1 & 1, (k >> 1 & 1) + x), slice(k & 1, (k & 1) + y)))
                for k in range(8)]

    def element(self, u):
        return torch.stack([u[c][s] for _, s in self.corners() for c in range(3)]).reshape(24, -1)

    def apply(self, u):
        f = (self.ke @ self.element(u)).reshape((24,) + self.scale.shape) * self.scale
        y = torch.zeros_like(u)
        for k, s in self.corners():
            for c in range(3):
                y[c][s] += f[3 * k + c]
        return y.masked_fill_(self.fixed, 0.0)

    def solve(self, f):
        """Jacobi-preconditioned CG to a residual of 1e-11."""
        w = torch.where((self.diag > 0) & ~self.fixed, 1 / self.diag, torch.zeros_like(self.diag))
        f = f.masked_fill(self.fixed, 0.0)
        u, r = torch.zeros_like(f), f.clone()
        p = w * r
        rz, stop = (r * p).sum(), 1e-11 * f.norm()
        for it in range(6000):
            q = self.apply(p)
            a = rz / (p * q).sum()
            u += a * p
            r -= a * q
            if it % 20 == 0 and r.norm() < stop:
                break
            z = w * r
            new = (r * z).sum()
            p = z + new / rz * p
            rz = new
        return u


def exact(case, seed):
    n = (case["nelx"] + 1) * (case["nely"] + 1) * (case["nelz"] + 1)
    kind = case["kind"]
    if kind == "vcycle" or n > (EXACT_OPERATOR_NODES if kind == "operator" else EXACT_NODES):
        return None
    _, fixed, loads, rho, solid, node = _part(case, seed)
    dev = _device()
    scale = solid.double()
    if rho is not None:
        scale[solid] = torch.tensor(rho, device=dev) ** 3
    at = torch.nonzero(node.reshape(-1)).reshape(-1)               # compact id - 1 -> dense node
    fix = torch.zeros(node.numel(), dtype=torch.bool, device=dev)
    fix[at[torch.tensor(fixed - 1, device=dev).long()]] = True
    m = _Model(case, scale, fix.reshape(node.shape))

    def dense(v):
        d = torch.zeros((3, node.numel()), dtype=torch.float64, device=dev)
        d[:, at] = v.reshape(-1, 3).T
        return d.reshape((3,) + node.shape)

    def compact(d):
        return d.reshape(3, -1)[:, at].T.contiguous()

    if kind == "operator":
        return {"y": compact(m.apply(dense(_field(case, seed, len(at))))).reshape(-1)}
    f = torch.zeros((len(at), 3), dtype=torch.float64, device=dev)
    f[torch.tensor(loads[:, 0], device=dev).long() - 1] = torch.tensor(loads[:, 1:], device=dev)
    u = m.solve(dense(f))
    if kind == "gradient":
        ue = m.element(u)
        energy = (ue * (m.ke @ ue)).sum(0).reshape(scale.shape)[solid]
        return {"j": (dense(f) * u).sum(), "grad": -3 * torch.tensor(rho, device=dev) ** 2 * energy}
    if kind == "solve":
        return {"u": compact(u).reshape(-1), "iterations": None}
    ue, d = m.element(u), torch.tensor(_hooke(), device=dev)
    nodal = torch.zeros((6,) + node.shape, dtype=torch.float64, device=dev)
    for k, s in m.corners():
        b = torch.tensor(_strain(case, k >> 2, k >> 1 & 1, k & 1), device=dev)
        nodal[(slice(None),) + s] += (d @ b @ ue).reshape((6,) + scale.shape) * scale
    nodal = (nodal / _node_sum(solid.double()).clamp_(min=1)).reshape(6, -1)[:, at].T.contiguous()
    centre = torch.tensor(_strain(case, 0.5, 0.5, 0.5), device=dev)
    voxel = ((d @ centre @ ue).reshape((6,) + scale.shape) * scale)[:, solid].T.contiguous()
    return {"u": compact(u).reshape(-1), "nodal": nodal, "voxel": voxel, "iterations": None}
