"""Performance cases of the voxel-elasticity solve path, by public entry points.

Each case is a dict of plain values.  ``prepare`` builds what a program holds
before the call (the solver context with its hierarchy, boundary conditions
and moduli, the load), ``run`` makes the call, ``work`` counts the bytes and
operations that the call cannot do without, ``exact`` gives the answer in 64
bits from plain torch and numpy.

Kinds:

* ``kbyu``: one matrix-free K*u on device vectors, the operator that a user's
  own Krylov loop calls (the reference's Solving_KbyU_MatrixFree);
* ``analysis``: new moduli, assembly and one solve, what a static analysis or
  a user's own design loop does per step; ``fp64`` is the reference's form,
  ``mixed_df`` the fast one;
* ``load``: one more load case on an assembled irregular model;
* ``block``: several load cases of one model in one call, from host vectors;
* ``study``: the learned start of a load-case study, a held-out case after
  training cases;
* ``simp``: iterations of the SIMP loop with its filter and OC update;
* ``stress``: nodal stress and von Mises recovery of a displacement field;
* ``net``: loss and gradient of the U-Net that proposes starts.

Solves run to tolerances of 1e-9 and 1e-10, as the runs do that others are
judged by: their displacements are then the system's own, whatever the
rounding on the way.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from sgldbench_gb300 import _lib, domains
from sgldbench_gb300.net import UNet
from sgldbench_gb300.solver import LoadCases, VoxelSolver

OMEGA = 0.6                  # Jacobi weight of the benchmark configurations
GAUSS = 0.577350269189626    # the reference's Gauss point, as it writes it


def listed():
    return [
        # the smallest benchmark model (64 x 32 x 32): launches and latency count
        {"name": "kbyu_64x32x32", "kind": "kbyu", "shape": "box", "nx": 64, "ny": 32, "nz": 32, "levels": 4,
         "step4": True},
        # the SIMP-graded benchmark model, 12.8 M DOFs
        {"name": "kbyu_256x128x128", "kind": "kbyu", "shape": "box", "nx": 256, "ny": 128, "nz": 128, "levels": 5,
         "step4": False},
        # a quick static analysis in the reference's own form
        {"name": "fp64_64x32x32", "kind": "analysis", "shape": "box", "nx": 64, "ny": 32, "nz": 32, "levels": 4,
         "step4": True, "precision": "fp64", "tol": 1e-9},
        # the plain FP64 solve that others are judged by, at 12.8 M DOFs
        {"name": "fp64_256x128x128", "kind": "analysis", "shape": "box", "nx": 256, "ny": 128, "nz": 128, "levels": 5,
         "step4": False, "precision": "fp64", "tol": 1e-9},
        # the same two models through the mixed solve
        {"name": "mixed_64x32x32", "kind": "analysis", "shape": "box", "nx": 64, "ny": 32, "nz": 32, "levels": 4,
         "step4": True, "precision": "mixed_df", "tol": 1e-9},
        {"name": "mixed_256x128x128", "kind": "analysis", "shape": "box", "nx": 256, "ny": 128, "nz": 128,
         "levels": 5, "step4": False, "precision": "mixed_df", "tol": 1e-9},
        # the large stress analysis's shape family (thresholded blobs, 30 % solid): most of the
        # grid is empty
        {"name": "load_blobs_384x192x192", "kind": "load", "shape": "blobs", "nx": 384, "ny": 192, "nz": 192,
         "levels": 6, "step4": False, "precision": "mixed_df", "tol": 1e-9},
        # four load cases on one irregular part, sizes that need padding, host vectors in and out
        {"name": "block4_blobs_125x61x67", "kind": "block", "shape": "blobs", "nx": 125, "ny": 61, "nz": 67,
         "levels": 4, "step4": False, "precision": "mixed", "tol": 1e-10, "loads": 4},
        # a held-out case of a load-case study, started from what three training solves taught
        {"name": "study_blobs_192x96x96", "kind": "study", "shape": "blobs", "nx": 192, "ny": 96, "nz": 96,
         "levels": 5, "step4": False, "precision": "mixed_df", "tol": 1e-9, "loads": 3},
        # the first iterations of a topology optimisation
        {"name": "simp_96x48x48", "kind": "simp", "shape": "box", "nx": 96, "ny": 48, "nz": 48, "levels": 4,
         "step4": False, "precision": "mixed_df", "tol": 1e-9, "loops": 4},
        # stress recovery of a finished solve, everything back on the host
        {"name": "stress_blobs_192x96x96", "kind": "stress", "shape": "blobs", "nx": 192, "ny": 96, "nz": 96,
         "levels": 5, "step4": False},
        # one gradient of the start network on the grid it has in the large analysis
        {"name": "net_65x33x33", "kind": "net", "nx": 65, "ny": 33, "nz": 33},
    ]


def _levels(nx, ny, nz):
    """Dyadic levels that leave about a thousand elements on the coarsest, as the benchmark models have."""
    return max(3, 1 + math.ceil(math.log2(max(2.0, (nx * ny * nz / 1024) ** (1 / 3))) - 0.2))


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["kbyu", "kbyu", "analysis", "analysis", "load", "block", "study", "simp", "stress", "net"])
    if kind == "net":
        return {"kind": kind, "nx": log_int(17, 65), "ny": log_int(9, 33), "nz": log_int(9, 33)}
    irregular = kind in ("load", "block", "study") or (kind in ("kbyu", "stress") and rng.random() < 0.5)
    # the long side; the others are around half of it, as in the benchmark models
    top = {"kbyu": 256, "analysis": 160, "load": 256, "block": 128, "study": 192, "simp": 96, "stress": 192}[kind]
    nx = log_int(96 if irregular else 24, top)
    ny, nz = (max(48 if irregular else 12, int(nx * rng.uniform(0.4, 0.52))) for _ in range(2))
    case = {"kind": kind, "shape": "blobs" if irregular else "box", "nx": nx, "ny": ny, "nz": nz,
            "levels": _levels(nx, ny, nz), "step4": False}
    if kind == "analysis":
        case["precision"] = rng.choice(["fp64", "mixed", "mixed_df"])
        case["tol"] = 1e-9
    elif kind == "block":
        case["precision"], case["tol"], case["loads"] = "mixed", 1e-10, rng.randint(2, 4)
    elif kind in ("load", "study", "simp"):
        case["precision"], case["tol"] = rng.choice(["mixed", "mixed_df"]), 1e-9
        if kind == "study":
            case["loads"] = rng.randint(2, 3)
        if kind == "simp":
            case["loops"] = rng.randint(2, 4)
    return case


# ---- inputs -------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _voxels(shape, nx, ny, nz):
    """The model, (ny, nx, nz): a file that a user has; the seed draws what acts on it."""
    return domains.cuboid(nx, ny, nz) if shape == "box" else domains.gaussian_blobs(nx, ny, nz, seed=0)


@functools.lru_cache(maxsize=4)
def _padded(shape, nx, ny, nz, levels):
    m = 2 ** (levels - 1)
    out = np.zeros([-(-d // m) * m for d in (ny, nx, nz)], bool)
    out[:ny, :nx, :nz] = _voxels(shape, nx, ny, nz)
    return out


def _grid(case):
    return _padded(case["shape"], case["nx"], case["ny"], case["nz"], case["levels"])


@functools.lru_cache(maxsize=8)
def _node_numbers(shape, nx, ny, nz, levels):
    """(1-based full-grid numbers of the compact nodes, active nodes, active elements)."""
    v = _padded(shape, nx, ny, nz, levels)
    n = np.zeros([d + 1 for d in v.shape], bool)
    for dy in (0, 1):
        for dx in (0, 1):
            for dz in (0, 1):
                n[dy:dy + v.shape[0], dx:dx + v.shape[1], dz:dz + v.shape[2]] |= v
    numbers = np.flatnonzero(n.reshape(-1, order="F")) + 1
    return numbers, numbers.size, int(v.sum())


def _numbers(case):
    return _node_numbers(case["shape"], case["nx"], case["ny"], case["nz"], case["levels"])


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _modulus(case, seed):
    """SIMP-graded moduli of the model's elements on the GPU: smoothed noise as density, E = Emin + rho^3 (1 - Emin)."""
    v = _grid(case)
    r = torch.rand((1, 1, v.shape[2], v.shape[1], v.shape[0]), generator=_generator(seed), device="cuda",
                   dtype=torch.float64)
    for ax in (2, 3, 4):   # three-voxel binomial smoothing, twice per axis
        for _ in range(2):
            a = r.narrow(ax, 0, 1)
            b = r.narrow(ax, r.shape[ax] - 1, 1)
            p = torch.cat([a, r, b], ax)
            n = r.shape[ax]
            r = 0.25 * p.narrow(ax, 0, n) + 0.5 * p.narrow(ax, 1, n) + 0.25 * p.narrow(ax, 2, n)
    rho = (r - r.min()) / (r.max() - r.min()) * (1.0 - 1e-1) + 1e-1
    e = (1e-9 + rho ** 3 * (1.0 - 1e-9)).reshape(-1)   # z slowest, y fastest: the column-major element order
    on = torch.from_numpy(v.reshape(-1, order="F").copy()).cuda()
    return e[on].contiguous()


def _fixed_and_loads(case, seed, count):
    v, numbers = _grid(case), _numbers(case)[0]
    rng = np.random.default_rng(seed)
    if case["shape"] == "box":
        F, fixed = domains.cantilever3(v, numbers, nelx=case["nx"])
        on = np.flatnonzero(F)
        loads = []
        for _ in range(count):   # the edge load, turned by up to 30 degrees
            d = np.array([0.0, 0.0, -1.0]) + np.tan(np.deg2rad(30)) * rng.uniform(-0.5, 0.5, 3)
            d /= np.linalg.norm(d)
            f = np.zeros((numbers.size, 3))
            f[on // 3] = d / on.size
            loads.append(f.reshape(-1))
        return fixed, loads
    fixed = domains.fix_bottom_layers(v, numbers)
    cases = domains.perturbed_patch_cases(v, numbers, count, seed=seed)
    return fixed, [domains.dense_load(numbers.size, c) for c in cases]


def _solver(case, fixed, modulus):
    s = VoxelSolver(_grid(case), num_levels=case["levels"], non_dyadic=int(case["step4"]), omega=OMEGA, pad=False)
    s.set_fixed_dofs(fixed)
    s.set_modulus_device(modulus.data_ptr())
    return s


def _net_inputs(case, seed):
    rng = np.random.default_rng(seed)
    v = case["nx"] * case["ny"] * case["nz"]
    x = rng.standard_normal((v, 8), dtype=np.float32)
    x[:, 7] = rng.random(v) < 0.3   # the active-node mask
    x[:, :7] *= x[:, 7:]
    t = rng.standard_normal((v, 3), dtype=np.float32) * x[:, 7:]
    return x, t, np.ascontiguousarray(x[:, 7])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "net":
        x, t, m = _net_inputs(case, seed)
        return {"case": case, "net": UNet((case["ny"], case["nx"], case["nz"]), 8, 3, levels=4, seed=1), "x": x,
                "t": t, "m": m}
    count = case.get("loads", 1) + (kind == "study")
    fixed, loads = _fixed_and_loads(case, seed, count)
    solid = kind in ("load", "block", "study")
    modulus = (torch.ones(_numbers(case)[2], dtype=torch.float64, device="cuda") if solid else _modulus(case, seed))
    torch.cuda.synchronize()   # the library's stream does not wait for torch's
    s = _solver(case, fixed, modulus)
    st = {"case": case, "solver": s, "modulus": modulus}
    if kind == "kbyu":
        st["u"] = torch.randn(s.numDOFs, generator=_generator(seed + 1), device="cuda", dtype=torch.float64)
        st["y"] = torch.empty_like(st["u"])
    elif kind == "stress":
        st["u"] = np.random.default_rng(seed).standard_normal(s.numDOFs)
    elif kind == "simp":
        st["load"] = loads[0]
    else:
        s.Solving_AssembleFEAstencil()
        if kind == "block":
            st["loads"] = np.stack(loads)
        else:
            st["b"] = torch.from_numpy(loads[-1]).cuda()
            st["x"] = torch.zeros_like(st["b"])
        if kind == "study":
            st["study"] = LoadCases(s, max_basis=8)
            for f in loads[:-1]:
                st["study"].solve(f, train=True, tol=case["tol"], precision=case["precision"])
    torch.cuda.synchronize()
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "net":
        loss, grad = state["net"].grad(state["x"], state["t"], state["m"])
        return {"loss": loss, "grad": grad}
    s = state["solver"]
    if kind == "kbyu":
        s._check(_lib.load().sgld_kbyu_device(s.ctx, ctypes.c_void_p(state["u"].data_ptr()),
                                              ctypes.c_void_p(state["y"].data_ptr())))
        return state["y"]
    if kind == "stress":
        nodal, vm_node, vm_element = s.FEA_StressAnalysis(state["u"])
        return {"nodal": nodal, "vm_node": vm_node, "vm_element": vm_element}
    if kind == "simp":
        xphys, history = s.TopOpti_GlobalVolumeConstraint(state["load"], volfrac=0.3, rMin=1.5, nLoop=case["loops"],
                                                          tol=case["tol"], maxIT=5000, precision=case["precision"])
        return {"xphys": xphys, "compliance": [h["compliance"] for h in history]}
    if kind == "block":
        u, _ = s.solve_block(state["loads"], tol=case["tol"], maxIT=5000, precision=case["precision"])
        return u
    b, x = state["b"], state["x"]
    if kind == "study":
        state["study"].solve_device(b.data_ptr(), x.data_ptr(), tol=case["tol"], precision=case["precision"])
        return x
    if kind == "analysis":
        s.set_modulus_device(state["modulus"].data_ptr())
        s.Solving_AssembleFEAstencil()
    s.pcg_device(b.data_ptr(), x.data_ptr(), case["tol"], 5000, precision=case["precision"])
    return x


# ---- what a call cannot do without -------------------------------------------------
# Operations of one K*u per active element with every butterfly shared between the
# elements around an edge and a face, and of one multigrid V-cycle and the vector
# updates of an iteration per active node; iterations at 1e-9 as the method takes
# them on these models.
KU_OPS, CYCLE_OPS, ITERATIONS = 130, 150, 90


def work(case):
    kind = case["kind"]
    if kind == "net":
        v = case["nx"] * case["ny"] * case["nz"]
        # multiply-adds per finest voxel of the four-level network, forward and twice backward
        per = 27 * (8 * 16 + 2 * 16 * 16) + 27 * (16 * 32 + 2 * 32 * 32 + 32 * 16) / 8 \
            + 27 * (32 * 48 + 2 * 48 * 48 + 48 * 32) / 64 + 27 * (48 * 64 + 64 * 64 + 64 * 48) / 512 + 16 * 3
        return {"bytes": 4.0 * 12 * v, "flops": 2.0 * 3 * per * v}
    _, nodes, elements = _numbers(case)
    vector, moduli = 24.0 * nodes, 8.0 * elements
    step = KU_OPS * elements + CYCLE_OPS * nodes
    if kind == "kbyu":
        return {"bytes": 2 * vector + moduli, "flops": float(KU_OPS * elements)}
    if kind == "stress":
        # 9 differences and Hooke's law per corner, averages, two von Mises values
        return {"bytes": vector + moduli + 56.0 * nodes + 8.0 * elements, "flops": 250.0 * nodes}
    passes = {"simp": case.get("loops", 1), "block": case.get("loads", 1)}.get(kind, 1)
    return {"bytes": passes * (2 * vector + moduli), "flops": float(passes * ITERATIONS * step)}


# ---- the same in 64 bits ------------------------------------------------------------
OFFSETS = [(dy, dx, dz) for dz in (0, 1) for dx in (0, 1) for dy in (0, 1)]   # (row, x, z) corners


def _strain(s, t, p):
    """6 x 24 strain-displacement matrix of the unit voxel at (s, t, p); rows run against t."""
    b = np.zeros((6, 24))
    for n, (dy, dx, dz) in enumerate(OFFSETS):
        ns, nt, np_ = 2 * dx - 1, 1 - 2 * dy, 2 * dz - 1
        ds = 0.25 * ns * (1 + nt * t) * (1 + np_ * p)
        dt = 0.25 * nt * (1 + ns * s) * (1 + np_ * p)
        dp = 0.25 * np_ * (1 + ns * s) * (1 + nt * t)
        b[0, 3 * n], b[1, 3 * n + 1], b[2, 3 * n + 2] = ds, dt, dp
        b[3, 3 * n + 1], b[3, 3 * n + 2] = dp, dt
        b[4, 3 * n], b[4, 3 * n + 2] = dp, ds
        b[5, 3 * n], b[5, 3 * n + 1] = dt, ds
    return b


def _hooke(nu=0.3):
    d = np.zeros((6, 6))
    d[:3, :3] = nu / ((1 + nu) * (1 - 2 * nu))
    d[range(3), range(3)] = (1 - nu) / ((1 + nu) * (1 - 2 * nu))
    d[range(3, 6), range(3, 6)] = 0.5 / (1 + nu)
    return d


GAUSS_POINTS = [(s, t, p) for p in (-GAUSS, GAUSS) for t in (-GAUSS, GAUSS) for s in (-GAUSS, GAUSS)]


class _Exact:
    """The model's elements in plain torch: corner nodes per element, K*u, corner stresses."""

    def __init__(self, case, fixed):
        v = _grid(case)
        ny, nx, nz = v.shape
        numbers, self.nodes, self.elements = _numbers(case)
        full = torch.full(((ny + 1) * (nx + 1) * (nz + 1),), -1, dtype=torch.int64, device="cuda")
        full[torch.from_numpy(numbers - 1).cuda()] = torch.arange(self.nodes, device="cuda")
        e = torch.from_numpy(np.flatnonzero(v.reshape(-1, order="F"))).cuda()
        y, x, z = e % ny, (e // ny) % nx, e // (ny * nx)
        self.corner = torch.stack([full[(y + dy) + (ny + 1) * ((x + dx) + (nx + 1) * (z + dz))]
                                   for dy, dx, dz in OFFSETS], 1)
        ke = sum(_strain(*g).T @ _hooke() @ _strain(*g) for g in GAUSS_POINTS) / 8
        self.ke = torch.from_numpy(ke).cuda()
        self.free = torch.from_numpy(~fixed).cuda().double()

    def kbyu(self, u, modulus):
        ue = u.reshape(-1, 3)[self.corner].reshape(-1, 24)
        f = (ue @ self.ke) * modulus[:, None]
        y = torch.zeros(self.nodes, 3, dtype=torch.float64, device="cuda")
        for k in range(8):
            y.index_add_(0, self.corner[:, k], f[:, 3 * k:3 * k + 3])
        return y.reshape(-1) * self.free

    def diagonal(self, modulus):
        d = torch.zeros(self.nodes, 3, dtype=torch.float64, device="cuda")
        kd = torch.diagonal(self.ke)
        for k in range(8):
            d.index_add_(0, self.corner[:, k], modulus[:, None] * kd[3 * k:3 * k + 3][None, :])
        return d.reshape(-1)

    def solve(self, b, modulus, most=6000):
        """Jacobi-preconditioned CG to 1e-13."""
        d = self.diagonal(modulus)
        x = torch.zeros_like(b)
        r = b.clone()
        z = r / d * self.free
        p = z.clone()
        rz = r @ z
        stop = 1e-13 * float(b.norm())
        for k in range(most):
            q = self.kbyu(p, modulus)
            a = rz / (p @ q)
            x += a * p
            r -= a * q
            if k % 50 == 49 and float(r.norm()) < stop:
                return x
            z = r / d * self.free
            new = r @ z
            p = z + (new / rz) * p
            rz = new
        return None

    def stress(self, u, modulus):
        shape = np.array([[(1 + (2 * dx - 1) * s) * (1 + (1 - 2 * dy) * t) * (1 + (2 * dz - 1) * p) / 8
                           for dy, dx, dz in OFFSETS] for s, t, p in GAUSS_POINTS])
        at_gauss = np.stack([_hooke() @ _strain(*g) for g in GAUSS_POINTS])
        at_corner = np.einsum("ng,gkj->nkj", np.linalg.inv(shape), at_gauss)
        m = torch.from_numpy(at_corner.reshape(48, 24).T.copy()).cuda()
        ue = u.reshape(-1, 3)[self.corner].reshape(-1, 24)
        c = ((ue @ m) * modulus[:, None]).reshape(-1, 8, 6)
        total = torch.zeros(self.nodes, 6, dtype=torch.float64, device="cuda")
        count = torch.zeros(self.nodes, dtype=torch.float64, device="cuda")
        for k in range(8):
            total.index_add_(0, self.corner[:, k], c[:, k])
            count.index_add_(0, self.corner[:, k], torch.ones(self.elements, dtype=torch.float64, device="cuda"))
        nodal = total / count[:, None]

        def mises(v):
            a, b, d = v[:, 0] - v[:, 1], v[:, 1] - v[:, 2], v[:, 2] - v[:, 0]
            return torch.sqrt(0.5 * (a * a + b * b + d * d) + 3 * (v[:, 3:] ** 2).sum(1))

        return nodal, mises(nodal), torch.sqrt(mises(nodal[self.corner].mean(1)))


def _exact_net(case, seed):
    """The network's loss and gradient in float64, from the library's own initial weights."""
    net = UNet((case["ny"], case["nx"], case["nz"]), 8, 3, levels=4, seed=1)
    params = torch.from_numpy(net.get_params()).cuda().double().requires_grad_()
    net.close()
    x, t, mask = (torch.from_numpy(a).cuda().double() for a in _net_inputs(case, seed))
    widths, dims, at = [16, 32, 48, 64], [(case["nz"], case["nx"], case["ny"])], 0
    for _ in range(3):
        dims.append(tuple((d + 1) // 2 for d in dims[-1]))

    def conv(v, cout, taps=27):   # v: (z, x, y, channels), zero padding
        nonlocal at
        cin = v.shape[3]
        w = params[at:at + taps * cin * cout].reshape(taps, cin, cout)
        b = params[at + taps * cin * cout:at + taps * cin * cout + cout]
        at += taps * cin * cout + cout
        if taps == 1:
            return v @ w[0] + b
        nz, nx, ny, _ = v.shape
        p = torch.nn.functional.pad(v, (0, 0, 1, 1, 1, 1, 1, 1))
        out = b
        for k in range(27):
            dz, dx, dy = k // 9, (k // 3) % 3, k % 3
            out = out + p[dz:dz + nz, dx:dx + nx, dy:dy + ny] @ w[k]
        return out

    def pool(v, size):   # mean over the children that exist
        one = torch.ones_like(v[..., :1])
        grow = (0, 0) + sum(((0, 2 * n - o) for n, o in zip(reversed(size), reversed(v.shape[:3]))), ())
        v, one = torch.nn.functional.pad(v, grow), torch.nn.functional.pad(one, grow)

        def halves(a):
            return a.reshape(size[0], 2, size[1], 2, size[2], 2, -1).sum((1, 3, 5))

        return halves(v) / halves(one)

    v, skips = x.reshape(*dims[0], 8), []
    for level in range(4):
        if level:
            v = pool(v, dims[level])
        v = torch.relu(conv(v, widths[level]))
        v = torch.relu(conv(v, widths[level]))
        skips.append(v)
    for level in (2, 1, 0):
        v = torch.relu(conv(v, widths[level]))
        nz, nx, ny = dims[level]
        v = v.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)[:nz, :nx, :ny] + skips[level]
        v = torch.relu(conv(v, widths[level]))
    y = conv(v, 3, taps=1).reshape(-1, 3)
    loss = (mask[:, None] * (y - t) ** 2).sum() / (3 * mask.sum())
    loss.backward()
    return {"loss": float(loss.detach()), "grad": params.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "net":
        return _exact_net(case, seed)
    if kind not in ("kbyu", "stress", "analysis"):
        return None
    if kind == "analysis" and _numbers(case)[2] > 100_000:
        return None   # plain CG takes too long
    fixed, loads = _fixed_and_loads(case, seed, 1)
    modulus = _modulus(case, seed)
    model = _Exact(case, fixed)
    if kind == "kbyu":
        u = torch.randn(3 * model.nodes, generator=_generator(seed + 1), device="cuda", dtype=torch.float64)
        return model.kbyu(u, modulus)
    if kind == "analysis":
        return model.solve(torch.from_numpy(loads[0]).cuda(), modulus)
    u = torch.from_numpy(np.random.default_rng(seed).standard_normal(3 * model.nodes)).cuda()
    nodal, vm_node, vm_element = model.stress(u, modulus)
    return {"nodal": nodal, "vm_node": vm_node, "vm_element": vm_element}
