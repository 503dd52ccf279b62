"""The work that users of this library have it do, as cases to be measured.

Each case is one call (or one short loop of calls) through the package's public entry points:

* apply64     one FP64 operator apply on device vectors (MatrixFreeOperator.matvec_dev), as a caller's own
              Krylov loop or eigensolver uses it
* apply32     one FP32 tensor-core apply on device vectors (MatrixFreeOperator.matvec_f32_dev)
* solve       one Jacobi-PCG solve on device vectors (PcgSolver.solve_dev), FP64 or mixed precision
* immersed    the same solve of a fictitious-domain problem: the unit cube minus three cylinders, elements
              scaled by SIMP density times volume fraction
* batched     several uneven designs solved by one call on host arrays (solve_batched)
* topopt      a few design iterations of the SIMP cantilever with several load cases (CantileverTopOpt.run)

Sizes are the ones of the repository's benchmark and tests (24x16x12, 128x64x64, 256x128x128, 96^3 cylinders,
uneven 2k x k x k designs) and odd ones between them.  Solves run to 1e-10 (the SIMP loop's default state
tolerance), the worse conditioned immersed ones to 1e-12: there the solution no longer depends on the order
of a sum.  The solution is what
a solve returns here; iteration counts and the last residual norm describe the way to it.
"""
import math

import numpy as np
import torch

import immersed_catmull_clark_b200 as icc
from immersed_catmull_clark_b200 import workloads as W

YOUNG, POISSON = 1.0, 0.3
MASKS = {"none": icc.MASK_NONE, "zero": icc.MASK_ZERO, "identity": icc.MASK_IDENTITY}
PRECISION = {"fp64": icc.FP64, "mixed": icc.MIXED}


# ---- the cases -----------------------------------------------------------------------------------


def listed():
    return [
        # the smallest grid of the benchmark: launch latency decides
        {"name": "apply64_24x16x12", "kind": "apply64", "nx": 24, "ny": 16, "nz": 12, "mask": "zero", "smooth": False},
        # odd sizes, the closure that keeps fixed rows as identity rows
        {"name": "apply64_97x53x41", "kind": "apply64", "nx": 97, "ny": 53, "nz": 41, "mask": "identity", "smooth": False},
        # the benchmark's main grid
        {"name": "apply64_128x64x64", "kind": "apply64", "nx": 128, "ny": 64, "nz": 64, "mask": "zero", "smooth": True},
        # odd and small, no mask
        {"name": "apply32_61x35x29", "kind": "apply32", "nx": 61, "ny": 35, "nz": 29, "mask": "none", "smooth": False},
        # the topology loop's grid: the largest of the benchmark
        {"name": "apply32_256x128x128", "kind": "apply32", "nx": 256, "ny": 128, "nz": 128, "mask": "zero", "smooth": True},
        # a small FP64 solve, as a design study runs thousands of
        {"name": "solve64_24x16x12", "kind": "solve", "nx": 24, "ny": 16, "nz": 12, "precision": "fp64", "smooth": False, "tol": 1e-10},
        # the main grid in plain FP64
        {"name": "solve64_128x64x64", "kind": "solve", "nx": 128, "ny": 64, "nz": 64, "precision": "fp64", "smooth": True, "tol": 1e-10},
        # mixed precision on a mid-size odd grid
        {"name": "mixed_53x31x27", "kind": "solve", "nx": 53, "ny": 31, "nz": 27, "precision": "mixed", "smooth": False, "tol": 1e-10},
        # the headline: the main grid in mixed precision
        {"name": "mixed_128x64x64", "kind": "solve", "nx": 128, "ny": 64, "nz": 64, "precision": "mixed", "smooth": True, "tol": 1e-10},
        # the immersed benchmark geometry: cut cells with small scales, inactive cells, many masked DOFs
        {"name": "immersed_96", "kind": "immersed", "n": 96, "precision": "mixed", "tol": 1e-12},
        # uneven designs in one call on host arrays
        {"name": "batched_12", "kind": "batched", "count": 12, "kmin": 8, "kmax": 27, "sizes": 2026, "precision": "mixed", "tol": 1e-10},
        # design iterations with four load cases: state solves, energies, filter, optimality criteria
        {"name": "topopt_48x24x24", "kind": "topopt", "nx": 48, "ny": 24, "nz": 24, "loads": 4, "iterations": 3, "precision": "mixed", "tol": 1e-10},
    ]


def _log_uniform(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def _box(rng, lo, hi):
    """Element counts of a box of about log-uniform volume in [lo, hi], longest along x."""
    vol = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ax, ay = rng.uniform(1.5, 2.2), rng.uniform(0.9, 1.4)
    k = (vol / (ax * ay)) ** (1.0 / 3.0)
    return {"nx": max(2, round(ax * k)), "ny": max(2, round(ay * k)), "nz": max(2, round(k))}


def draw(rng):
    kind = rng.choice(["apply64", "apply64", "apply32", "apply32", "solve", "solve", "immersed", "batched", "topopt"])
    if kind in ("apply64", "apply32"):
        return {"kind": kind, **_box(rng, 3e3, 6e5 if kind == "apply64" else 3e6),
                "mask": rng.choice(["none", "zero", "identity"]), "smooth": rng.random() < 0.5}
    if kind == "solve":
        return {"kind": kind, **_box(rng, 3e3, 2.5e5), "precision": rng.choice(["fp64", "mixed"]),
                "smooth": rng.random() < 0.5, "tol": 1e-10}
    if kind == "immersed":
        return {"kind": kind, "n": _log_uniform(rng, 20, 64), "precision": rng.choice(["fp64", "mixed"]), "tol": 1e-12}
    if kind == "batched":
        kmin = rng.randint(4, 12)
        return {"kind": kind, "count": rng.randint(2, 14), "kmin": kmin, "kmax": kmin + rng.randint(2, 14),
                "sizes": rng.randrange(1 << 20), "precision": "mixed", "tol": 1e-10}
    return {"kind": kind, **_box(rng, 2e3, 2.5e4), "loads": rng.randint(1, 4), "iterations": rng.randint(1, 3),
            "precision": rng.choice(["fp64", "mixed"]), "tol": 1e-10}


# ---- inputs ---------------------------------------------------------------------------------------


def _gen(seed, device="cuda"):
    g = torch.Generator(device=device)
    g.manual_seed(int(seed) * 7919 + 13)
    return g


def _cantilever(nel, smooth, seed):
    """SIMP scale s_e, free mask (x = 0 clamped) and the unit traction on x = 2 of the box [0,2]x[0,1]x[0,1];
    densities U[0.01, 1], smoothed by a clamped 3x3x3 mean or not (as a design between two filter steps)."""
    nx, ny, nz = nel
    rho = torch.rand((nz, ny, nx), generator=_gen(seed), device="cuda", dtype=torch.float64) * 0.99 + 0.01
    if smooth:
        p = torch.nn.functional.pad(rho[None, None], (1,) * 6, mode="replicate")
        rho = torch.nn.functional.avg_pool3d(p, 3, stride=1)[0, 0]
    scale = (W.EMIN + rho ** W.PENAL * (W.E0 - W.EMIN)).reshape(-1).cpu().numpy()
    cx, cy, cz = nx + 2, ny + 2, nz + 2
    free = np.ones((3, cz, cy, cx), dtype=np.uint8)
    free[:, :, :, 0] = 0
    force = np.zeros((3, cz, cy, cx))
    wy, wz = W.open_knot_integrals(ny, 1.0), W.open_knot_integrals(nz, 1.0)
    force[2, :, :, cx - 1] = -np.outer(wz, wy)
    # a seeded part of the load along the other directions, so every seed has its own right-hand side
    a = np.random.default_rng(seed).uniform(-0.5, 0.5, 2)
    force[0, :, :, cx - 1] = a[0] * np.outer(wz, wy)
    force[1, :, :, cx - 1] = a[1] * np.outer(wz, wy)
    return scale, free.reshape(-1), (force * free).reshape(-1)


BOX = np.array([[0.0, 2.0], [0.0, 1.0], [0.0, 1.0]])
CUBE = np.array([[0.0, 1.0]] * 3)


def _immersed(n, seed):
    """Cube minus three orthogonal cylinders of radius 0.25: scale E_min + rho^3 (E0 - E_min) alpha on active
    cells (alpha >= 1e-3), seeded densities in [0.3, 1], z = 0 clamped, control points without an active cell
    fixed, pressure on the top face's control points."""
    alpha, _ = icc.cylinder_weights((n, n, n), (8, 8, 8), 0.25)
    rho = torch.rand(n ** 3, generator=_gen(seed), device="cuda", dtype=torch.float64).cpu().numpy() * 0.7 + 0.3
    active = alpha >= 1e-3
    scale = np.where(active, W.EMIN + rho ** W.PENAL * (W.E0 - W.EMIN) * np.maximum(alpha, 1e-6), 0.0)
    act = active.reshape(n, n, n)
    touched = np.zeros((n + 2,) * 3, dtype=bool)
    for dz in range(3):
        for dy in range(3):
            for dx in range(3):
                touched[dz:dz + n, dy:dy + n, dx:dx + n] |= act
    touched[0] = False
    free = np.broadcast_to(touched, (3,) + touched.shape).astype(np.uint8)
    w = W.open_knot_integrals(n, 1.0)
    force = np.zeros((3,) + touched.shape)
    force[2, n + 1] = -np.outer(w, w)
    return scale, np.ascontiguousarray(free).reshape(-1), (force * free).reshape(-1)


def _field(nel, seed, dtype):
    """A displacement-like vector: a bending field with a rough part, as the directions of a PCG are."""
    cx, cy, cz = nel[0] + 2, nel[1] + 2, nel[2] + 2
    x = torch.linspace(0, 2, cx, device="cuda", dtype=torch.float64)[None, None, :]
    y = torch.linspace(0, 1, cy, device="cuda", dtype=torch.float64)[None, :, None]
    z = torch.linspace(0, 1, cz, device="cuda", dtype=torch.float64)[:, None, None]
    u = torch.stack([x * (2 - x) * (z - 0.5) + 0 * y, 0.3 * x * (y - 0.5) * (z - 0.5), -0.5 * x * x * (1 - x / 6) + 0 * y + 0 * z])
    r = torch.randn(u.shape, generator=_gen(seed + 1), device="cuda", dtype=torch.float64)
    return (u + 0.05 * r).reshape(-1).to(dtype).contiguous()


def _nel(case):
    return (int(case["nx"]), int(case["ny"]), int(case["nz"]))


def _batch_sizes(case):
    ks = np.random.default_rng(int(case["sizes"])).integers(case["kmin"], case["kmax"] + 1, size=int(case["count"]))
    return [(2 * int(k), int(k), int(k)) for k in ks]


def _loads(case, seed):
    """Load cases on the tip face: the consistent shear, axial and torsion loads with seeded factors."""
    nel = _nel(case)
    base = W.tip_load_cases(nel, (1.2, 0.6, 0.3))
    a = np.random.default_rng(seed).uniform(0.5, 1.5, (4, 4)) * (0.2 + 0.8 * np.eye(4))
    f = (a @ base).reshape(4, 3, nel[2] + 2, nel[1] + 2, nel[0] + 2)[: int(case["loads"])]
    f[..., 0] = 0.0
    return f.reshape(int(case["loads"]), -1)


def prepare(case, seed):
    kind = case["kind"]
    lam, mu = icc.lame(YOUNG, POISSON)
    if kind in ("apply64", "apply32"):
        nel, dt = _nel(case), torch.float64 if kind == "apply64" else torch.float32
        scale, free, _ = _cantilever(nel, case["smooth"], seed)
        sp = icc.SpaceBox(BOX, nel, 2)
        op = icc.MatrixFreeOperator(sp, (lam, mu), scale, None if case["mask"] == "none" else free, MASKS[case["mask"]])
        x = _field(nel, seed, dt)
        return {"kind": kind, "op": op, "x": x, "y": torch.empty_like(x)}
    if kind in ("solve", "immersed"):
        if kind == "solve":
            nel, bounds = _nel(case), BOX
            scale, free, force = _cantilever(nel, case["smooth"], seed)
        else:
            nel, bounds = (int(case["n"]),) * 3, CUBE
            scale, free, force = _immersed(int(case["n"]), seed)
        sp = icc.SpaceBox(bounds, nel, 2)
        op = icc.MatrixFreeOperator(sp, (lam, mu), scale, free, icc.MASK_ZERO)
        diag = 0
        if kind == "immersed":   # the immersed solve's preconditioner: the diagonal clamped at 1e-6
            diag = torch.from_numpy(np.maximum(op.diagonal(), 1e-6)).cuda()
        b = torch.from_numpy(force).cuda()
        solver = icc.PcgSolver(20 * sp.ndof, case["tol"], precision=PRECISION[case["precision"]])
        return {"kind": kind, "op": op, "solver": solver, "b": b, "diag": diag, "x": torch.empty_like(b)}
    if kind == "batched":
        ops, bs = [], []
        for i, nel in enumerate(_batch_sizes(case)):
            scale, free, force = _cantilever(nel, False, seed * 131 + i)
            ops.append(icc.MatrixFreeOperator(icc.SpaceBox(BOX, nel, 2), (lam, mu), scale, free, icc.MASK_ZERO))
            bs.append(force)
        return {"kind": kind, "ops": ops, "bs": bs, "tol": case["tol"], "precision": PRECISION[case["precision"]]}
    t = icc.CantileverTopOpt(_nel(case), pcg_tol=case["tol"], precision=PRECISION[case["precision"]])
    t.set_loads(_loads(case, seed))
    return {"kind": kind, "topopt": t, "iterations": int(case["iterations"])}


def run(state):
    kind = state["kind"]
    if kind == "apply64":
        state["op"].matvec_dev(state["x"].data_ptr(), state["y"].data_ptr())
        return state["y"]
    if kind == "apply32":
        state["op"].matvec_f32_dev(state["x"].data_ptr(), state["y"].data_ptr())
        return state["y"]
    if kind in ("solve", "immersed"):
        d = state["diag"]
        op = state["op"]
        state["solver"].solve_dev(op.n, state["b"].data_ptr(), d.data_ptr() if torch.is_tensor(d) else 0,
                                  state["x"].data_ptr(), op)
        return state["x"]
    if kind == "batched":
        xs, _, _, _ = icc.solve_batched(state["ops"], state["bs"], tol=state["tol"], precision=state["precision"])
        return xs
    h = state["topopt"].run(state["iterations"])
    return {"density": h.density, "compliance": h.compliance}


# ---- what a pass cannot do without ----------------------------------------------------------------

# Operations of one element in the sum-factorised form: three components through three directions and back
# (3 x 27 values, about 4 operations per value and direction), and the ~225 couplings of the material law.
FLOPS_PER_ELEMENT = 2 * 3 * 27 * 3 * 2 + 2 * 225


def _size(nel):
    n = 3 * (nel[0] + 2) * (nel[1] + 2) * (nel[2] + 2)
    return n, nel[0] * nel[1] * nel[2]


def _solve_work(nel, iterations):
    """b and s_e read, x written; `iterations` applies and their vector steps (six multiply-adds per DOF)."""
    n, ne = _size(nel)
    return 8.0 * (2 * n + ne), iterations * (FLOPS_PER_ELEMENT * ne + 12.0 * n)


def work(case):
    kind = case["kind"]
    if kind in ("apply64", "apply32"):
        n, ne = _size(_nel(case))
        sz = 8 if kind == "apply64" else 4
        return {"bytes": float(sz * (2 * n + ne) + (n if case["mask"] != "none" else 0)), "flops": float(FLOPS_PER_ELEMENT * ne)}
    if kind in ("solve", "immersed"):
        # iterations grow with the elements along the longest side (about 13 per element at 1e-10; 9 immersed)
        nel = _nel(case) if kind == "solve" else (int(case["n"]),) * 3
        b, f = _solve_work(nel, (13 if kind == "solve" else 9) * max(nel))
        return {"bytes": b, "flops": f}
    if kind == "batched":
        w = [_solve_work(nel, 13 * max(nel)) for nel in _batch_sizes(case)]
        return {"bytes": sum(a for a, _ in w), "flops": sum(b for _, b in w)}
    nel = _nel(case)
    b, f = _solve_work(nel, 15 * max(nel))
    k = case["loads"] * case["iterations"]
    return {"bytes": b * k, "flops": f * k}


# ---- 64-bit values in plain torch -----------------------------------------------------------------


class _Reference:
    """y = sum_e s_e K_e u_e by Gauss quadrature of the weak form, from the open-knot quadratic B-splines."""

    def __init__(self, bounds, nel, scale):
        self.nel = nel
        self.lam = YOUNG * POISSON / ((1 + POISSON) * (1 - 2 * POISSON))
        self.mu = YOUNG / (2 * (1 + POISSON))
        self.tabs = []
        gx, gw = np.polynomial.legendre.leggauss(3)
        for d in range(3):
            n, length = nel[d], bounds[d, 1] - bounds[d, 0]
            kn = np.concatenate([[0.0, 0.0], np.arange(n + 1) / n, [1.0, 1.0]])
            t = np.zeros((2, n, 3, 3))   # value / derivative, element, point, local function
            for e in range(n):
                for q in range(3):
                    x = (e + 0.5 * (gx[q] + 1.0)) / n
                    k = kn[e:e + 6]      # knots of the three functions of element e (its span is k[2], k[3])
                    l1, r1, l2, r2 = x - k[2], k[3] - x, x - k[1], k[4] - x
                    b0, b1 = r1 / (r1 + l1), l1 / (r1 + l1)
                    t[0, e, q] = [b0 * r1 / (r1 + l2), b0 * l2 / (r1 + l2) + b1 * r2 / (r2 + l1), b1 * l1 / (r2 + l1)]
                    t[1, e, q] = np.array([-2 * b0 / (r1 + l2), 2 * b0 / (r1 + l2) - 2 * b1 / (r2 + l1), 2 * b1 / (r2 + l1)]) / length
            self.tabs.append(torch.from_numpy(t).cuda())
        w = [0.5 * gw * (bounds[d, 1] - bounds[d, 0]) / nel[d] for d in range(3)]
        self.w = torch.from_numpy(w[2][:, None, None] * w[1][None, :, None] * w[0][None, None, :]).cuda()
        self.scale = torch.from_numpy(scale).cuda().reshape(nel[2], nel[1], nel[0])
        self.step = max(1, 60000 // (nel[0] * nel[1]))   # element layers at a time

    def _grad(self, p, kx, ky, kz, z0, z1):
        # p [z, y, x, az, ay, ax] -> values at the points [z, y, x, qz, qy, qx]
        X, Y, Z = self.tabs[0][kx], self.tabs[1][ky], self.tabs[2][kz][z0:z1]
        p = torch.einsum("zyxcba,xqa->zyxcbq", p, X)
        p = torch.einsum("zyxcbq,yrb->zyxcrq", p, Y)
        return torch.einsum("zyxcrq,zsc->zyxsrq", p, Z)

    def _gradt(self, s, kx, ky, kz, z0, z1):
        X, Y, Z = self.tabs[0][kx], self.tabs[1][ky], self.tabs[2][kz][z0:z1]
        s = torch.einsum("zyxsrq,zsc->zyxcrq", s, Z)
        s = torch.einsum("zyxcrq,yrb->zyxcbq", s, Y)
        return torch.einsum("zyxcbq,xqa->zyxcba", s, X)

    def apply(self, u):
        nx, ny, nz = self.nel
        u = u.reshape(3, nz + 2, ny + 2, nx + 2)
        y = torch.zeros_like(u)
        D = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
        for z0 in range(0, nz, self.step):
            z1 = min(nz, z0 + self.step)
            g = [[None] * 3 for _ in range(3)]
            for c in range(3):
                p = u[c, z0:z1 + 2].unfold(0, 3, 1).unfold(1, 3, 1).unfold(2, 3, 1)
                for d in range(3):
                    g[c][d] = self._grad(p, *D[d], z0, z1)
            ws = self.scale[z0:z1, :, :, None, None, None] * self.w
            tr = self.lam * (g[0][0] + g[1][1] + g[2][2])
            for c in range(3):
                f = 0
                for d in range(3):
                    s = self.mu * (g[c][d] + g[d][c])
                    if c == d:
                        s = s + tr
                    f = f + self._gradt(ws * s, *D[d], z0, z1)
                for az in range(3):
                    for ay in range(3):
                        for ax in range(3):
                            y[c, z0 + az:z1 + az, ay:ay + ny, ax:ax + nx] += f[..., az, ay, ax]
        return y.reshape(-1)

    def diagonal(self):
        nx, ny, nz = self.nel
        d = torch.zeros((3, nz + 2, ny + 2, nx + 2), dtype=torch.float64, device="cuda")
        D = [(1, 0, 0), (0, 1, 0), (0, 0, 1)]
        sq = [t * t for t in self.tabs]
        for c in range(3):
            e = 0
            for k in range(3):
                X, Y, Z = sq[0][D[k][0]], sq[1][D[k][1]], sq[2][D[k][2]]
                m = torch.einsum("zsc,yrb,xqa,srq->zyxcba", Z, Y, X, self.w)
                e = e + (self.lam + 2 * self.mu if k == c else self.mu) * m
            e = e * self.scale[..., None, None, None]
            for az in range(3):
                for ay in range(3):
                    for ax in range(3):
                        d[c, az:az + nz, ay:ay + ny, ax:ax + nx] += e[..., az, ay, ax]
        return d.reshape(-1)


def _exact_solve(bounds, nel, scale, free, force, clamp, tol=1e-14):
    """Jacobi-PCG in 64 bits, restarted from the true residual until that no longer falls."""
    A = _Reference(bounds, nel, scale)
    m = torch.from_numpy(free.astype(np.float64)).cuda()
    b = torch.from_numpy(force).cuda()
    d = torch.clamp(A.diagonal(), min=clamp)
    inv = torch.where(m > 0, 1 / d, torch.zeros_like(d))
    x = torch.zeros_like(b)
    nb = float(b.norm())
    for _ in range(2):
        r = b - m * A.apply(m * x)
        z = inv * r
        p, rz = z.clone(), r @ z
        for i in range(40 * max(nel) + 200):
            ap = m * A.apply(p)
            a = rz / (p @ ap)
            x += a * p
            r -= a * ap
            if i % 16 == 0 and float(r.norm()) < tol * nb:
                break
            z = inv * r
            rz, old = r @ z, rz
            p = z + (rz / old) * p
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("apply64", "apply32"):
        nel = _nel(case)
        scale, free, _ = _cantilever(nel, case["smooth"], seed)
        x = _field(nel, seed, torch.float64 if kind == "apply64" else torch.float32).double()
        A = _Reference(BOX, nel, scale)
        m = torch.from_numpy(free.astype(np.float64)).cuda()
        if case["mask"] == "none":
            return A.apply(x)
        y = m * A.apply(m * x)
        return y if case["mask"] == "zero" else y + (1 - m) * x
    if kind == "solve":
        nel = _nel(case)
        if nel[0] * nel[1] * nel[2] * max(nel) > 4e6:
            return None   # too many iterations of this plain form
        return _exact_solve(BOX, nel, *_cantilever(nel, case["smooth"], seed), 0.0)
    if kind == "immersed":
        n = int(case["n"])
        if n > 36:
            return None
        return _exact_solve(CUBE, (n, n, n), *_immersed(n, seed), 1e-6)
    return None
