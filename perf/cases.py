"""Timed workloads of the solve path, each through a public entry point of the package.

A case is a dict of plain values; `listed()` names twelve of them and `draw(rng)` gives more
of the same ranges.  `prepare` makes the inputs from a seed, `run` is one pass, `work` the
bytes and operations a pass cannot do without, and `exact` the same outputs computed in
float64 with plain torch (projected Newton, conjugate gradients, dense eigenvectors).
"""
import math

import numpy as np
import torch

import symx_gb300 as sg
from symx_gb300 import problems

SPACING = 0.01  # m, as every configuration of symx_gb300.problems
YOUNGS, POISSON, DENSITY, DT, K_BC = 1e5, 0.3, 1000.0, 1.0 / 60.0, 1e8
NODES = {"tet4": 4, "tet10": 10, "hex8": 8}
NEWTON = {"cg_rel_tolerance": 1e-3}  # the benchmark's forcing


def _case(name, op, cells=(0, 0, 0), **kw):
    nx, ny, nz = cells
    return {"name": name, "op": op, "nx": nx, "ny": ny, "nz": nz, **kw}


def listed():
    return [
        # the smallest simulation step: a 1,331-vertex box in double precision, where launches
        # and round trips count
        _case("newton_tet4_10_fp64", "newton", (10, 10, 10), kind="tet4", precision="fp64"),
        # an ordinary mixed-precision step on a box with unequal sides
        _case("newton_tet4_27x21x33_mixed", "newton", (27, 21, 33), kind="tet4", precision="mixed"),
        # the benchmark's step: 274,625 vertices, 1,572,864 tetrahedra
        _case("newton_tet4_64_mixed", "newton", (64, 64, 64), kind="tet4", precision="mixed"),
        # a slab of hexahedra with a log-normal stiffness field
        _case("newton_hex8_41x37x11_mixed", "newton", (41, 37, 11), kind="hex8", precision="mixed"),
        # quadratic tetrahedra: 30 x 30 element Hessians
        _case("newton_tet10_11x10x9_mixed", "newton", (11, 10, 9), kind="tet10", precision="mixed"),
        # backward: the adjoint of a step and the material and state gradients
        _case("adjoint_tet4_19x23x17_fp64", "adjoint", (19, 23, 17), kind="tet4", precision="fp64"),
        # energy and gradient at a host state (an outer optimiser's call)
        _case("gradient_tet4_32", "gradient", (32, 32, 32), kind="tet4", precision="fp64"),
        # projection alone: a Tet4 mesh's element Hessians in float, Hex8 ones in double
        {"name": "project_12_f32", "op": "project", "n": 12, "count": 200003, "dtype": "float32"},
        {"name": "project_24_f64", "op": "project", "n": 24, "count": 2001, "dtype": "float64"},
        # one product with the benchmark's matrix
        _case("spmv_64_f32", "spmv", (64, 64, 64), dtype="float32"),
        # linear solves with a caller's matrix: an ordinary one and a small one in double
        _case("pcg_40_f32", "pcg", (40, 40, 40), dtype="float32", rel_tol=1e-6),
        _case("pcg_9_f64", "pcg", (9, 9, 9), dtype="float64", rel_tol=1e-10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["newton", "newton", "newton", "adjoint", "gradient", "project", "spmv", "pcg"])
    if op == "project":
        n, dtype = rng.choice([12, 24, 30]), rng.choice(["float32", "float64"])
        most = {(12, "float32"): 400000, (24, "float32"): 30000, (30, "float32"): 20000,
                (12, "float64"): 60000, (24, "float64"): 3000, (30, "float64"): 2000}[n, dtype]
        return {"op": op, "n": n, "count": _log_int(rng, 100, most), "dtype": dtype}
    if op in ("spmv", "pcg"):
        dtype = rng.choice(["float32", "float64"])
        most = 64 if op == "spmv" else 48 if dtype == "float32" else 32
        c = {"op": op, **{k: _log_int(rng, 4, most) for k in ("nx", "ny", "nz")}, "dtype": dtype}
        if op == "pcg":
            c["rel_tol"] = 1e-6 if dtype == "float32" else 1e-10
        return c
    kind, precision = rng.choice(["tet4", "tet4", "hex8", "tet10"]), rng.choice(["fp64", "mixed"])
    if op == "adjoint":
        kind, precision, most = "tet4", "fp64", 24
    elif op == "gradient":
        precision, most = "fp64", {"tet4": 40, "hex8": 28, "tet10": 14}[kind]
    else:
        most = {("tet4", "mixed"): 44, ("hex8", "mixed"): 28, ("tet10", "mixed"): 11,
                ("tet4", "fp64"): 18, ("hex8", "fp64"): 11, ("tet10", "fp64"): 5}[kind, precision]
    return {"op": op, **{k: _log_int(rng, 3, most) for k in ("nx", "ny", "nz")}, "kind": kind, "precision": precision}


# ---------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _problem(case, seed):
    """The package's seeded implicit-Euler step of a clamped box (symx_gb300.problems)."""
    cfg = {"kind": case["kind"], "cells": (case["nx"], case["ny"], case["nz"]), "h": SPACING, "perturb": 0.05,
           "seed": int(seed) % 1000003}
    if case["kind"] == "hex8":
        cfg.update(perturb=0.0, youngs_lognormal_sigma=0.5)
    p = problems.step_problem(cfg, youngs=YOUNGS, poisson=POISSON, density=DENSITY, dt=DT, k_bc=K_BC)
    if case["op"] == "adjoint":
        # a state near equilibrium: the rest shape with a small jitter (its Hessian is positive
        # definite), and a loss gradient
        k = cfg["seed"] * 1000
        p["x_init"] = p["X"] + 1e-4 * SPACING * problems.normal(k + 11, p["X"].size).reshape(-1, 3)
        p["dLdx"] = problems.normal(k + 12, p["X"].size)
    return p


def _element_hessians(case, seed):
    """`count` unprojected Neo-Hookean element Hessians (row-major, n x n, float64) of deformed
    Tet4 (12), Hex8 (24) or Tet10 (30) elements of the step problem's spacing and jitter."""
    g, dev, n, count = _generator(seed), _device(), case["n"], case["count"]
    kind = {12: "tet4", 24: "hex8", 30: "tet10"}[n]
    if kind == "hex8":
        X, conn = problems.cuboid_hex8(1, 1, 1, (SPACING,) * 3)
    else:
        X, conn = (problems.cuboid_tet4 if kind == "tet4" else problems.cuboid_tet10)(1, 1, 1, (SPACING,) * 3)
    X = torch.as_tensor(X[conn], device=dev)
    Xe = X[torch.randint(X.shape[0], (count,), generator=g, device=dev)]
    xe = Xe + 0.1 * SPACING * (2 * torch.rand(Xe.shape, generator=g, device=dev, dtype=torch.float64) - 1)
    E = YOUNGS * torch.exp(0.5 * torch.randn(count, generator=g, device=dev, dtype=torch.float64))
    mu, lam = problems.lame(1.0, POISSON)
    return torch.cat([_NeoHookean(kind, Xe[i:i + 50000], float(mu) * E[i:i + 50000], float(lam) * E[i:i + 50000])
                      .hessian(xe[i:i + 50000]) for i in range(0, count, 50000)])


def _matrix(case, seed):
    """BCSR matrix of an implicit step at the rest shape of a Tet4 box with a log-normal
    stiffness field (element Hessians + mass / dt^2 + the clamped face's penalty), float64:
    row_ptr, cols and (nnzb, 3, 3) values, assembled by adding grid slices."""
    dev, f64 = _device(), torch.float64
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    X, conn = problems.cuboid_tet4(1, 1, 1, (SPACING,) * 3)
    mu, lam = problems.lame(YOUNGS, POISSON)
    Xe = torch.as_tensor(X[conn], device=dev)
    Ht = _NeoHookean("tet4", Xe, torch.full((6,), float(mu), device=dev, dtype=f64),
                     torch.full((6,), float(lam), device=dev, dtype=f64)).hessian(Xe).reshape(6, 4, 3, 4, 3)
    E = torch.exp(0.3 * torch.randn((6, nx, ny, nz), generator=_generator(seed), device=dev, dtype=f64))
    corner = [(v // 4, v // 2 % 2, v % 2) for v in range(8)]  # vertex index of the 1-cell box
    pairs = {}
    for t in range(6):
        for a in range(4):
            for b in range(4):
                ca, cb = corner[conn[t, a]], corner[conn[t, b]]
                pairs.setdefault(tuple(q - p for p, q in zip(ca, cb)), []).append((t, a, b, ca))
    offsets = sorted(pairs)  # ascending columns: the vertex index is lexicographic in (i, j, k)
    shape = (nx + 1, ny + 1, nz + 1)
    index = torch.arange(math.prod(shape), device=dev).reshape(shape)
    vals, used = torch.zeros((*shape, len(offsets), 3, 3), device=dev, dtype=f64), []
    for o, off in enumerate(offsets):
        for t, a, b, (i, j, k) in pairs[off]:
            vals[i:i + nx, j:j + ny, k:k + nz, o] += E[t, ..., None, None] * Ht[t, a, :, b, :]
        ok = torch.ones(shape, dtype=torch.bool, device=dev)
        for axis, d in enumerate(off):
            at = torch.arange(shape[axis], device=dev) + d
            ok &= ((at >= 0) & (at < shape[axis])).reshape([-1 if x == axis else 1 for x in range(3)])
        used.append(ok)
        if off == (0, 0, 0):
            eye = torch.eye(3, device=dev, dtype=f64)
            vals[:, :, :, o] += DENSITY * SPACING ** 3 / DT ** 2 * eye
            vals[0, :, :, o] += K_BC * eye
    used = torch.stack(used, -1)
    step = torch.tensor([(i * shape[1] + j) * shape[2] + k for i, j, k in offsets], device=dev)
    cols = (index[..., None] + step)[used].to(torch.int32)
    row_ptr = torch.zeros(index.numel() + 1, dtype=torch.int64, device=dev)
    row_ptr[1:] = used.reshape(-1, len(offsets)).sum(1).cumsum(0)
    return row_ptr.to(torch.int32), cols, vals[used]


def _vector(case, n_rows, seed):
    return torch.randn(3 * n_rows, generator=_generator(int(seed) + 1), device=_device(), dtype=getattr(torch, case["dtype"]))


def prepare(case, seed):
    if case["op"] in ("newton", "adjoint", "gradient"):
        p = _problem(case, seed)
        s = sg.ElasticSolver(p)
        s.set_settings(precision=case["precision"], **NEWTON)
        if case["op"] == "adjoint":
            s.set_state(p["x_init"], p["x0"], p["v0"])
            s.upload()
        return {"op": case["op"], "solver": s, "p": p}
    if case["op"] == "project":
        return {"op": "project", "H": _element_hessians(case, seed).to(getattr(torch, case["dtype"]))}
    row_ptr, cols, vals = _matrix(case, seed)
    n = row_ptr.numel() - 1
    v = _vector(case, n, seed)
    return {"op": case["op"], "row_ptr": row_ptr, "cols": cols, "v": v, "out": torch.empty_like(v),
            "vals": sg.component_major(vals.to(v.dtype)), "rel_tol": case.get("rel_tol")}


def run(state):
    op = state["op"]
    if op == "newton":  # one step: new host state in, converged positions out
        s, p = state["solver"], state["p"]
        s.set_state(p["x_init"], p["x0"], p["v0"])
        s.solve()
        return s.get_positions()
    if op == "adjoint":
        out = state["solver"].adjoint(state["p"]["dLdx"], rel_tol=1e-12)
        return {k: out[k] for k in ("lambda", "dLdmu", "dLdlam", "dLdx0", "dLdv0")}
    if op == "gradient":
        s, p = state["solver"], state["p"]
        s.set_state(p["x_init"], p["x0"], p["v0"])
        return s.evaluate()
    if op == "project":  # in place, on a copy: the caller keeps its matrices
        H = state["H"].clone()
        sg.project_pd(H)
        return H
    A = state["row_ptr"], state["cols"], state["vals"]
    if op == "spmv":
        sg.bcsr_spmv(*A, state["v"], state["out"])
    else:
        sg.bcsr_pcg(*A, state["v"], state["out"], rel_tol=state["rel_tol"], max_iterations=5000)
    return state["out"]


def work(case):
    """Inputs and outputs once each, and the operations of the algorithm the entry point is
    defined by.  Newton: five iterations and 1.6 PCG iterations per cell of the mean side each,
    as the benchmark's step takes."""
    if case["op"] == "project":
        n, b = case["n"], 4 if case["dtype"] == "float32" else 8
        return {"bytes": 2.0 * b * case["count"] * n * n, "flops": 9.0 * case["count"] * n ** 3}
    cells = case["nx"] * case["ny"] * case["nz"]
    side = cells ** (1.0 / 3.0)
    rows = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
    if case["op"] in ("spmv", "pcg"):
        b = 4 if case["dtype"] == "float32" else 8
        once = 15.0 * rows * (9 * b + 4) + rows * (4 + 6 * b)
        return {"bytes": once, "flops": 270.0 * rows * (1 if case["op"] == "spmv" else 3.0 * side)}
    kind = case["kind"]
    m = 3 * NODES[kind]
    elements = cells * (1 if kind == "hex8" else 6)
    points = {"tet4": 1, "tet10": 4, "hex8": 8}[kind]
    vertices = 8 * rows if kind == "tet10" else rows
    blocks = vertices * {"tet4": 15, "tet10": 28, "hex8": 27}[kind]
    io = 8.0 * (12 * vertices + 2 * vertices + 2 * elements) + 4.0 * elements * NODES[kind]
    gradient = 20.0 * elements * points * m
    hessian = 10.0 * elements * points * m * m
    if case["op"] == "gradient":
        return {"bytes": io, "flops": gradient}
    if case["op"] == "adjoint":
        return {"bytes": io, "flops": gradient + hessian + 5.0 * side * 18 * blocks}
    return {"bytes": io, "flops": 5.0 * (gradient + hessian + 9.0 * elements * m ** 3 + 1.6 * side * 18 * blocks)}


# ---------------------------------------------------------------- exact values
class _NeoHookean:
    """Element energies, gradients and Hessians of the classic Neo-Hookean density in float64."""

    def __init__(self, kind, Xe, mu, lam):
        f = dict(device=Xe.device, dtype=torch.float64)
        if kind == "hex8":
            g = 1.0 / math.sqrt(3.0)
            signs = [(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)]
            dN, w = [], [1.0] * 8
            for q in signs:
                half = [[0.5 * (1 + s * g * t) for s, t in zip(a, q)] for a in signs]
                dN.append([[0.5 * a[0] * h[1] * h[2], 0.5 * a[1] * h[0] * h[2], 0.5 * a[2] * h[0] * h[1]]
                           for a, h in zip(signs, half)])
        elif kind == "tet4":
            dN, w = [[[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]], [1.0 / 6.0]
        else:
            a, b = 0.58541020, 0.13819660
            grad = [[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]
            edges = [(0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3)]
            dN, w = [], [0.041666667] * 4
            for xi in ((a, b, b), (b, a, b), (b, b, a), (b, b, b)):
                L = (1 - sum(xi), *xi)
                dN.append([[(4 * L[i] - 1) * d for d in grad[i]] for i in range(4)] +
                          [[4 * (L[i] * e + L[j] * d) for d, e in zip(grad[i], grad[j])] for i, j in edges])
        dN = torch.tensor(dN, **f)
        J = torch.einsum("eai,qaj->eqij", Xe, dN)
        self.B = torch.einsum("qaj,eqji->eqai", dN, torch.linalg.inv(J))  # shape gradients at rest
        self.w = torch.linalg.det(J) * torch.tensor(w, **f)
        self.mu, self.lam = mu[:, None], lam[:, None]

    def _at(self, xe):
        F = torch.einsum("eai,eqaj->eqij", xe, self.B)
        return F, torch.linalg.inv(F).transpose(-1, -2), torch.log(torch.linalg.det(F))

    def energy(self, xe):
        F, _, lj = self._at(xe)
        psi = 0.5 * self.mu * (F.square().sum((-1, -2)) - 3) - self.mu * lj + 0.5 * self.lam * lj.square()
        return (psi * self.w).sum(1)

    def stress(self, xe):
        F, G, lj = self._at(xe)
        return self.mu[..., None, None] * F + (self.lam * lj - self.mu)[..., None, None] * G

    def gradient(self, xe):
        return torch.einsum("eqij,eqaj,eq->eai", self.stress(xe), self.B, self.w)

    def hessian(self, xe):
        _, G, lj = self._at(xe)
        BG = torch.einsum("eqaj,eqij->eqai", self.B, G)
        n = xe.shape[1]
        H = torch.einsum("eq,eqai,eqbk->eaibk", self.lam * self.w, BG, BG)
        H += torch.einsum("eq,eqak,eqbi->eaibk", (self.mu - self.lam * lj) * self.w, BG, BG)
        H += torch.einsum("eq,eqaj,eqbj,ik->eaibk", self.mu * self.w, self.B, self.B,
                          torch.eye(3, device=xe.device, dtype=xe.dtype))
        return H.reshape(-1, 3 * n, 3 * n)

    def material_gradient(self, xe, le):
        """lambda . dg/dmu and lambda . dg/dlam per element."""
        F, G, lj = self._at(xe)
        dF = torch.einsum("eai,eqaj->eqij", le, self.B)
        return ((((F - G) * dF).sum((-1, -2)) * self.w).sum(1), ((lj[..., None, None] * G * dF).sum((-1, -2)) * self.w).sum(1))


def _project(H, eps=1e-10):
    out = torch.empty(H.shape, device=H.device, dtype=torch.float64)
    for i in range(0, H.shape[0], 20000):
        w, V = torch.linalg.eigh(H[i:i + 20000].double())
        out[i:i + 20000] = (V * w.clamp(min=eps)[:, None]) @ V.transpose(-1, -2)
    return out


def _cg(product, D, b, tol, most):
    """Conjugate gradients with the inverse diagonal blocks D, (n, 3) vectors."""
    x, r = torch.zeros_like(b), b.clone()
    stop = tol * b.norm()
    z = torch.einsum("nij,nj->ni", D, r)
    p, rz = z.clone(), (r * z).sum()
    for _ in range(most):
        q = product(p)
        alpha = rz / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        if r.norm() <= stop:
            break
        z = torch.einsum("nij,nj->ni", D, r)
        old, rz = rz, (r * z).sum()
        p = z + rz / old * p
    return x


class _Step:
    """One implicit-Euler step in float64: element Hessians, matrix-free products."""

    def __init__(self, p, kind):
        t = lambda v: torch.as_tensor(np.asarray(v), device=_device())  # noqa: E731
        self.conn, self.mass, self.bc = t(p["conn"]).long(), t(p["mass"])[:, None], t(p["bc_idx"]).long()
        self.target, self.mu, self.lam = t(p["bc_target"]), t(p["mu"]), t(p["lam"])
        self.y = t(p["x0"]) + p["dt"] * t(p["v0"]) + p["dt"] ** 2 * t(p["gravity"])
        self.nh = _NeoHookean(kind, t(p["X"])[self.conn], self.mu, self.lam)
        self.x = t(p["x_init"])

    def energy(self, x):
        return float(self.nh.energy(x[self.conn]).sum() + (0.5 * self.mass * (x - self.y).square()).sum() / DT ** 2 +
                     0.5 * K_BC * (x[self.bc] - self.target).square().sum())

    def gradient(self, x):
        g = self.mass * (x - self.y) / DT ** 2
        g[self.bc] += K_BC * (x[self.bc] - self.target)
        return g.index_add(0, self.conn.reshape(-1), self.nh.gradient(x[self.conn]).reshape(-1, 3))

    def solve(self, H, b, tol, most=3000):
        diag = (self.mass / DT ** 2)[:, :, None] * torch.eye(3, device=b.device, dtype=b.dtype)
        diag[self.bc] += K_BC * torch.eye(3, device=b.device, dtype=b.dtype)
        own = diag.clone()
        for a in range(self.conn.shape[1]):
            own.index_add_(0, self.conn[:, a], H[:, 3 * a:3 * a + 3, 3 * a:3 * a + 3])
        flat = self.conn.reshape(-1)

        def product(v):
            Hv = torch.einsum("eij,ej->ei", H, v[self.conn].reshape(H.shape[0], -1))
            return torch.einsum("nij,nj->ni", diag, v).index_add(0, flat, Hv.reshape(-1, 3))

        return _cg(product, torch.linalg.inv(own), b, tol, most)

    def newton(self):
        x, g = self.x, self.gradient(self.x)
        for _ in range(30):
            if float(g.abs().max()) < 1e-9:
                break
            dx = self.solve(_project(self.nh.hessian(x[self.conn])), -g, 1e-6)
            E, slope, step = self.energy(x), float((g * dx).sum()), 1.0
            while step > 1e-6 and float(g.abs().max()) > 1e-4 and not self.energy(x + step * dx) < E + 1e-4 * step * slope:
                step *= 0.5
            x = x + step * dx
            g = self.gradient(x)
        return x


def exact(case, seed):
    op = case["op"]
    if op == "project":
        H = _element_hessians(case, seed).to(getattr(torch, case["dtype"]))
        return _project(H)
    if op in ("newton", "adjoint", "gradient"):
        if op != "gradient" and case["nx"] * case["ny"] * case["nz"] * NODES[case["kind"]] ** 2 > 150000:
            return None  # more than a few seconds of dense element algebra in float64
        p = _problem(case, seed)
        s = _Step(p, case["kind"])
        if op == "gradient":
            return (s.energy(s.x), s.gradient(s.x).reshape(-1).cpu().numpy())
        if op == "newton":
            return s.newton().cpu().numpy()
        b = torch.as_tensor(p["dLdx"], device=_device()).reshape(-1, 3)
        lam = s.solve(s.nh.hessian(s.x[s.conn]), b, 1e-14)
        dmu, dlam = s.nh.material_gradient(s.x[s.conn], lam[s.conn])
        out = {"lambda": lam, "dLdmu": -dmu, "dLdlam": -dlam, "dLdx0": s.mass * lam / DT ** 2, "dLdv0": s.mass * lam / DT}
        return {k: v.reshape(-1).cpu().numpy() for k, v in out.items()}
    row_ptr, cols, vals = _matrix(case, seed)
    n = row_ptr.numel() - 1
    v = _vector(case, n, seed).double().reshape(n, 3)
    vals = vals.to(getattr(torch, case["dtype"])).double()  # the matrix as the caller holds it
    rows = torch.repeat_interleave(torch.arange(n, device=cols.device), (row_ptr[1:] - row_ptr[:-1]).long())
    cols = cols.long()

    def product(x):
        return torch.zeros_like(x).index_add_(0, rows, torch.einsum("kij,kj->ki", vals, x[cols]))

    if op == "spmv":
        return product(v).reshape(-1)
    return _cg(product, torch.linalg.inv(vals[rows == cols]), v, 1e-14, 3000).reshape(-1)
