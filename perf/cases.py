"""Performance cases: the calls that a user of this package makes, over the sizes it is used at.

Every case is one pass through public entry points (``LinearGmres``, ``SteadyHeatGpu``,
``TransientTransportGpu``, ``SteadyFlowGpu``, ``Mesh``). A case's mesh depends on its sizes alone;
the seed makes the fields on it. As in a user's program the mesh and the operator handle on it are
built once and kept, and every pass brings new fields, so a pass pays for assembly, factorisation
and solve. ``exact`` restates the discretisation and the solves in float64 with torch, from the
mesh's dual.
"""
from __future__ import annotations

import math
from collections import OrderedDict

import numpy as np
import torch

import vfvchem_vfvm3d_b200 as vfv
from vfvchem_vfvm3d_b200 import _lib as L
from vfvchem_vfvm3d_b200.flow import flow_options
from vfvchem_vfvm3d_b200.problems import HEAT_BND_KIND, lid_cavity


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # the drop-in for the reference's linear solver on its smallest example (8,000 vertices, Jacobi,
        # FP64): host triplets in, host solution out; launches and latency
        {"name": "linear_8k", "kind": "linear", "n": 20, "precond": "jacobi"},
        # the same drop-in with the ILU(0) preconditioner at an odd, ordinary size (50,653 vertices)
        {"name": "linear_51k_ilu", "kind": "linear", "n": 37, "precond": "ilu0"},
        # a nonlinear iteration's matrix and right-hand side, and A T: assembly and FP64 SpMV at 10^6 vertices
        {"name": "heat_residual_1m", "kind": "residual", "n": 100},
        # the heterogeneous heat problem solved from host fields, mixed precision, swept ILU(0), ordinary size
        {"name": "heat_mixed_104k", "kind": "heat", "n": 47, "precision": "mixed", "device": False},
        # the same at 10^6 vertices, fields resident on the device: the package's headline configuration
        {"name": "heat_mixed_1m", "kind": "heat", "n": 100, "precision": "mixed", "device": True},
        # the plain FP64 solver with the exact multicolour ILU(0), 262,144 vertices
        {"name": "heat_fp64_262k", "kind": "heat", "n": 64, "precision": "fp64", "device": True},
        # one evaluation of a parameter gradient: forward solve and adjoint solve, FP64 (125,000 vertices)
        {"name": "heat_gradient_125k", "kind": "gradient", "n": 50},
        # implicit time steps of a few small independent meshes: latency
        {"name": "transport_3", "kind": "transport", "meshes": 3, "steps": 10, "order": "multicolor", "sweeps": 0},
        # the same for a batch of 64 uneven meshes, natural-order ILU(0) with 3 sweeps
        {"name": "transport_64", "kind": "transport", "meshes": 64, "steps": 20, "order": "natural", "sweeps": 3},
        # checkpointed adjoint of a batch's diffusivity
        {"name": "transport_adjoint_16", "kind": "transport_adjoint", "meshes": 16, "steps": 8, "every": 4},
        # the coupled Navier-Stokes system assembled at a state and applied to it (442,368 unknowns)
        {"name": "flow_residual_48", "kind": "flow_residual", "n": 48},
        # two Picard iterations of the lid-driven cavity, FP64 GMRES(100) + 4x4 block-Jacobi (131,072 unknowns)
        {"name": "flow_picard_32", "kind": "flow_picard", "n": 32},
    ]


def draw(rng):
    def grid(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["linear", "residual", "heat", "heat", "gradient", "transport", "transport", "transport_adjoint", "flow_residual",
                       "flow_picard"])
    if kind == "linear":
        return {"kind": kind, "n": grid(10, 40), "precond": rng.choice(["jacobi", "ilu0"])}
    if kind == "residual":
        return {"kind": kind, "n": grid(12, 100)}
    if kind == "heat":
        return {"kind": kind, "n": grid(16, 90), "precision": rng.choice(["mixed", "fp64"]), "device": rng.random() < 0.5}
    if kind == "gradient":
        return {"kind": kind, "n": grid(12, 56)}
    if kind == "transport":
        order, sweeps = rng.choice([("natural", 3), ("natural", 2), ("multicolor", 0)])
        return {"kind": kind, "meshes": grid(1, 64), "steps": rng.randint(4, 20), "order": order, "sweeps": sweeps}
    if kind == "transport_adjoint":
        return {"kind": kind, "meshes": grid(1, 16), "steps": rng.randint(4, 8), "every": rng.randint(2, 4)}
    if kind == "flow_residual":
        return {"kind": kind, "n": grid(8, 48)}
    return {"kind": kind, "n": grid(8, 32)}


# ---------------------------------------------------------------- meshes and handles, kept as a program keeps them
_KEPT: OrderedDict = OrderedDict()
_KEEP = 8


def _keep(key, make):
    if key not in _KEPT:
        while len(_KEPT) >= _KEEP:
            _KEPT.popitem(last=False)
        _KEPT[key] = make()
    _KEPT.move_to_end(key)
    return _KEPT[key]


class _CubeMesh:
    """A jittered cube with the arrays that callers read from it."""

    def __init__(self, n):
        self.mesh = vfv.Mesh.jitter_cube(n, 42, 0.25)
        self.n = self.mesh.n_tot
        self.pos, nb, _ = self.mesh.export()
        self.node_bnd = np.full(self.n, -1, np.int32)
        self.node_bnd[self.mesh.n_pts:] = nb


def _cube(n):
    return _keep(("cube", n), lambda: _CubeMesh(n))


def _heat(n):
    return _keep(("heat", n), lambda: vfv.SteadyHeatGpu(_cube(n).mesh, HEAT_BND_KIND))


def _batch_sizes(case):
    rng = np.random.default_rng(4 + case["meshes"])
    nmax = 5000 if case["meshes"] < 8 else 50000
    return np.rint(np.cbrt(np.exp(rng.uniform(np.log(2000), np.log(nmax), case["meshes"])))).astype(np.int32)


def _batch(case):
    def make():
        sizes = _batch_sizes(case)
        meshes = vfv.Mesh.jitter_cubes_device_dual(vfv.default_context(), sizes, 1000 + np.arange(sizes.size, dtype=np.uint64))
        tr = vfv.TransientTransportGpu(meshes, 1e-2)
        return tr, np.concatenate([m.export()[0] for m in meshes])
    return _keep(("batch", case["meshes"]), make)


def _flow(n):
    def make():
        prob = lid_cavity(n)
        return prob, vfv.SteadyFlowGpu(prob), prob.mesh.export()[0]
    return _keep(("flow", n), make)


# ---------------------------------------------------------------- inputs
def _heat_fields(n, seed, prod=0.0):
    """Heterogeneous conductivity and source, Dirichlet T = 0 / 1 on x = 0 / 1, zero flux elsewhere."""
    c = _cube(n)
    rng = np.random.default_rng(seed)
    k = np.exp(rng.standard_normal(c.n))
    q = rng.uniform(0.0, 1.0, c.n)
    s = np.full(c.n, float(prod))
    bc = np.where(c.node_bnd == 1, 1.0, 0.0)
    T0 = bc.copy()
    return k, q, s, T0, bc


def _state_T(n, seed):
    """A temperature state in the middle of a nonlinear iteration."""
    c = _cube(n)
    rng = np.random.default_rng(seed + 1_000_000)
    T = c.pos[:, 0] + 0.1 * rng.standard_normal(c.n)
    T[c.node_bnd == 0], T[c.node_bnd == 1] = 0.0, 1.0
    return T


def _transport_fields(case, seed, pos):
    rng = np.random.default_rng(seed)
    x, y, z = pos.T
    a = rng.uniform(0.5, 1.0, 3)
    ph = rng.uniform(0, 2 * np.pi, 3)
    vel = np.stack([a[0] * np.sin(np.pi * y), a[1] * np.sin(np.pi * z), a[2] * np.sin(np.pi * x)])
    c0 = 1.0 + 0.5 * np.sin(np.pi * x + ph[0]) * np.sin(np.pi * y + ph[1]) * np.sin(np.pi * z + ph[2])
    return vel, c0, 1e-3 * rng.uniform(0.5, 1.5)


def _flow_state(prob, pos, seed):
    """A velocity and pressure state of the cavity: a swirl with noise, the lid's velocity on the boundary."""
    rng = np.random.default_rng(seed)
    x, y, z = pos.T
    u = np.stack([np.sin(np.pi * x) * np.cos(np.pi * z), 0.3 * np.sin(np.pi * y), -0.5 * np.cos(np.pi * x) * z])
    u = rng.uniform(0.5, 1.0) * u + 0.05 * rng.standard_normal(u.shape)
    nodes = prob.node_bnd >= 0
    u[:, nodes] = prob.bc_vel[:, nodes]
    p = 0.2 * np.cos(np.pi * x) * np.sin(np.pi * y) + 0.1 * z
    return np.concatenate([u.reshape(-1), p])


def _cavity_start(prob, pos, seed):
    """The cavity at rest with the lid's velocity on the boundary and a weak perturbation inside."""
    x = prob.initial_state()
    rng = np.random.default_rng(seed)
    swirl = np.stack([np.sin(np.pi * pos[:, (c + 1) % 3]) for c in range(3)]) * rng.uniform(0.005, 0.02, (3, 1))
    inside = np.tile(prob.node_bnd < 0, 3)
    x[:3 * prob.n][inside] += swirl.reshape(-1)[inside]
    return x


def _heat_options(case):
    if case["precision"] == "mixed":
        return vfv.GmresOptions(tol=1e-14, restart=50, max_outer=2000, precond=L.PRECOND_ILU0, precision=L.MIXED, inner_rtol=1e-6,
                                ilu_order=L.ILU_NATURAL, ilu_sweeps=4, ilu_sweep_half=1, engine=L.ENGINE_OVERLAP)
    return vfv.GmresOptions(tol=1e-13, restart=50, max_outer=2000, precond=L.PRECOND_ILU0, engine=L.ENGINE_OVERLAP)


def _heat_triplets(n, fields):
    """The operators' triplets as the caller's assembly loop pushes them: per face the neighbour's
    coefficient and its negative on the diagonal, then the boundary rows."""
    c = _cube(n)
    v, nb, cf, _, b = _heat_system(c, fields, "cpu")
    own = (c.node_bnd[v] < 0) | (c.node_bnd[v] > 1)
    v, nb, cf = v[own], nb[own], cf.numpy()[own]
    dirichlet = np.nonzero((c.node_bnd == 0) | (c.node_bnd == 1))[0]
    rows = np.concatenate([np.repeat(v, 2), dirichlet]).astype(np.uint64)
    cols = np.concatenate([np.stack([nb, v], 1).reshape(-1), dirichlet]).astype(np.uint64)
    vals = np.concatenate([np.stack([cf, -cf], 1).reshape(-1), np.ones(dirichlet.size)])
    return rows, cols, vals, b.numpy()


def prepare(case, seed):
    kind = case["kind"]
    st = {"case": dict(case)}
    if kind == "linear":
        rows, cols, vals, b = _heat_triplets(case["n"], _heat_fields(case["n"], seed))
        pre = L.PRECOND_JACOBI if case["precond"] == "jacobi" else L.PRECOND_ILU0
        lin = vfv.LinearGmres.new_with_options(1, 1e-10, 50, 2000, precond=pre)
        lin.update_sparse((rows, cols, vals), b.size)
        st |= {"lin": lin, "trip": (rows, cols, vals), "b": b, "x0": np.zeros(b.size)}
    elif kind in ("residual", "heat", "gradient"):
        n = case["n"]
        k, q, s, T0, bc = _heat_fields(n, seed, prod=-0.3 if kind == "residual" else 0.0)
        st["heat"] = heat = _heat(n)
        if kind == "residual":
            T0 = _state_T(n, seed)
        st["host"] = (k, q, s, T0, bc)
        if kind == "gradient":
            rng = np.random.default_rng(seed + 17)
            st["sensors"] = rng.choice(k.size, min(1000, k.size // 4), replace=False)
            st["targets"] = rng.uniform(0.0, 1.0, st["sensors"].size)
            st["opts"] = vfv.GmresOptions(tol=1e-12, restart=50, max_outer=2000, precond=L.PRECOND_ILU0)
        elif kind == "heat":
            st["opts"] = _heat_options(case)
        if kind == "residual" or case.get("device"):
            st["dev"] = [torch.tensor(a, device="cuda") for a in st["host"]]
            st["out"] = torch.empty(k.size, dtype=torch.float64, device="cuda")
            view = type("View", (), {"__cuda_array_interface__": {"shape": (k.size,), "typestr": "<f8", "version": 2,
                                                                  "data": (heat.rhs_device_ptr, False)}})
            st["rhs"] = torch.as_tensor(view(), device="cuda")
            torch.cuda.synchronize()
    elif kind in ("transport", "transport_adjoint"):
        tr, pos = _batch(case)
        vel, c0, D = _transport_fields(case, seed, pos)
        st |= {"tr": tr, "vel": vel, "c0": c0, "D": D}
        if kind == "transport":
            order = L.ILU_NATURAL if case["order"] == "natural" else L.ILU_MULTICOLOR
            st["opts"] = vfv.GmresOptions(tol=1e-12, restart=30, max_outer=200, precond=L.PRECOND_ILU0, precision=L.MIXED, inner_rtol=1e-6,
                                          ilu_order=order, ilu_sweeps=case["sweeps"])
        else:
            st["target"] = np.full(c0.size, float(np.mean(c0)))
    else:
        prob, fl, pos = _flow(case["n"])
        st["flow"] = fl
        if kind == "flow_residual":
            st["x"] = _flow_state(prob, pos, seed)
            st["xd"] = torch.tensor(st["x"], device="cuda")
            st["bd"], st["ax"] = torch.empty_like(st["xd"]), torch.empty_like(st["xd"])
            torch.cuda.synchronize()
        else:
            st["x"] = _cavity_start(prob, pos, seed)
            st["opts"] = flow_options(tol=1e-8, max_outer=100)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "linear":
        a = st["lin"].build_matrix(st["trip"])
        return {"x": st["lin"].solve_matrix(a, st["b"], st["x0"], st["b"].size)}
    if kind == "residual":
        p = [t.data_ptr() for t in st["dev"]]
        st["heat"].assemble_device(*p)
        st["heat"].pattern.spmv_device(p[3], st["out"].data_ptr())
        return {"AT": st["out"], "b": st["rhs"]}
    if kind == "heat":
        heat = st["heat"]
        if case["device"]:
            p = [t.data_ptr() for t in st["dev"]]
            heat.assemble_device(*p)
            heat.pattern.solve_device(heat.rhs_device_ptr, p[3], st["out"].data_ptr(), st["opts"])
            return {"T": st["out"]}
        k, q, s, T0, bc = st["host"]
        b = heat.assemble(k, q, s, T0, bc)
        return {"T": heat.pattern.solve(b, T0, st["opts"])[0]}
    if kind == "gradient":
        heat = st["heat"]
        k, q, s, T0, bc = st["host"]
        b = heat.assemble(k, q, s, T0, bc)
        T = heat.pattern.solve(b, T0, st["opts"])[0]
        g = np.zeros(T.size)
        g[st["sensors"]] = T[st["sensors"]] - st["targets"]
        _, dlogk, dq, _ = heat.adjoint(T, g, st["opts"])
        return {"T": T, "dlogk": dlogk, "dq": dq}
    if kind == "transport":
        st["tr"].assemble(st["D"], st["vel"])
        return {"c": st["tr"].run(st["c0"], case["steps"], st["opts"])[0]}
    if kind == "transport_adjoint":
        st["tr"].assemble(st["D"], st["vel"])
        J, dJdD = st["tr"].adjoint_D(st["c0"], case["steps"], st["target"], every=case["every"])
        return {"J": J, "dJdD": dJdD}
    fl = st["flow"]
    if kind == "flow_residual":
        fl.assemble_device(st["xd"].data_ptr(), st["bd"].data_ptr())
        fl.pattern.spmv_device(st["xd"].data_ptr(), st["ax"].data_ptr())
        return {"Ax": st["ax"], "b": st["bd"]}
    r = fl.picard(st["x"], max_iter=2, tol=1e-300, damp=0.8, opts=st["opts"], raise_on_error=False)
    return {"x": r.x, "change": np.asarray(r.residuals)}


# ---------------------------------------------------------------- bytes and operations
def work(case):
    """Inputs read once and outputs written once: the fields, the dual's geometry (about 15.3 directed
    faces per vertex, 15.4 + 179 n_u for the coupled system) and the results."""
    kind = case["kind"]
    if kind in ("transport", "transport_adjoint"):
        rows = float(np.sum(_batch_sizes(case).astype(np.float64) ** 3))
        nnz, solves = 16.3 * rows, case["steps"] * (1 if kind == "transport" else 3)
        # geometry once; the matrix (FP64) once per implicit step
        return {"bytes": 15.3 * rows * 100 + solves * (12 * nnz + 24 * rows), "flops": solves * 2 * nnz}
    rows = float(case["n"]) ** 3
    if kind.startswith("flow"):
        nnz, passes = 179.0 * 4 * rows, 1 if kind == "flow_residual" else 2
        return {"bytes": passes * (15.3 * rows * 92 + 20 * nnz + 96 * rows), "flops": passes * 6 * nnz}
    nnz, passes = 16.1 * rows, 2 if kind == "gradient" else 1
    if kind == "linear":
        return {"bytes": 16 * 15.3 * 2 * rows + 20 * nnz + 24 * rows, "flops": 2 * nnz}
    return {"bytes": passes * (72 * 15.3 * rows + 20 * nnz + 48 * rows), "flops": passes * 40 * nnz}


# ---------------------------------------------------------------- the same in float64 with torch
def _dual(meshes, device):
    """Directed faces of the concatenated meshes: owners, neighbours and geometry."""
    out = {k: [] for k in ("v", "nb", "area", "dist", "cvol", "norm", "skew", "gw", "cskew")}
    ptr, rows, faces = [np.zeros(1, np.int64)], 0, 0
    for m in meshes:
        d = m.dual()
        out["v"].append(rows + np.repeat(np.arange(m.n_tot), np.diff(d["nbr_ptr"])))
        out["nb"].append(rows + d["nbr_idx"].astype(np.int64))
        for k, src in (("area", "area"), ("dist", "dist"), ("cvol", "cvol"), ("norm", "norm"), ("skew", "skew"), ("gw", "grad_wgt"),
                       ("cskew", "cskew")):
            out[k].append(np.asarray(d[src]))
        ptr.append(faces + d["nbr_ptr"][1:])
        rows, faces = rows + m.n_tot, faces + m.n_dir
    g = {k: torch.tensor(np.concatenate(a, axis=-1), device=device) for k, a in out.items()}
    g["ptr"], g["rows"] = torch.tensor(np.concatenate(ptr), device=device), rows
    return g


def _sum_rows(g, x):
    """Sums over each vertex's faces (last axis)."""
    c = torch.zeros(x.shape[:-1] + (g["rows"],), dtype=x.dtype, device=x.device)
    return c.index_add(-1, g["v"], x)


def _grad(g, f):
    return _sum_rows(g, g["gw"] * (f[g["nb"]] - f[g["v"]]))


def _face_cond(g, k):
    """Harmonic-mean face coefficient with the guarded skew correction, times area over distance."""
    v, nb = g["v"], g["nb"]
    gk = _grad(g, k)
    km = 2 * k[v] * k[nb] / (k[v] + k[nb])
    kf = km + 0.5 * (g["skew"] * (gk[:, v] + gk[:, nb])).sum(0)
    return torch.where(kf > 0, kf, km) * g["area"] / g["dist"]


def _heat_b(c, g, q, s, T, bc):
    """Right-hand side and the production's diagonal (zero-flux or Dirichlet boundaries)."""
    gq, gs, gT = _grad(g, q), _grad(g, s), _grad(g, T)
    cs = g["cskew"]
    b = -s * (gT * cs).sum(0) * g["cvol"] - (q + (gq * cs).sum(0)) * g["cvol"]
    dirichlet = torch.tensor((c.node_bnd == 0) | (c.node_bnd == 1), device=b.device)
    return torch.where(dirichlet, bc, b), (s + (gs * cs).sum(0)) * g["cvol"], dirichlet


def _heat_system(c, fields, device):
    """(owners, neighbours, face coefficients, production diagonal, right-hand side)"""
    k, q, s, T, bc = (torch.tensor(a, device=device) for a in fields)
    g = _dual([c.mesh], device)
    b, prod, _ = _heat_b(c, g, q, s, T, bc)
    return g["v"].cpu().numpy(), g["nb"].cpu().numpy(), _face_cond(g, k), prod, b


def _matvec(g, off):
    """x -> sum over faces of off * x[neighbour] (a CSR product)."""
    m = torch.sparse_csr_tensor(g["ptr"], g["nb"], off, size=(g["rows"], g["rows"]))
    return lambda x: torch.mv(m, x)


def _solve_spd(mv, diag, free, b, x):
    """Conjugate gradients, restarted on the true residual, for the symmetric block of the free rows."""
    x = x.clone()
    inv = torch.where(free, 1 / diag, torch.zeros_like(diag))
    best, best_x = math.inf, x
    for _ in range(12):
        r = torch.where(free, b - mv(x), torch.zeros_like(b))
        rn = float(r.norm())
        if not rn < 0.3 * best:
            break
        best, best_x = rn, x.clone()
        d, z = torch.zeros_like(x), inv * r
        p, rz = z.clone(), torch.dot(r, inv * r)
        for it in range(4000):
            ap = torch.where(free, mv(p), torch.zeros_like(p))
            a = rz / torch.dot(p, ap)
            d += a * p
            r = r - a * ap
            z = inv * r
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
            if it % 50 == 49 and float(r.norm()) < 1e-9 * rn:
                break
        x = x + d
    return best_x


def _heat_solve(g, cond, dirichlet, b, transpose=False):
    """A x = b (or A^T x = b): rows of the Dirichlet nodes are the identity."""
    free = ~dirichlet
    zero = torch.zeros_like(cond)
    inner = _matvec(g, torch.where(free[g["v"]] & free[g["nb"]], cond, zero))
    diag = _sum_rows(g, cond)
    edge = torch.where(free[g["v"]] & ~free[g["nb"]], cond, zero)  # A[free, dirichlet]

    def mv(x):
        return diag * x - inner(x)
    if transpose:
        x = _solve_spd(mv, diag, free, -b, torch.zeros_like(b))
        lam = torch.where(free, x, torch.zeros_like(x))
        at = torch.zeros_like(b).index_add(0, g["nb"], edge * lam[g["v"]])
        return torch.where(dirichlet, b - at, lam)
    xd = torch.where(dirichlet, b, torch.zeros_like(b))
    x = _solve_spd(mv, diag, free, -(b - _sum_rows(g, edge * xd[g["nb"]])), torch.zeros_like(b))
    return torch.where(dirichlet, b, x)


def _exact_heat(case, seed):
    n, kind = case["n"], case["kind"]
    c = _cube(n)
    fields = list(_heat_fields(n, seed, prod=-0.3 if kind == "residual" else 0.0))
    if kind == "residual":
        fields[3] = _state_T(n, seed)
    g = _dual([c.mesh], "cuda")
    k, q, s, T, bc = (torch.tensor(a, device="cuda") for a in fields)
    b, prod, dirichlet = _heat_b(c, g, q, s, T, bc)
    cond = _face_cond(g, k)
    if kind == "residual":
        at = _sum_rows(g, cond * T[g["nb"]]) + (prod - _sum_rows(g, cond)) * T
        return {"AT": torch.where(dirichlet, T, at), "b": b}
    x = _heat_solve(g, cond, dirichlet, b)
    if kind == "linear":
        return {"x": x}
    if kind == "heat":
        return {"T": x}
    rng = np.random.default_rng(seed + 17)
    sensors = torch.tensor(rng.choice(k.numel(), min(1000, k.numel() // 4), replace=False), device="cuda")
    targets = torch.tensor(rng.uniform(0.0, 1.0, sensors.numel()), device="cuda")
    dJdT = torch.zeros_like(x)
    dJdT[sensors] = x[sensors] - targets
    lam = _heat_solve(g, cond, dirichlet, dJdT, transpose=True)
    logk, qv = torch.log(k).requires_grad_(True), q.clone().requires_grad_(True)
    cond = _face_cond(g, torch.exp(logk))
    b, _, _ = _heat_b(c, g, qv, s, T, bc)
    res = torch.where(dirichlet, x, _sum_rows(g, cond * (x[g["nb"]] - x[g["v"]]))) - b
    dlogk, dq = torch.autograd.grad(-(lam * res).sum(), (logk, qv))
    return {"T": x, "dlogk": dlogk, "dq": dq}


def _transport_off(g, flux, D):
    """Off-diagonal coefficients (diffusion plus power-law advection) of every directed face."""
    cond = D * g["area"] / g["dist"]
    return cond * torch.clamp(1 - 0.1 * (flux / cond).abs(), min=0) ** 5 + torch.clamp(-flux, min=0)


def _exact_transport(case, seed):
    tr, pos = _batch(case)
    vel, c0, D = _transport_fields(case, seed, pos)
    g = _dual(tr.meshes, "cuda")
    v, nb = g["v"], g["nb"]
    vel, c0 = torch.tensor(vel, device="cuda"), torch.tensor(c0, device="cuda")
    flux = torch.zeros_like(g["area"])
    for a in range(3):
        gu = _grad(g, vel[a])
        uf = 0.5 * (vel[a][v] + vel[a][nb]) + 0.5 * (g["skew"] * (gu[:, v] + gu[:, nb])).sum(0)
        flux = flux + uf * g["norm"][a]
    flux = flux * g["area"]
    D = torch.tensor(D, dtype=torch.float64, device="cuda")
    off = _transport_off(g, flux, D)
    mass = g["cvol"] / 1e-2
    diag = mass + _sum_rows(g, off)
    mv = _matvec(g, off)

    def step(c):  # (diag - off) x = mass c, an M-matrix: Jacobi iterations
        x = c
        for _ in range(200):
            new = (mv(x) + mass * c) / diag
            if float((new - x).abs().max()) < 1e-16:
                return new
            x = new
        return x
    states = [c0]
    for _ in range(case["steps"]):
        states.append(step(states[-1]))
    if case["kind"] == "transport":
        return {"c": states[-1]}
    r = states[-1] - float(np.mean(c0.cpu().numpy()))

    def step_t(b):  # (diag - off)^T x = b
        x = b / diag
        for _ in range(300):
            new = (torch.zeros_like(b).index_add(0, nb, off * x[v]) + b) / diag
            if float((new - x).abs().max()) < 1e-16 * float(x.abs().max()):
                return new
            x = new
        return x
    Dg = D.clone().requires_grad_(True)
    total, lam = 0.0, step_t(-r)  # A = off - diag, so A^T lam = r
    for k in range(case["steps"], 0, -1):
        c = states[k]
        o = _transport_off(g, flux, Dg)
        total -= float(torch.autograd.grad((lam * _sum_rows(g, o * (c[nb] - c[v]))).sum(), Dg)[0])
        if k > 1:
            lam = step_t(mass * lam)
    return {"J": 0.5 * float((r * r).sum()), "dJdD": total}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("linear", "residual", "heat", "gradient"):
        return _exact_heat(case, seed)
    if kind in ("transport", "transport_adjoint"):
        return _exact_transport(case, seed)
    return None  # the coupled flow system has no short restatement
