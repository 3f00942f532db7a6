"""The work that programs have this library do, for timing it.

Every case goes through the public entry points of ``espreso_b200.feti4i`` (the FETI4I C API) or
``espreso_b200.adjoint``, with caller data where such callers hold it: host arrays for FETI4I, device
arrays for the allocation-free SYMV.  Kinds:

solve    one load step on a kept instance: new right-hand side, dual PCG, displacements
multi    several load cases of one structure solved together
create   a new structure: element matrices in, one solve, everything released
adjoint  one design step: densities -> displacements, and the gradient of a loss on them
symv     the allocation-free batched SYMV on tiles that the caller keeps

Meshes, materials and loads are those of ``espreso_b200.problems``; the seed draws conductivities,
moduli, densities and loads.
"""
from __future__ import annotations

import functools
import math
from dataclasses import replace

import numpy as np
import torch

from espreso_b200 import adjoint as A
from espreso_b200 import feti4i as F
from espreso_b200 import problems

PRECOND = {"none": F.PREC_NONE, "lumped": F.PREC_LUMPED, "dirichlet": F.PREC_DIRICHLET}
STORAGE = {"fp64": F.FP64, "fp32": F.FP32}
# dual PCG iterations to the stop rule, for work(): typical of each set-up, not of one mesh
ITERATIONS = {"lumped": 30, "dirichlet": 20, "none": 60, "hybrid": 60}


def _case(name, kind, **kw):
    c = dict(kind=kind, physics="heat", clusters=1, domains=4, elements=8, levels=0, hybrid=False,
             storage="fp64", precond="lumped", explicit=True, nrhs=1, matrices=0, order_lo=0, order_hi=0)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small model: every launch and every host step shows
        _case("solve_heat_8_tiny", "solve", domains=2, elements=4),
        # linear elasticity at the 64-subdomain size, the library's default FP64 storage
        _case("solve_elasticity_64", "solve", physics="elasticity", domains=4, elements=8),
        # the headline workload: heat, 512 subdomains, FP32 tiles with FP64 residual replacement
        _case("solve_heat_512_fp32", "solve", domains=8, elements=10, storage="fp32"),
        # a partitioner's subdomains: unequal sizes, ragged tile edges
        _case("solve_uneven_64_fp32", "solve", physics="elasticity", domains=1, elements=40, levels=6, storage="fp32"),
        # the reference's default preconditioner
        _case("solve_dirichlet_27", "solve", physics="elasticity", domains=3, elements=6, precond="dirichlet"),
        # Hybrid Total FETI: clusters with corner constraints, a small coarse problem
        _case("solve_hybrid_64", "solve", physics="elasticity", clusters=2, domains=2, elements=6, hybrid=True),
        # a full batch of load cases on the headline workload
        _case("multi_heat_512_fp32_32", "multi", domains=8, elements=10, storage="fp32", nrhs=32),
        # a few load cases, not a power of two, FP64
        _case("multi_elasticity_64_11", "multi", physics="elasticity", domains=4, elements=6, nrhs=11),
        # a new structure per call (parameter studies)
        _case("create_heat_125", "create", domains=5, elements=9),
        # topology optimisation: new densities, forward and backward
        _case("adjoint_64", "adjoint", physics="elasticity", domains=4, elements=6),
        # the caller's own tiles: a handful of small matrices, and a full set of unequal ones
        _case("symv_small", "symv", matrices=8, order_lo=60, order_hi=130),
        _case("symv_large", "symv", matrices=512, order_lo=333, order_hi=1111),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["solve", "solve", "solve", "multi", "multi", "create", "adjoint", "symv"])
    if kind == "symv":
        lo = log(1, 800)
        return _case(None, kind, matrices=log(1, 900), order_lo=lo, order_hi=min(1200, lo + log(1, 600)))
    if kind == "adjoint":
        return _case(None, kind, physics="elasticity", domains=rng.randint(2, 4), elements=rng.randint(3, 6))
    physics = rng.choice(["heat", "elasticity"])
    if kind == "create":
        d, e = (rng.randint(2, 5), rng.randint(3, 9)) if physics == "heat" else (rng.randint(2, 4), rng.randint(3, 6))
        return _case(None, kind, physics=physics, domains=d, elements=e, storage=rng.choice(["fp64", "fp32"]))
    d, e = (rng.randint(2, 8), rng.randint(3, 10)) if physics == "heat" else (rng.randint(2, 4), rng.randint(3, 8))
    c = _case(None, kind, physics=physics, domains=d, elements=e, storage=rng.choice(["fp64", "fp32"]))
    if kind == "multi":
        c["nrhs"] = rng.randint(2, 32)
        return c
    form = rng.choice(["plain", "plain", "dirichlet", "hybrid", "uneven", "implicit"])
    if form == "dirichlet":
        c["precond"] = "dirichlet"
    elif form == "hybrid":
        c.update(hybrid=True, clusters=rng.randint(2, 3), domains=2, elements=rng.randint(3, 6))
    elif form == "uneven":
        # 8 or 64 subdomains
        levels, elements = rng.choice([(3, rng.randint(12, 20)), (6, rng.randint(24, 40))])
        c.update(domains=1, levels=levels, elements=elements)
    elif form == "implicit":
        c.update(explicit=False, storage="fp64")
    return c


# ---- inputs ----------------------------------------------------------------------------------------

@functools.lru_cache(maxsize=4)
def _mesh(physics, clusters, domains, elements, levels):
    """The mesh with the element matrices of the unit material; a program keeps it over its materials."""
    d3, e3, c3 = (domains,) * 3, (elements,) * 3, (clusters,) * 3
    if levels:
        # pieces of 6..14 elements per side at the 40^3 grid, in proportion at the others
        lo, hi = (elements // 3, elements // 2 + 2) if levels == 3 else (elements * 3 // 20, elements * 7 // 20)
        kw = dict(k_range=(1.0, 1.0)) if physics == "heat" else dict(E=1.0)
        return problems.uneven_cube(physics, side=e3, levels=levels, lo=lo, hi=hi, seed=0, **kw)
    if physics == "heat":
        return problems.heat_cube(c3, d3, e3, k_range=(1.0, 1.0))
    return problems.elasticity_cube(c3, d3, e3, E=1.0)


def _problem(case, seed):
    """(mesh with this seed's material, its right-hand side)"""
    P = _mesh(case["physics"], case["clusters"], case["domains"], case["elements"], case["levels"])
    rng = np.random.default_rng(seed)
    nel = P.elem_nodes.shape[0]
    if case["physics"] == "heat":
        scale = 10.0 ** rng.uniform(0.0, 2.0, nel)        # conductivity, log-uniform on [1, 100]
    else:
        scale = 2.1e11 * rng.uniform(0.5, 1.5, nel)       # Young's modulus
    dofs = P.elem_dofs()
    f = np.bincount(dofs.ravel(), P.fe.ravel(), minlength=P.ndofs)
    f *= 1.0 + 0.25 * rng.standard_normal(f.size)
    return replace(P, Ke=P.Ke * scale[:, None, None]), f


def _instance(P, f, case):
    F.set_extended(F.EXT_SCHUR_PRECISION, STORAGE[case["storage"]])
    F.set_extended(F.EXT_SCHUR_EXPLICIT, 1 if case["explicit"] else 0)
    M = F.Matrix(0)
    try:
        M.add_elements(P.elem_nodes, P.elem_dofs(), P.Ke)
        M.set_partition(P.elem_domain)
        if case["hybrid"]:
            M.set_clusters(P.sub_cluster())
        dd, dv = P.dirichlet_dofs()
        return F.Instance(M, f, dd, dv,
                          iopts={F.PRECONDITIONER: PRECOND[case["precond"]], F.VERBOSE_LEVEL: 0,
                                 F.MAX_ITERATIONS: 2000, F.FETI_METHOD: 1 if case["hybrid"] else 0},
                          ropts={F.PRECISION: 1e-8})
    finally:
        M.destroy()
        F.set_extended(F.EXT_SCHUR_PRECISION, F.FP64)
        F.set_extended(F.EXT_SCHUR_EXPLICIT, 1)


class _State:
    inst = None

    def __del__(self):
        if self.inst is not None:
            self.inst.destroy()


def _orders(case):
    """Matrix orders: the caller's structure, the same for every seed."""
    rng = np.random.default_rng(case["matrices"])
    return rng.integers(case["order_lo"], case["order_hi"] + 1, case["matrices"])


def _symv_inputs(case, seed):
    """Symmetric positive definite matrices (upper 32x32 tiles, zero beyond the order) and vectors, on the GPU."""
    order = _orders(case)
    T = (order + 31) // 32
    ntiles = T * (T + 1) // 2
    off = np.concatenate([[0], np.cumsum(ntiles)])
    voff = np.concatenate([[0], np.cumsum(order)])
    g = torch.Generator(device="cuda").manual_seed(seed)
    tiles = torch.randn(int(off[-1]), 32, 32, dtype=torch.float64, device="cuda", generator=g)
    x = torch.randn(int(voff[-1]), dtype=torch.float64, device="cuda", generator=g)
    # row-major upper tiles (I <= J): masks by position, the same for every matrix size
    I = np.concatenate([np.repeat(np.arange(t), np.arange(t, 0, -1)) for t in T])
    J = np.concatenate([np.concatenate([np.arange(i, t) for i in range(t)]) for t in T])
    n = torch.from_numpy(np.repeat(order, ntiles)).cuda()
    I, J = torch.from_numpy(I).cuda(), torch.from_numpy(J).cuda()
    k = torch.arange(32, device="cuda")
    diag = torch.nonzero(I == J).ravel()
    d = tiles[diag]
    tiles[diag] = d + d.transpose(1, 2) + 3.0 * n[diag].double().sqrt()[:, None, None] * torch.eye(32, device="cuda")
    tiles *= ((32 * I)[:, None] + k < n[:, None])[:, :, None]
    tiles *= ((32 * J)[:, None] + k < n[:, None])[:, None, :]
    return order, off, voff, tiles, x, I, J


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    if s.kind == "symv":
        s.order, off, voff, s.tiles, s.x, _, _ = _symv_inputs(case, seed)
        s.off = torch.from_numpy(off[:-1].astype(np.int64)).cuda()
        s.dorder = torch.from_numpy(s.order.astype(np.int32)).cuda()
        s.voff = torch.from_numpy(voff[:-1].astype(np.int32)).cuda()
        s.max_order = int(s.order.max())
        s.y, s.dot = torch.empty_like(s.x), torch.empty(1, dtype=torch.float64, device="cuda")
    elif s.kind == "adjoint":
        P = _mesh("elasticity", 1, case["domains"], case["elements"], 0)
        f, rho = _design(P, seed)
        s.rho = torch.from_numpy(rho)
        s.model = A.SIMPModel(P, P.Ke, rhs=f, precision=1e-10)
        s.model.solve(rho)                               # the design loop's first state
        s.target = torch.from_numpy(np.random.default_rng(seed + 1).standard_normal(P.ndofs))
    else:
        s.P, s.f = _problem(case, seed)
        s.case = case
        if s.kind != "create":
            s.inst = _instance(s.P, s.f, case)
            s.out = np.zeros(s.P.ndofs)
        if s.kind == "multi":
            s.R = problems.traction_loads(s.P, case["nrhs"], seed=seed)
    return s


def _design(P, seed):
    rng = np.random.default_rng(seed)
    rho = rng.uniform(0.3, 1.0, P.elem_nodes.shape[0])
    f = np.zeros(P.ndofs)
    tip = np.nonzero(np.abs(P.coords[:, 0] - P.coords[:, 0].max()) < 1e-12)[0]
    f[3 * tip + 2] = -1e6 * rng.uniform(0.5, 1.5, tip.size)
    return f, rho


def run(s):
    if s.kind == "symv":
        F.tiled_symv_noalloc(s.tiles.data_ptr(), s.off.data_ptr(), s.dorder.data_ptr(), s.voff.data_ptr(),
                             s.order.size, s.max_order, s.x.data_ptr(), s.y.data_ptr(), s.dot.data_ptr(),
                             torch.cuda.current_stream().cuda_stream)
        return s.y, s.dot
    if s.kind == "solve":
        s.inst.update_rhs(s.f)
        return s.inst.solve(s.out)
    if s.kind == "multi":
        return s.inst.solve_multi(s.R)
    if s.kind == "create":
        inst = _instance(s.P, s.f, s.case)
        try:
            return inst.solve()
        finally:
            inst.destroy()
    rho = s.rho.clone().requires_grad_(True)
    u = A.solve(rho, s.model)
    (u * s.target).sum().backward()
    return u.detach(), rho.grad


# ---- what a pass cannot do without -------------------------------------------------------------------

def _boxes(case):
    """(element counts, interfaces per axis, clamped face) of every subdomain."""
    if case["levels"]:
        n = 2 ** case["levels"]
        side = case["elements"] / n ** (1 / 3)           # the mean box
        return [(side, side, side, 2 - 2 / n ** (1 / 3), 2 - 2 / n ** (1 / 3), 2 - 2 / n ** (1 / 3), 0)] * n
    n, e = case["clusters"] * case["domains"], case["elements"]
    cut = [(0 if n == 1 else 1 if i in (0, n - 1) else 2) for i in range(n)]
    return [(e, e, e, cut[i], cut[j], cut[k], int((i if case["physics"] != "heat" else k) == 0))
            for k in range(n) for j in range(n) for i in range(n)]


def work(case):
    if case["kind"] == "symv":
        n = _orders(case).astype(float)
        return {"bytes": float(np.sum(n * (n + 1) / 2 * 8 + 16 * n)), "flops": float(np.sum(2 * n * n))}
    dpn = 1 if case["physics"] == "heat" else 3
    its = ITERATIONS["hybrid" if case["hybrid"] else case["precond"]]
    size = 4 if case["storage"] == "fp32" else 8
    tri = rows = dofs = elim = nnz = 0.0
    for ex, ey, ez, cx, cy, cz, clamp in _boxes(case):
        nodes = (ex + 1) * (ey + 1) * (ez + 1)
        r = dpn * ((ex + 1 + cx) * (ey + 1 + cy) * (ez + 1 + cz) - nodes + clamp * (ey + 1) * (ex + 1))
        n = dpn * nodes
        t = dpn * (nodes - (ex - 1) * (ey - 1) * (ez - 1))   # interface DOFs
        tri, rows, dofs = tri + r * (r + 1) / 2, rows + r, dofs + n
        nnz += ex * ey * ez * (8 * dpn) ** 2
        elim += (n ** 3 - t ** 3) / 3 + ((t + r) ** 3 - r ** 3) / 3
    nr = case["nrhs"]
    # per solve: each iteration reads the S_i triangles once and the dual vectors of every load case;
    # the load goes in, the displacements come out, the element matrices are the K^+ solves' input
    solve = {"bytes": its * (tri * size + nr * rows * 16) + 16.0 * nr * dofs + 2 * 8 * nnz,
             "flops": its * 4.0 * nr * tri}
    if case["kind"] in ("create", "adjoint"):
        n = 2 if case["kind"] == "adjoint" else 1
        return {"bytes": n * solve["bytes"] + 8 * nnz + 8 * tri, "flops": n * solve["flops"] + elim}
    return solve


def tolerance(case):
    if case["kind"] == "symv":
        return {"rel": 4e-15, "max": 4e-14}              # FP64 sums in another order
    if case["kind"] == "adjoint":
        return {"rel": 1e-9, "max": 1e-8}                # two solves to 1e-10
    # the PCG stops where |w| < 1e-8 of its start: solutions of equally good iterations differ by about
    # their error, seen at up to 1.7e-9
    return {"rel": 1e-8, "max": 1e-7}


# ---- the same in 64 bits ------------------------------------------------------------------------------

def _cg(dofs, Ke, fixed, f):
    """K u = f with u = 0 at the fixed DOFs: Jacobi-preconditioned CG over the element matrices, to the
    accuracy of 64 bits.  f (ndofs, columns)."""
    E, nd = dofs.shape
    free = torch.ones(f.shape[0], 1, dtype=torch.float64, device=f.device)
    free[fixed] = 0.0
    flat = dofs.reshape(-1)

    def mul(u):
        return torch.zeros_like(u).index_add_(0, flat, torch.bmm(Ke, u[flat].reshape(E, nd, -1)).reshape(E * nd, -1)) * free

    diag = torch.zeros(f.shape[0], 1, dtype=torch.float64, device=f.device)
    diag.index_add_(0, flat, torch.diagonal(Ke, dim1=1, dim2=2).reshape(-1, 1))
    u, r = torch.zeros_like(f), f * free
    stop = 1e-14 * r.norm(dim=0)
    z = r / diag
    p, rz = z.clone(), (r * z).sum(0)
    for it in range(20000):
        q = mul(p)
        a = rz / (p * q).sum(0).clamp_min(1e-300)
        u, r = u + a * p, r - a * q
        if it % 20 == 19 and bool((r.norm(dim=0) <= stop).all()):
            break
        z = r / diag
        new = (r * z).sum(0)
        p = z + (new / rz.clamp_min(1e-300)) * p
        rz = new
    return u


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["kind"] == "symv":
        order, off, voff, tiles, x, I, J = _symv_inputs(case, seed)
        y = torch.zeros_like(x)
        for m in range(order.size):
            n, t = int(order[m]), (int(order[m]) + 31) // 32
            a, b = int(off[m]), int(off[m + 1])
            S = torch.zeros(t, t, 32, 32, dtype=torch.float64, device=x.device)
            S[I[a:b], J[a:b]] = tiles[a:b]
            S[J[a:b], I[a:b]] = tiles[a:b].transpose(1, 2)
            S = S.permute(0, 2, 1, 3).reshape(32 * t, 32 * t)[:n, :n]
            y[int(voff[m]):int(voff[m + 1])] = S @ x[int(voff[m]):int(voff[m + 1])]
        return y, (x * y).sum().reshape(1)
    if case["kind"] == "adjoint":
        P = _mesh("elasticity", 1, case["domains"], case["elements"], 0)
        f, rho = _design(P, seed)
        E = 1e-9 + rho ** 3 * (2.1e11 - 1e-9)
        Ke, R = P.Ke * E[:, None, None], f[None]
    else:
        P, f = _problem(case, seed)
        Ke = P.Ke
        R = problems.traction_loads(P, case["nrhs"], seed=seed) if case["kind"] == "multi" else f[None]
    dofs = torch.from_numpy(P.elem_dofs()).to(dev)
    Ke = torch.from_numpy(Ke).to(dev)
    fixed = torch.from_numpy(P.dirichlet_dofs()[0].astype(np.int64)).to(dev)
    u = _cg(dofs, Ke, fixed, torch.from_numpy(np.ascontiguousarray(R.T)).to(dev))
    if case["kind"] != "adjoint":
        return u.T.contiguous() if case["kind"] == "multi" else u[:, 0].contiguous()
    g = torch.from_numpy(np.random.default_rng(seed + 1).standard_normal(P.ndofs)).to(dev)
    v = _cg(dofs, Ke, fixed, g[:, None])
    energy = torch.einsum("ei,eij,ej->e", v[:, 0][dofs], Ke, u[:, 0][dofs])
    dE = 3.0 * torch.from_numpy(rho ** 2).to(dev) * (2.1e11 - 1e-9) / torch.from_numpy(E).to(dev)
    return u[:, 0].contiguous(), -dE * energy
