"""The calls whose speed a user of this library sees, as measurable cases.

A case is a dict of plain values; ``prepare`` builds what a user's program holds before the
call (mesh, CRS pattern, a matrix with the seed's material, right-hand side), ``run`` makes one
pass through the public entry points, ``exact`` gives the same result from plain torch in
64 bits.  Kinds:

solve     SolveLinearSystem of one assembled system (scaling, preconditioner, Krylov loop,
          back-scaling): hex Poisson, tet Poisson on a randomly numbered mesh (bandwidth
          optimisation accepted, no shared column offsets), 3-DOF hex elasticity; host vectors
          (``Matrix.solve``) or device vectors (``Matrix.solve_dev``); FP64 or mixed
batch     many systems of uneven size in one batched mixed solve, solutions read back
residual  the matrix side of a nonlinear or time step: element assembly with new material,
          Dirichlet rows, and the product A u
product   A u alone on device vectors (Matrix Vector Proc)
"""
from __future__ import annotations

import collections
import math

import numpy as np
import torch

import elmerfem_b200 as eg
from elmerfem_b200 import _lib, meshgen

TOL = 1e-10
METHODS = {"cg": eg.CG, "bicgstab": eg.BICGSTAB}
PRECONDS = {"jacobi": eg.PREC_DIAGONAL, "ilu0": eg.PREC_ILU0}
PRECISIONS = {"fp64": eg.FP64, "mixed": eg.MIXED}


def listed():
    return [
        # the smallest call: a host program's 17^3-node Poisson problem, every step a few
        # microseconds of device work, so launches and latency count
        {"name": "hex16_cg_fp64_host", "kind": "solve", "mesh": "hex", "m": 16, "method": "cg", "precond": "jacobi",
         "precision": "fp64", "sigma": 0.0, "host": True},
        # the plain drop-in configuration: 32^3 hexahedra, BiCGStab + ILU0 from host vectors
        {"name": "hex32_bicgstab_ilu0_fp64_host", "kind": "solve", "mesh": "hex", "m": 32, "method": "bicgstab",
         "precond": "ilu0", "precision": "fp64", "sigma": 0.0, "host": True},
        # the same system as a mixed-precision request on device vectors
        {"name": "hex32_bicgstab_ilu0_mixed", "kind": "solve", "mesh": "hex", "m": 32, "method": "bicgstab",
         "precond": "ilu0", "precision": "mixed", "sigma": 0.0, "host": False},
        # the headline system: 128^3 hexahedra (2.1 M unknowns), log-normal conductivity, CG + Jacobi
        {"name": "hex128_cg_fp64", "kind": "solve", "mesh": "hex", "m": 128, "method": "cg", "precond": "jacobi",
         "precision": "fp64", "sigma": 1.0, "host": False},
        {"name": "hex128_cg_mixed", "kind": "solve", "mesh": "hex", "m": 128, "method": "cg", "precond": "jacobi",
         "precision": "mixed", "sigma": 1.0, "host": False},
        # bulk assembly of that mesh and one product with the matrix, as a nonlinear step does
        {"name": "hex128_residual", "kind": "residual", "mesh": "hex", "m": 128, "sigma": 1.0},
        # the matrix-vector product alone, at an odd size
        {"name": "hex101_product", "kind": "product", "mesh": "hex", "m": 101, "sigma": 1.0},
        # an unstructured numbering: rows without common column offsets
        {"name": "tet40_renumbered_cg_mixed", "kind": "solve", "mesh": "tet", "m": 40, "method": "cg",
         "precond": "jacobi", "precision": "mixed", "sigma": 0.5, "host": False},
        # elasticity with 3 unknowns a node (824 k unknowns, 65 M entries), BiCGStab + ILU0
        {"name": "elastic64_bicgstab_ilu0_fp64", "kind": "solve", "mesh": "elastic", "m": 64, "method": "bicgstab",
         "precond": "ilu0", "precision": "fp64", "sigma": 0.0, "host": False},
        # its assembly with new material constants, and one product
        {"name": "elastic48_residual", "kind": "residual", "mesh": "elastic", "m": 48, "sigma": 0.0},
        # batched solves of independent systems of uneven size: tets with CG + Jacobi, ...
        {"name": "batch96_tet_cg", "kind": "batch", "mesh": "tet", "systems": 96, "m_lo": 8, "m_hi": 60, "sizes": 1,
         "method": "cg", "precond": "jacobi", "sigma": 0.5},
        # ... and what the solve server steps through: hexahedra, BiCGStab + ILU0 by two sweeps
        {"name": "batch16_hex_bicgstab_ilu0", "kind": "batch", "mesh": "hex", "systems": 16, "m_lo": 16, "m_hi": 96,
         "sizes": 2, "method": "bicgstab", "precond": "ilu0", "sigma": 1.0},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["cg", "cg", "ilu0", "renumbered", "elastic", "residual", "residual", "product", "batch"])
    if kind == "cg":
        return {"kind": "solve", "mesh": "hex", "m": _log_int(rng, 12, 128), "method": "cg", "precond": "jacobi",
                "precision": rng.choice(["fp64", "mixed"]), "sigma": rng.choice([0.0, 0.5, 1.0]),
                "host": rng.random() < 0.3}
    if kind == "ilu0":
        return {"kind": "solve", "mesh": "hex", "m": _log_int(rng, 12, 80), "method": "bicgstab", "precond": "ilu0",
                "precision": rng.choice(["fp64", "mixed"]), "sigma": rng.choice([0.0, 0.5, 1.0]),
                "host": rng.random() < 0.3}
    if kind == "renumbered":
        return {"kind": "solve", "mesh": "tet", "m": _log_int(rng, 10, 60), "method": "cg", "precond": "jacobi",
                "precision": rng.choice(["fp64", "mixed"]), "sigma": 0.5, "host": False}
    if kind == "elastic":
        return {"kind": "solve", "mesh": "elastic", "m": _log_int(rng, 8, 56), "method": "bicgstab",
                "precond": "ilu0", "precision": "fp64", "sigma": 0.0, "host": rng.random() < 0.3}
    if kind == "residual":
        mesh = rng.choice(["hex", "tet", "elastic"])
        return {"kind": "residual", "mesh": mesh, "m": _log_int(rng, 12, {"hex": 128, "tet": 72, "elastic": 56}[mesh]),
                "sigma": 0.0 if mesh == "elastic" else 1.0}
    if kind == "product":
        mesh = rng.choice(["hex", "tet", "elastic"])
        return {"kind": "product", "mesh": mesh, "m": _log_int(rng, 16, {"hex": 128, "tet": 96, "elastic": 56}[mesh]),
                "sigma": 0.0 if mesh == "elastic" else 1.0}
    if rng.random() < 0.5:
        return {"kind": "batch", "mesh": "tet", "systems": _log_int(rng, 8, 128), "m_lo": 8,
                "m_hi": rng.randint(24, 60), "sizes": rng.randrange(1 << 20), "method": "cg", "precond": "jacobi",
                "sigma": 0.5}
    return {"kind": "batch", "mesh": "hex", "systems": _log_int(rng, 4, 24), "m_lo": 16, "m_hi": rng.randint(32, 80),
            "sizes": rng.randrange(1 << 20), "method": "bicgstab", "precond": "ilu0", "sigma": 1.0}


# ---------------------------------------------------------------- what a program keeps
# one context, and the mesh, pattern and bound prototype matrix of the meshes in use: a program
# builds these once per mesh and clones the prototype for each system
_ctx = None
_protos = collections.OrderedDict()
KEEP_MESHES = 24


def _context():
    global _ctx
    if _ctx is None:
        _ctx = eg.Context(0)
    return _ctx


def _batch_sizes(case):
    """The systems' mesh sizes: log-uniform over eight meshes between m_lo and m_hi."""
    rng = np.random.Generator(np.random.PCG64(int(case["sizes"])))
    grid = np.unique(np.round(np.exp(np.linspace(math.log(case["m_lo"]), math.log(case["m_hi"]), 8))).astype(int))
    return [int(grid[i]) for i in rng.integers(0, grid.size, int(case["systems"]))]


def _numbering(m):
    """new node number of every lexicographic node (0-based): one fixed random numbering per size"""
    return np.random.Generator(np.random.PCG64(7919 + m)).permutation((m + 1) ** 3)


def _mesh(kind, m, renumber):
    mesh = meshgen.tet_cube(m) if kind == "tet" else meshgen.hex_cube(m)
    if renumber:
        new = _numbering(m)
        coords = np.empty_like(mesh.coords)
        coords[new] = mesh.coords
        mesh = meshgen.Mesh(coords, mesh.elem_code, (new[mesh.elements - 1] + 1).astype(np.int32), mesh.bnd_code,
                            (new[mesh.bnd_elements - 1] + 1).astype(np.int32), mesh.bnd_ids, mesh.dims)
    return mesh


def _proto(kind, m, renumber, precond):
    key = (kind, m, renumber)
    if key not in _protos:
        while len(_protos) >= KEEP_MESHES:
            _protos.popitem(last=False)
        dofs = 3 if kind == "elastic" else 1
        mesh = _mesh(kind, m, renumber)
        pat = eg.create_matrix(mesh, dofs=dofs)
        P = eg.Matrix(_context(), pat)
        P.bind_assembly(mesh)
        nodes = mesh.boundary_nodes([1] if kind == "elastic" else range(1, 7))
        con = np.sort((dofs * (pat.perm[nodes - 1] - 1)[:, None] + np.arange(1, dofs + 1)).ravel()).astype(np.int32)
        _protos[key] = (mesh, pat, P, con)
    _protos.move_to_end(key)
    if precond is not None:
        _protos[key][2].prepare(precond)
    return _protos[key]


def _elastic_constants(seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    return (200e9 * rng.uniform(0.7, 1.3), rng.uniform(0.25, 0.35),
            [float(v) for v in rng.uniform(-0.2, 0.2, 2) * 1e4] + [-1e4])


def _material(case, m, seed):
    """(conductivity per element, nodal load) of one Poisson system: log-normal and a smooth
    positive source with noise, in the mesh's element order and lexicographic node order"""
    rng = np.random.Generator(np.random.PCG64(seed))
    nelem = m ** 3 * (6 if case["mesh"] == "tet" else 1)
    k = np.exp(rng.normal(0.0, case["sigma"], nelem)) if case["sigma"] > 0 else np.full(nelem, 1.0)
    load = 1.0 + rng.random((m + 1) ** 3)
    return k, load


def _rhs_random(con, n, seed):
    b = np.random.Generator(np.random.PCG64(seed + 1)).random(n)
    b[con - 1] = 0.0
    return b


def _params(case):
    return eg.SolverParams(method=METHODS[case["method"]], precond=PRECONDS[case["precond"]], tol=TOL, max_iter=20000,
                           precision=PRECISIONS[case.get("precision", "mixed")])


def prepare(case, seed):
    ctx = _context()
    renumber = case["kind"] == "solve" and case["mesh"] == "tet"
    s = {"case": case, "ctx": ctx, "stream": torch.cuda.ExternalStream(ctx.stream)}
    if case["kind"] == "batch":
        prm = _params(case)
        if case["precond"] == "ilu0":
            prm.ilu_sweeps = 2
        s["params"], s["mats"], s["b"] = prm, [], []
        for i, m in enumerate(_batch_sizes(case)):
            mesh, pat, P, con = _proto(case["mesh"], m, False, prm.precond)
            A = eg.Matrix.clone(P)
            k, load = _material(case, m, 1000 * seed + i)
            A.assemble_poisson(elem_k=k, load=load if case["mesh"] == "hex" else None)
            A.dirichlet(con, symmetric=case["method"] == "cg")
            s["mats"].append(A)
            s["b"].append(None if case["mesh"] == "hex"
                          else torch.from_numpy(_rhs_random(con, A.n, 1000 * seed + i)).cuda())
        return s
    m = case["m"]
    prm = _params(case) if case["kind"] == "solve" else None
    mesh, pat, P, con = _proto(case["mesh"], m, renumber, prm.precond if prm else None)
    A = eg.Matrix.clone(P)
    s.update(A=A, con=con, params=prm)
    if case["mesh"] == "elastic":
        s["elastic"] = _elastic_constants(seed)
        A.assemble_elastic(*s["elastic"])
        symmetric = False
    else:
        k, load = _material(case, m, seed)
        if renumber:
            moved = np.empty_like(load)
            moved[_numbering(m)] = load
            load = moved
        s["k"] = k
        A.assemble_poisson(elem_k=k, load=load if case["kind"] == "solve" else None)
        symmetric = case["kind"] != "solve" or case["method"] == "cg"
    A.dirichlet(con, symmetric=symmetric)
    s["symmetric"] = symmetric
    if case["kind"] == "solve":
        s["b"] = A.rhs()
        if not case["host"]:
            s["b"] = torch.from_numpy(s["b"]).cuda()
            s["x"] = torch.zeros(A.n, dtype=torch.float64, device="cuda")
        if renumber:
            s["perm"] = torch.from_numpy(pat.perm.astype(np.int64) - 1).cuda()
    else:
        u = torch.from_numpy(np.random.Generator(np.random.PCG64(seed + 2)).normal(size=A.n))
        s["u"], s["v"] = u.cuda(), torch.zeros(A.n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return s


def _product(s):
    _lib.check(_lib.lib().egpu_mv_dev(s["A"].handle, s["u"].data_ptr(), s["v"].data_ptr()), s["ctx"].handle,
               "egpu_mv_dev")
    return s["v"]


def run(state):
    s, case = state, state["case"]
    if case["kind"] == "batch":
        B = eg.Batch(s["ctx"], s["params"])
        ids = [B.add_matrix(A, None if b is None else b.data_ptr()) for A, b in zip(s["mats"], s["b"])]
        B.solve()
        x = np.concatenate([B.solution(i) for i in ids])
        B.free()
        return x
    if case["kind"] == "product":
        return _product(s)
    if case["kind"] == "residual":
        if case["mesh"] == "elastic":
            s["A"].assemble_elastic(*s["elastic"])
        else:
            s["A"].assemble_poisson(elem_k=s["k"])
        s["A"].dirichlet(s["con"], symmetric=s["symmetric"])
        if case["mesh"] == "elastic":
            return _product(s), s["A"].rhs()
        return _product(s)
    if case["host"]:
        return s["A"].solve(s["b"], params=s["params"])[0]
    with torch.cuda.stream(s["stream"]):  # the initial guess, on the stream that the solve runs on
        s["x"].zero_()
    s["A"].solve_dev(s["b"].data_ptr(), s["x"].data_ptr(), s["params"])
    if "perm" in s:  # the solution by node, as Elmer reads it through Perm
        return s["x"][s["perm"]]
    return s["x"]


def _sizes(mesh, m):
    """(unknowns, stored entries) of the structured meshes: 27-point and 15-point stencils"""
    nodes = (m + 1) ** 3
    if mesh == "tet":
        e, f, v = 3 * m * (m + 1) ** 2, 3 * m * m * (m + 1), m ** 3  # edges, face and body diagonals
        return nodes, nodes + 2 * (e + f + v)
    z = (3 * m + 1) ** 3
    return (3 * nodes, 9 * z) if mesh == "elastic" else (nodes, z)


def work(case):
    """Bytes and operations of one pass: a solve streams the matrix (values and columns; FP32
    values in a mixed solve) and about ten vectors once per product it cannot avoid."""
    if case["kind"] == "batch":
        parts = [work({**case, "kind": "solve", "m": m, "precision": "mixed", "host": False})
                 for m in _batch_sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, z = _sizes(case["mesh"], case["m"])
    if case["kind"] == "product":
        return {"bytes": 12.0 * z + 20.0 * n, "flops": 2.0 * z}
    if case["kind"] == "residual":
        m3 = case["m"] ** 3
        nelem, nen, flops = ((6 * m3, 4, 900.0) if case["mesh"] == "tet" else
                             (m3, 8, 5600.0) if case["mesh"] == "hex" else (m3, 8, 30000.0))
        # connectivity, coordinates and material once, the matrix written once and read once
        return {"bytes": nelem * (4.0 * nen + 8.0) + 24.0 * n + 20.0 * z + 20.0 * n, "flops": flops * nelem + 2.0 * z}
    m = case["m"]
    if case["method"] == "cg":
        its, products = (2.4 if case["mesh"] == "hex" else 2.0) * m + 20, 1.0
        factor = 0.0
    else:
        its, products = (2.6 if case["mesh"] == "elastic" else 0.5) * m + 4, 2.0
        factor = 2.0  # two applications of the ILU0 factors an iteration
    bz, bn = (12.0, 80.0) if case["precision"] == "fp64" else (8.0, 40.0)
    return {"bytes": its * ((products + factor) * bz * z + bn * n) + 32.0 * z,
            "flops": its * (2.0 * (products + factor) * z + 12.0 * n)}


# ---------------------------------------------------------------- the same in 64 bits, plain torch
def _gauss(code):
    """(weights, dN/dxi at the points, N at the points) on the reference element"""
    if code == "tet":  # linear: constant gradients, one point is exact
        dN = torch.tensor([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=torch.float64)[None]
        return torch.tensor([1.0 / 6.0], dtype=torch.float64), dN, torch.full((1, 4), 0.25, dtype=torch.float64)
    a = 1.0 / math.sqrt(3.0)
    sgn = torch.tensor([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1],
                        [-1, 1, 1]], dtype=torch.float64)
    f = 1.0 + sgn[None] * (a * sgn)[:, None]  # [point, node, axis]
    N = f.prod(2) / 8.0
    dN = torch.stack([sgn[None, :, 0] * f[..., 1] * f[..., 2], sgn[None, :, 1] * f[..., 0] * f[..., 2],
                      sgn[None, :, 2] * f[..., 0] * f[..., 1]], 2) / 8.0
    return torch.ones(8, dtype=torch.float64), dN, N


def _elements(mesh, m):
    """(element nodes, element corner offsets) of the unit cube's cells, 0-based lexicographic"""
    r = torch.arange(m)
    k, j, i = torch.meshgrid(r, r, r, indexing="ij")
    i, j, k = i.ravel(), j.ravel(), k.ravel()
    if mesh == "tet":
        tets = ((0, 1, 3, 7), (0, 1, 5, 7), (0, 2, 3, 7), (0, 2, 6, 7), (0, 4, 5, 7), (0, 4, 6, 7))
        corners = [[(c & 1, (c >> 1) & 1, (c >> 2) & 1) for c in t] for t in tets]
    else:
        corners = [[(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]]
    w = m + 1
    nodes = torch.stack([torch.stack([i + a + w * (j + b + w * (k + c)) for a, b, c in t], 1) for t in corners], 1)
    return nodes, torch.tensor(corners, dtype=torch.float64) / m  # [cell, type, node], [type, node, 3]


def _assembled(mesh, m, material):
    """CSR matrix (CUDA) without boundary conditions; material: k per element, or (E, nu)"""
    nodes, corners = _elements(mesh, m)
    wt, dN, _ = _gauss("tet" if mesh == "tet" else "hex")
    J = torch.einsum("tnc,gnx->tgcx", corners, dN)
    G = torch.einsum("gnx,tgxc->tgnc", dN, torch.linalg.inv(J))  # dN/d(coordinates)
    s = torch.linalg.det(J).abs() * wt
    nn, nen = (m + 1) ** 3, nodes.shape[2]
    if mesh == "elastic":
        E, nu = material
        cs = E / ((1 + nu) * (1 - 2 * nu))
        lam, mu = nu * cs, (0.5 - nu) * cs
        K = lam * torch.einsum("tg,tgpi,tgqj->tpiqj", s, G, G) + mu * torch.einsum("tg,tgpj,tgqi->tpiqj", s, G, G)
        K = K + mu * torch.einsum("tg,tgpk,tgqk,ij->tpiqj", s, G, G, torch.eye(3, dtype=torch.float64))
        K = K.reshape(1, 3 * nen, 3 * nen)
        dof = (3 * nodes[..., None] + torch.arange(3)).reshape(nodes.shape[0], 1, 3 * nen).cuda()
        n, val = 3 * nn, K.cuda().expand(nodes.shape[0], 1, -1, -1)
    else:
        K = torch.einsum("tg,tgpc,tgqc->tpq", s, G, G).cuda()
        dof, n = nodes.cuda(), nn
        val = torch.from_numpy(material).cuda().reshape(nodes.shape[0], nodes.shape[1], 1, 1) * K
    key = (dof[..., :, None] * n + dof[..., None, :]).reshape(-1)
    key, where = torch.unique(key, return_inverse=True)
    out = torch.zeros(key.numel(), dtype=torch.float64, device="cuda").index_add_(0, where, val.reshape(-1))
    row, col = key // n, key % n
    ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    diag = torch.zeros(n, dtype=torch.float64, device="cuda")
    diag[row[row == col]] = out[row == col]
    return torch.sparse_csr_tensor(ptr, col, out, (n, n)), diag


def _free(mesh, m):
    """1 for unknowns without a boundary condition"""
    g = torch.ones((m + 1,) * 3, dtype=torch.float64)
    g[:, :, 0] = 0
    if mesh == "elastic":
        return g.reshape(-1, 1).repeat(1, 3).reshape(-1).cuda()
    g[:, :, -1] = g[:, 0] = g[:, -1] = g[0] = g[-1] = 0
    return g.reshape(-1).cuda()


def _load_vector(mesh, m, load):
    """sum over elements of integral N_p (sum_q load_q N_q); load per node, or a body force"""
    nodes, corners = _elements(mesh, m)
    _, dN, N = _gauss("tet" if mesh == "tet" else "hex")
    vol = 1.0 / m ** 3
    if mesh == "elastic":
        f = torch.zeros((m + 1) ** 3, 3, dtype=torch.float64)
        f.index_add_(0, nodes.reshape(-1), (vol / 8.0 * torch.tensor(load, dtype=torch.float64)).expand(nodes.numel(), 3))
        return f.reshape(-1).cuda()
    if mesh == "tet":
        M = (vol / 6.0) / 20.0 * (torch.ones(4, 4, dtype=torch.float64) + torch.eye(4, dtype=torch.float64))
    else:
        M = vol / 8.0 * torch.einsum("gp,gq->pq", N, N)
    nodes = nodes.reshape(-1, nodes.shape[2]).cuda()
    f = torch.zeros((m + 1) ** 3, dtype=torch.float64, device="cuda")
    q = torch.from_numpy(load).cuda()[nodes] @ M.cuda()
    return f.index_add_(0, nodes.reshape(-1), q.reshape(-1))


def _cg(K, diag, free, b):
    """K x = b over the free unknowns (zero elsewhere), to the rounding level"""
    b = b * free
    minv = free / diag
    x, r = torch.zeros_like(b), b.clone()
    z = minv * r
    p, rz = z.clone(), torch.dot(r, z)
    stop = 1e-28 * rz
    for i in range(20000):
        q = free * (K @ p)
        a = rz / torch.dot(p, q)
        x += a * p
        r -= a * q
        z = minv * r
        new = torch.dot(r, z)
        if i % 16 == 0 and not bool(new > stop):
            break
        p = z + (new / rz) * p
        rz = new
    return x


def _exact_system(case, m, seed, b=None):
    mesh = case["mesh"]
    if mesh == "elastic":
        E, nu, force = _elastic_constants(seed)
        K, diag = _assembled(mesh, m, (E, nu))
        return _cg(K, diag, _free(mesh, m), _load_vector(mesh, m, force))
    k, load = _material(case, m, seed)
    K, diag = _assembled(mesh, m, k)
    f = _free(mesh, m)
    return _cg(K, diag, f, _load_vector(mesh, m, load) if b is None else b * f)


def exact(case, seed):
    mesh = case["mesh"]
    if case["kind"] == "batch":
        xs = []
        for i, m in enumerate(_batch_sizes(case)):
            b = None
            if mesh == "tet":  # the drawn right-hand side, zero on the boundary
                n = (m + 1) ** 3
                b = torch.from_numpy(np.random.Generator(np.random.PCG64(1000 * seed + i + 1)).random(n)).cuda()
            xs.append(_exact_system(case, m, 1000 * seed + i, b).cpu().numpy())
        return np.concatenate(xs)
    m = case["m"]
    if case["kind"] == "solve":
        x = _exact_system(case, m, seed)
        if mesh == "tet":  # by node of the renumbered mesh
            y = torch.empty_like(x)
            y[torch.from_numpy(_numbering(m)).cuda()] = x
            x = y
        return x.cpu().numpy() if case["host"] else x
    if mesh == "elastic":
        E, nu, force = _elastic_constants(seed)
        K, diag = _assembled(mesh, m, (E, nu))
    else:
        K, diag = _assembled(mesh, m, _material(case, m, seed)[0])
    f = _free(mesh, m)
    n = f.numel()
    u = torch.from_numpy(np.random.Generator(np.random.PCG64(seed + 2)).normal(size=n)).cuda()
    if mesh == "elastic":  # constrained rows become a_ii u_i = 0, columns stay
        return f * (K @ u) + (1 - f) * diag * u, (f * _load_vector(mesh, m, force)).cpu().numpy()
    return f * (K @ (f * u)) + (1 - f) * diag * u
