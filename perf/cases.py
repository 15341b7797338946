"""The work a program has this package do, as timed cases.

Every case is one call sequence of the elliptic-solve path on a jittered
unit-square or unit-cube mesh: a matrix-vector product, the assembly of a
system, a hierarchy set up for a new matrix, solves against a hierarchy that
is kept, batches of right-hand sides, the lazy preconditioner of a nonlinear
loop, and independent requests through the server.  Sizes reach from the
smallest meshes of the tests to the 64^3 benchmark workload.

Device inputs are made and used on the context's own stream, so nothing has
to be waited for between the caller's work and the library's.
"""
from __future__ import annotations

import math
import types

import numpy as np
import torch

from afepack_gb300 import _native as N
from afepack_gb300.amg import FP64, MIXED, AMGPreconditioner, AMGSolver
from afepack_gb300.fem import BoundaryConditionAdmin, Context, L2Discretize, Space, assemble
from afepack_gb300.mesh import Mesh, cube_mesh, square_mesh
from afepack_gb300.serve import Server
from afepack_gb300.workloads import ACC, Request, contrast_coefficient, gaussian_field, request_workload

TOL = 1e-12  # AMGSolver's own tolerance


def listed():
    return [
        # one product with a small matrix, as an iterative method of the caller's own does it: launch latency
        {"name": "vmult_2d_p1_24", "op": "vmult", "dim": 2, "degree": 1, "n": 24, "coef": False},
        # a new mesh on the host (an adaptive step): numbering, stiffness and mass, right-hand side, boundary data
        {"name": "system_2d_p1_181", "op": "system", "dim": 2, "degree": 1, "n": 181, "coef": False},
        # the stiffness and mass matrices again for a new coefficient, on a space that is kept; quadratic tetrahedra
        {"name": "assemble_3d_p2_21", "op": "assemble", "dim": 3, "degree": 2, "n": 21, "coef": True},
        # independent small requests, each with its own mesh, through the server (the served stream's small end)
        {"name": "served_2d_p1_8", "op": "served", "count": 8, "n_min": 32, "n_max": 100},
        # a new matrix each time, solved once: hierarchy and solve, the plain FP64 solver on a small 2D problem
        {"name": "new_2d_p1_97_fp64", "op": "new", "dim": 2, "degree": 1, "n": 97, "coef": True, "mixed": False},
        # the same at the size of the 3D benchmark workload, mixed precision
        {"name": "new_3d_p1_64_mixed", "op": "new", "dim": 3, "degree": 1, "n": 64, "coef": False, "mixed": True},
        # one right-hand side after another against a hierarchy that is kept (a time step), host vectors
        {"name": "pcg_3d_p1_48_mixed", "op": "pcg", "dim": 3, "degree": 1, "n": 48, "coef": False, "mixed": True},
        # the same in FP64 on quadratic triangles with a strongly varying coefficient: many iterations
        {"name": "pcg_2d_p2_121_fp64", "op": "pcg", "dim": 2, "degree": 2, "n": 121, "coef": True, "mixed": False},
        # the batched benchmark workload: 64 right-hand sides against one hierarchy, on the device
        {"name": "multi_3d_p1_64_x64_mixed", "op": "multi", "dim": 3, "degree": 1, "n": 64, "coef": False,
         "mixed": True, "k": 64},
        # a narrow, odd batch in FP64
        {"name": "multi_2d_p1_140_x7_fp64", "op": "multi", "dim": 2, "degree": 1, "n": 140, "coef": False,
         "mixed": False, "k": 7},
        # AMGSolver::solve as the reference's examples call it: 21 FP64 V-cycles, host vectors
        {"name": "stationary_2d_p1_256_fp64", "op": "stationary", "dim": 2, "degree": 1, "n": 256, "coef": False},
        # AMGPreconditioner in a nonlinear loop: new values on the same pattern, numeric re-setup, six V-cycles
        {"name": "lazy_3d_p2_13_fp64", "op": "lazy", "dim": 3, "degree": 2, "n": 13, "coef": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["vmult", "system", "assemble", "served", "new", "new", "pcg", "pcg", "multi", "multi", "stationary", "lazy"])
    if op == "served":
        return {"op": op, "count": rng.randint(3, 10), "n_min": rng.randint(24, 48), "n_max": rng.randint(60, 110)}
    kinds = {
        "vmult": {(2, 1): (16, 700), (3, 1): (6, 60), (2, 2): (12, 300), (3, 2): (5, 26)},
        "system": {(2, 1): (24, 300), (3, 1): (8, 36), (2, 2): (16, 160), (3, 2): (5, 16)},
        "assemble": {(2, 1): (24, 400), (3, 1): (8, 52), (2, 2): (16, 220), (3, 2): (6, 23)},
        "new": {(2, 1): (40, 220), (3, 1): (10, 44)},
        "pcg": {(2, 1): (40, 400), (3, 1): (10, 56), (2, 2): (24, 130)},
        "multi": {(2, 1): (40, 260), (3, 1): (10, 48)},
        "stationary": {(2, 1): (40, 360), (3, 1): (10, 44)},
        "lazy": {(2, 1): (40, 200), (2, 2): (16, 100), (3, 2): (6, 15)},
    }[op]
    dim, degree = rng.choice(sorted(kinds))
    case = {"op": op, "dim": dim, "degree": degree, "n": _log_int(rng, *kinds[(dim, degree)]),
            "coef": dim == 2 and rng.random() < 0.5}
    if op == "lazy":
        case["coef"] = True
    if op in ("new", "pcg", "multi"):
        case["mixed"] = rng.random() < 0.5
    if op == "multi":
        case["k"] = rng.choice([2, 3, 5, 8, 12, 16, 21, 32, 33, 48, 64])
    return case


# ------------------------------------------------------------------ inputs
_context = None


def _ctx() -> Context:
    """The program's one context, with its stream as torch sees it."""
    global _context
    if _context is None:
        _context = Context(0)
        _context.torch_stream = torch.cuda.ExternalStream(_context.stream())
    return _context


def _mesh(case, seed) -> Mesh:
    m = square_mesh(case["n"], 0.2, seed) if case["dim"] == 2 else cube_mesh(case["n"], 0.15, seed)
    m.cells = np.ascontiguousarray(m.cells, dtype=np.int32)
    return m


def _coef(case, mesh, seed):
    if not case["coef"]:
        return None
    rng = np.random.default_rng([seed, 1])
    if case["dim"] == 2 and case["degree"] == 2 and case["op"] == "pcg":
        # contrast 1e4, a smooth random field, as in the quadratic 2D benchmark workload
        field = contrast_coefficient(gaussian_field(case["n"], 0.05, rng), 1.0e4)
        return np.ascontiguousarray(np.repeat(field.reshape(-1), 2))
    return np.exp(rng.standard_normal(mesh.n_cell))


def _system(case, seed):
    """(space, K with zero Dirichlet data, M, b, boundary flags, mesh, coef): what a program holds before it solves."""
    ctx = _ctx()
    mesh = _mesh(case, seed)
    coef = _coef(case, mesh, seed)
    space = Space.numbered(ctx, mesh, case["degree"])
    _, mark, _ = space.dofs()
    K, M = assemble(space, *ACC[(case["dim"], case["degree"])], coef=coef)
    f = np.random.default_rng([seed, 2]).uniform(-1.0, 1.0, space.n_dof)
    b = M.vmult(f)
    _boundary(mark).apply(K, b)
    return space, K, M, b, mark, mesh, coef


def _boundary(mark) -> BoundaryConditionAdmin:
    bc = BoundaryConditionAdmin(types.SimpleNamespace(n_dof=mark.shape[0], dof_bmark=mark, dof_point=None))
    bc.add(1, 0.0)
    return bc


def _columns(seed, n, k):
    """n x k nodal data, columns independent."""
    return np.random.default_rng([seed, 3]).uniform(-1.0, 1.0, (n, k))


def _requests(case, seed):
    """Sizes evenly spaced in their logarithm, every second one with a coefficient of its own per cell."""
    ns = np.rint(np.geomspace(case["n_min"], case["n_max"], case["count"])).astype(int)
    return [request_workload(Request(i, int(n), i % 2 == 1, (seed % 1000003) * 100 + i)) for i, n in enumerate(ns)]


def prepare(case, seed):
    op = case["op"]
    ctx = _ctx()
    s = {"op": op}
    if op == "served":
        s["requests"] = _requests(case, seed)
        s["server"] = Server(workers=8, tol=TOL)
        return s
    if op == "system":
        s["mesh"], s["case"] = _mesh(case, seed), case
        n_dof = _counts(case)[0]
        s["u"] = np.random.default_rng([seed, 2]).uniform(-1.0, 1.0, n_dof)
        s["coef"] = _coef(case, s["mesh"], seed)
        return s
    if op == "assemble":
        s["mesh"] = _mesh(case, seed)
        s["space"] = Space.numbered(ctx, s["mesh"], case["degree"])
        s["coef"], s["acc"] = _coef(case, s["mesh"], seed), ACC[(case["dim"], case["degree"])]
        return s
    space, K, M, b, mark, _, _ = _system(case, seed)
    s["K"], s["b"] = K, b
    if op == "vmult":
        with torch.cuda.stream(ctx.torch_stream):
            s["x"] = torch.from_numpy(np.random.default_rng([seed, 5]).uniform(-1.0, 1.0, space.n_dof)).cuda()
        return s
    if op == "lazy":
        s["amg"] = AMGPreconditioner(K)
        s["values"] = torch.from_numpy(K.values() * (1.0 + 0.25 * np.sin(seed))).cuda()
        return s
    if op == "new":
        s["precision"] = MIXED if case["mixed"] else FP64
        return s
    s["amg"] = AMGSolver(K, precision=MIXED if case.get("mixed") else FP64)
    if op == "multi":
        rhs = _columns(seed, space.n_dof, case["k"])
        rhs[mark != 0] = 0.0
        with torch.cuda.stream(ctx.torch_stream):
            s["B"] = torch.from_numpy(rhs).cuda()
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ the pass
def _device_csr(K):
    """The matrix in AFEPack's layout, copied into device arrays of the caller's."""
    m, _, nnz = K.info()
    rp = torch.empty(m + 1, dtype=torch.int32, device="cuda")
    ci = torch.empty(nnz, dtype=torch.int32, device="cuda")
    va = torch.empty(nnz, dtype=torch.float64, device="cuda")
    N.call("afp_matrix_download", K.handle, N.ptr(rp), N.ptr(ci), N.ptr(va))
    return rp, ci, va


def run(s):
    op = s["op"]
    ctx = _ctx()
    if op == "served":
        tickets = [s["server"].submit(w) for w in s["requests"]]
        return [s["server"].wait(t)[0] for t in tickets]
    if op == "pcg":
        return s["amg"].pcg(s["b"], TOL)[0]
    if op == "new":
        return AMGSolver(s["K"], precision=s["precision"]).pcg(s["b"], TOL)[0]
    if op == "stationary":
        x = np.zeros_like(s["b"])
        s["amg"].solve(x, s["b"])
        return x
    if op == "system":
        case = s["case"]
        acc_s, acc_m = ACC[(case["dim"], case["degree"])]
        space = Space.numbered(ctx, s["mesh"], case["degree"])
        elem_dof, mark, point = space.dofs()
        K, M = assemble(space, acc_s, acc_m, s["coef"])
        f = L2Discretize(s["u"], space, acc_m)
        _boundary(mark).apply(K, f)
        rp, ci, va = K.download()
        return {"elem_dof": elem_dof, "mark": mark, "point": point, "rowptr": rp, "cols": ci, "stiff": va,
                "mass": M.values(), "f": f}
    with torch.cuda.stream(ctx.torch_stream):
        if op == "vmult":
            return s["K"].vmult(s["x"])
        if op == "assemble":
            K, M = assemble(s["space"], *s["acc"], coef=s["coef"])
            rp, ci, va = _device_csr(K)
            vm = torch.empty_like(va)
            N.call("afp_matrix_download", M.handle, None, None, N.ptr(vm))
            return {"rowptr": rp, "cols": ci, "stiff": va, "mass": vm}
        if op == "multi":
            return s["amg"].pcg_multi(s["B"], TOL)[0]
        if op == "lazy":
            s["K"].set_values(s["values"])
            s["amg"].reinit(s["K"])
            x = np.zeros_like(s["b"])
            s["amg"].vmult(x, s["b"])
            return x
    raise ValueError(op)


# ------------------------------------------------------------------ the least work
def _counts(case):
    """(DOFs, stored entries, cells, vertices) of the case's space."""
    n, d, p = case["n"], case["dim"], case["degree"]
    if d == 2:
        V, E, T = (n + 1) ** 2, 3 * n * n + 2 * n, 2 * n * n
        pairs = E if p == 1 else 3 * E + 6 * T
    else:
        V, E, T = (n + 1) ** 3, 3 * n * (n + 1) ** 2 + 3 * n * n * (n + 1) + n ** 3, 6 * n ** 3
        F = 12 * n ** 3 + 6 * n * n
        pairs = E if p == 1 else 3 * E + 6 * F + 3 * T
    dofs = V if p == 1 else V + E
    return dofs, dofs + 2 * pairs, T, V


def work(case):
    """Inputs read once, outputs written once; operations of one pass over them."""
    if case["op"] == "served":
        n = math.sqrt(case["n_min"] * case["n_max"])
        one = work({"op": "system", "dim": 2, "degree": 1, "n": n})
        return {"bytes": case["count"] * one["bytes"], "flops": case["count"] * one["flops"]}
    dofs, nnz, cells, verts = _counts(case)
    d, nd = case["dim"], {(2, 1): 3, (2, 2): 6, (3, 1): 4, (3, 2): 10}[(case["dim"], case["degree"])]
    matrix = 12 * nnz + 4 * (dofs + 1)
    mesh = 8 * d * verts + 4 * (d + 1) * cells
    if case["op"] in ("system", "assemble"):
        return {"bytes": mesh + 4 * nd * cells + matrix + 8 * nnz + 16 * dofs, "flops": 4 * cells * nd * nd * d}
    k = case.get("k", 1)
    return {"bytes": matrix + 16 * dofs * k, "flops": 2 * nnz * k}


# ------------------------------------------------------------------ the same in 64 bits, plainly
_EDGES = {2: ((1, 2), (0, 2), (0, 1)), 3: ((0, 1), (0, 2), (0, 3), (2, 3), (1, 3), (1, 2))}


def _numbering(mesh, degree):
    """DOF of every template node, numbered as the cells first meet them (vertices, then edges, of each cell)."""
    cells = mesh.cells.astype(np.int64)
    keys = cells
    if degree == 2:
        ends = cells[:, np.array(_EDGES[mesh.dim])]
        keys = np.concatenate([cells, mesh.n_vertex * (1 + ends.min(2)) + ends.max(2)], axis=1)
    _, first, back = np.unique(keys.reshape(-1), return_index=True, return_inverse=True)
    rank = np.empty(first.size, dtype=np.int64)
    rank[np.argsort(first)] = np.arange(first.size)
    dof = rank[back.reshape(-1)].reshape(keys.shape)
    mark = np.zeros(first.size, dtype=bool)
    vm = mesh.bmask.astype(np.int64)
    on = vm[cells] != 0
    if degree == 2:
        on = np.concatenate([on, (vm[ends[:, :, 0]] & vm[ends[:, :, 1]]) != 0], axis=1)
    mark[dof[on]] = True
    return dof, mark


def _element_matrices(mesh, degree, coef):
    """Stiffness and mass matrix of every cell: integrals of polynomials in barycentric coordinates."""
    d = mesh.dim
    v = torch.from_numpy(mesh.coords).cuda()[torch.from_numpy(mesh.cells.astype(np.int64)).cuda()]
    J = (v[:, 1:] - v[:, :1]).transpose(1, 2)
    vol = torch.linalg.det(J) / math.factorial(d)
    inv = torch.linalg.inv(J)
    G = torch.cat([-inv.sum(1, keepdim=True), inv], 1)  # gradients of the barycentric coordinates
    m = d + 1

    def integral(idx):  # of a product of barycentric coordinates, over the volume
        a = np.bincount(np.array(idx), minlength=m)
        return math.factorial(d) * math.prod(math.factorial(int(t)) for t in a) / math.factorial(d + len(idx))

    nodes = m if degree == 1 else m + len(_EDGES[d])
    if degree == 1:
        D, B = np.zeros((nodes, m, 1)), np.eye(m)
        D[np.arange(m), np.arange(m), 0] = 1.0
        W1 = np.ones((1, 1))
        mass = np.array([[integral((i, j)) for j in range(m)] for i in range(m)])
    else:
        D, B = np.zeros((nodes, m, m)), np.zeros((nodes, m, m))
        for i in range(m):
            D[i, i, :] = -1.0
            D[i, i, i] = 3.0
            B[i, i, :] = -1.0
            B[i, i, i] = 1.0
        for e, (a, b) in enumerate(_EDGES[d]):
            D[m + e, a, b] = D[m + e, b, a] = 4.0
            B[m + e, a, b] = 4.0
        W1 = np.array([[integral((i, j)) for j in range(m)] for i in range(m)])
        W2 = np.array([[[[integral((i, j, k, l)) for l in range(m)] for k in range(m)] for j in range(m)] for i in range(m)])
        mass = np.einsum("imn,jpq,mnpq->ij", B, B, W2)
    S = torch.from_numpy(np.einsum("ikm,jln,mn->ijkl", D, D, W1)).cuda().reshape(nodes * nodes, m * m)
    scale = vol if coef is None else vol * torch.from_numpy(coef).cuda()
    K = (torch.einsum("ekd,eld->ekl", G, G).reshape(-1, m * m) @ S.T) * scale[:, None]
    return K.reshape(-1, nodes, nodes), vol[:, None, None] * torch.from_numpy(mass).cuda()


def _csr(dof, n, *elements):
    """Rows as [diagonal, ascending others]: (rowptr, cols, values of each)."""
    t = torch.from_numpy(dof).cuda()
    r, c = t[:, :, None].expand(-1, -1, t.shape[1]), t[:, None, :].expand(-1, t.shape[1], -1)
    key = (r * (n + 1) + torch.where(r == c, torch.zeros_like(c), c + 1)).reshape(-1)
    keys, back = torch.unique(key, return_inverse=True)
    rows, cols = keys // (n + 1), keys % (n + 1) - 1
    cols = torch.where(cols < 0, rows, cols)
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return rp, rows, cols, [torch.zeros(keys.numel(), dtype=torch.float64, device="cuda").index_add_(0, back, e.reshape(-1)) for e in elements]


class _Exact:
    """The case's matrices in 64 bits, from the mesh and the coefficient alone."""

    def __init__(self, mesh, degree, coef, dirichlet=True):
        self.dof, self.mark = _numbering(mesh, degree)
        self.n = n = self.mark.shape[0]
        self.rp, self.rows, self.cols, (k, self.m) = _csr(self.dof, n, *_element_matrices(mesh, degree, coef))
        self.free = torch.from_numpy(~self.mark).cuda()
        off = (self.rows != self.cols) & ~(self.free[self.rows] & self.free[self.cols])
        self.k = torch.where(off, torch.zeros_like(k), k) if dirichlet else k

    def matrix(self, vals):
        return torch.sparse_csr_tensor(*self.sorted_rows(vals), size=(self.n, self.n), check_invariants=False)

    def sorted_rows(self, vals):
        order = torch.argsort(self.rows * self.n + self.cols)
        return self.rp, self.cols[order], vals[order]

    def mass_times(self, f):
        y = self.matrix(self.m) @ torch.from_numpy(f).cuda().reshape(self.n, -1)
        return torch.where(self.free[:, None], y, torch.zeros_like(y))

    def solve(self, B):
        """K X = B by conjugate gradients with the diagonal, to the rounding of 64 bits."""
        A = self.matrix(self.k)
        w = (1.0 / self.k[self.rp[:-1]])[:, None]
        X, R = torch.zeros_like(B), B.clone()
        Z = w * R
        P, rz = Z.clone(), (R * Z).sum(0)
        stop = 1e-15 * B.norm(dim=0)
        for it in range(12000):
            Q = A @ P
            live = (R.norm(dim=0) > stop).double() if it % 25 == 0 else live
            if it % 25 == 0 and not bool(live.any()):
                break
            a = live * rz / (P * Q).sum(0).clamp_min(1e-300)
            X += a * P
            R -= a * Q
            Z = w * R
            new = (R * Z).sum(0)
            P = Z + (new / rz.clamp_min(1e-300)) * P
            rz = new
        return X


def exact(case, seed):
    op = case["op"]
    if op in ("lazy", "stationary"):
        return None  # a fixed number of cycles, not run to convergence: no value of their own
    if op == "served":
        out = []
        for w in _requests(case, seed):
            e = _Exact(w.mesh, 1, w.coef)
            out.append(e.solve(e.mass_times(w.f)).reshape(-1))
        return out
    mesh = _mesh(case, seed)
    e = _Exact(mesh, case["degree"], _coef(case, mesh, seed), dirichlet=op != "assemble")
    if op in ("assemble", "system"):
        out = {"rowptr": None, "cols": None, "stiff": e.k, "mass": e.m}
        if op == "system":
            u = np.random.default_rng([seed, 2]).uniform(-1.0, 1.0, e.n)
            out |= {"elem_dof": None, "mark": None, "point": None, "f": e.mass_times(u).reshape(-1)}
        return out
    if op == "vmult":
        x = torch.from_numpy(np.random.default_rng([seed, 5]).uniform(-1.0, 1.0, e.n)).cuda()
        return (e.matrix(e.k) @ x[:, None]).reshape(-1)
    if op == "multi":
        rhs = _columns(seed, e.n, case["k"])
        rhs[e.mark] = 0.0
        return e.solve(torch.from_numpy(rhs).cuda())
    f = np.random.default_rng([seed, 2]).uniform(-1.0, 1.0, e.n)
    return e.solve(e.mass_times(f)).reshape(-1)
