"""Workloads of the assembly engine, timed through its public Python API.

Every case is something a program that uses ``cudolfinx`` does in its inner
loop: assemble a matrix into its pattern, assemble a whole system, assemble a
right-hand side, assemble many coefficient instances or many meshes at once,
solve.  Meshes are the unit cube of ``fem.create_unit_cube`` (n^3 hexes x 6
tets), with its vertices moved and, for some cases, in another numbering.

``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges;
``prepare`` makes what the program holds before the call (mesh, spaces, forms,
matrix, packed BCs), ``run`` is one pass, ``work`` its least bytes and
operations and ``exact`` its result from plain 64-bit torch and numpy.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(1, os.path.abspath("cuda-dolfinx_b200"))

import cudolfinx as cufem  # noqa: E402
from cudolfinx import fem  # noqa: E402

EDGES = ((2, 3), (1, 3), (1, 2), (0, 3), (0, 2), (0, 1))
DEGREE = {"p1": 1, "p2": 2, "p3": 3, "vp2": 2}

# largest n of each kind of call (a drawn case stays at or below the listed ones)
LARGEST = {"p1": 97, "p2": 96, "p3": 36, "vp2": 44}


def listed():
    return [
        # one time step of a small model: matrix and right-hand side by the
        # reference example's separate calls; launches and host calls count
        _case("p1_system_n12", op="system", element="p1", n=12, coef="const", calls="separate"),
        # the same at a size where the kernels begin to show, P2 with a P1 field
        _case("p2_system_n20", op="system", element="p2", n=20, coef="p1", calls="fused"),
        # a P1 matrix on a mesh numbered as a mesh generator's reordering leaves it
        _case("p1_matrix_n45_reordered", op="matrix", element="p1", n=45, coef="p1", order="reordered"),
        # a large P1 matrix with a cellwise coefficient that is already on the device
        _case("p1_matrix_n97", op="matrix", element="p1", n=97, coef="dg0"),
        # the headline: P2 Poisson, k a P1 field uploaded on every call
        _case("p2_matrix_n96", op="matrix", element="p2", n=96, coef="p1"),
        # its right-hand side (load, lifting, set_bc), a size down
        _case("p2_rhs_n61", op="rhs", element="p2", n=61, coef="p1", calls="fused"),
        # elasticity, FP32 element tensors into FP64 values
        _case("vp2_matrix_n44_fp32", op="matrix", element="vp2", n=44, coef="dg0", precision="fp32"),
        # cubic elements
        _case("p3_matrix_n36", op="matrix", element="p3", n=36, coef="dg0"),
        # many coefficient samples on one mesh (uncertainty quantification)
        _case("p1_batch_n33x56", op="batch", element="p1", n=33, coef="dg0", count=56),
        # many meshes of uneven size in one captured graph
        _case("graph_14_meshes", op="graph", element="p1", n=26, coef="dg0", count=14, precision="fp32"),
        # assemble-and-solve services spend most of a request here
        _case("p2_solve_n22", op="solve", element="p2", n=22, coef="p1"),
        # any other form: an FFCx tabulate_tensor body compiled at run time
        _case("ffcx_p2_matrix_n37", op="ffcx", element="p2", n=37, coef="p1"),
    ]


def _case(name=None, **kw):
    c = {"op": "matrix", "element": "p1", "n": 8, "coef": "const", "precision": "fp64", "order": "natural",
         "calls": "fused", "count": 1}
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(("system", "system", "matrix", "matrix", "matrix", "matrix", "rhs", "batch", "graph", "solve",
                     "ffcx"))
    order = rng.choice(("natural", "natural", "reordered"))
    calls = rng.choice(("separate", "fused"))
    if op == "batch":
        el = rng.choice(("p1", "p2"))
        return _case(op=op, element=el, n=size(8, 33 if el == "p1" else 20), coef="dg0",
                     count=rng.randint(5, 56), order=order)
    if op == "graph":
        return _case(op=op, n=size(10, 26), coef="dg0", count=rng.randint(3, 14),
                     precision=rng.choice(("fp32", "fp64")))
    if op == "solve":
        return _case(op=op, element=rng.choice(("p1", "p2")), n=size(6, 22), coef=rng.choice(("const", "p1")))
    if op == "ffcx":
        el = rng.choice(("p1", "p2"))
        return _case(op=op, element=el, n=size(6, 37), coef="p1", order=order)
    el = rng.choice(("p1", "p1", "p2", "p2", "p3", "vp2"))
    coef = {"p1": ("const", "dg0", "p1"), "p2": ("const", "dg0", "p1"), "p3": ("const", "dg0"), "vp2": ("dg0",)}[el]
    precision = "fp64" if el == "p1" else rng.choice(("fp64", "fp32"))
    return _case(op=op, element=el, n=size(6, LARGEST[el] // (2 if op == "system" else 1)), coef=rng.choice(coef),
                 precision=precision, order=order, calls=calls)


# ---------------------------------------------------------------------------
# meshes, dofmaps and inputs (plain numpy / torch)
# ---------------------------------------------------------------------------
def _spread(v):
    """Bits of v three apart (Morton code of one coordinate)."""
    r = np.zeros_like(v)
    for b in range(10):
        r |= ((v >> b) & 1) << (3 * b)
    return r


def _mesh(n, order, element, seed):
    """Vertices, cells, each vertex's grid index and whether vertices keep the grid's numbering."""
    rng = np.random.default_rng([seed, 1])
    n1 = n + 1
    v = np.arange(n1 ** 3, dtype=np.int32)
    idx = np.stack([v % n1, (v // n1) % n1, v // (n1 * n1)], axis=1)
    # vertices up to 0.2 h off the grid, except normal to the faces of the cube
    d = rng.uniform(-0.2 / n, 0.2 / n, size=idx.shape)
    d[(idx == 0) | (idx == n)] = 0.0
    x = idx / float(n) + d
    h = np.arange(n, dtype=np.int32)
    v0 = (h[:, None, None] * (n1 * n1) + h[None, :, None] * n1 + h[None, None, :]).ravel()
    o = np.array([0, 1, n1, n1 + 1, n1 * n1, n1 * n1 + 1, n1 * n1 + n1, n1 * n1 + n1 + 1], dtype=np.int32)
    tets = np.array([[0, 1, 3, 7], [0, 1, 7, 5], [0, 5, 7, 4], [0, 3, 2, 7], [0, 6, 4, 7], [0, 2, 6, 7]])
    cells = (v0[:, None, None] + o[tets][None]).reshape(-1, 4)
    if order == "reordered":
        # cells along a space-filling curve, each with its vertices in some order of its own
        q = idx[cells].sum(axis=1)
        key = _spread(q[:, 0]) | (_spread(q[:, 1]) << 1) | (_spread(q[:, 2]) << 2)
        cells = cells[np.argsort(key, kind="stable")]
        turn = rng.permuted(np.tile(np.arange(4), (len(cells), 1)), axis=1)
        cells = np.take_along_axis(cells, turn, axis=1)
        if element == "p1":
            # vertices too (P2 and P3 spaces are numbered from the grid's vertices)
            key = _spread(idx[:, 0]) | (_spread(idx[:, 1]) << 1) | (_spread(idx[:, 2]) << 2)
            old = np.argsort(key, kind="stable")
            new = np.empty_like(old)
            new[old] = np.arange(len(old))
            x, idx, cells = x[old], idx[old], new[cells]
    return np.ascontiguousarray(x), np.ascontiguousarray(cells, dtype=np.int32), idx


def _weights(degree):
    """Barycentric coordinates of the element's nodes, times the degree (basix order, equispaced)."""
    unit = np.eye(4, dtype=np.int64)
    w = [degree * unit[a] for a in range(4)]
    for a, b in EDGES:
        w += [(degree - s) * unit[a] + s * unit[b] for s in range(1, degree)]
    if degree == 3:
        w += [1 - unit[f] for f in range(4)]
    return np.array(w)


def _dofs(cells, idx, n, degree):
    """Cell dofs of degree 1..3 by the numbering of fem.FunctionSpace."""
    if degree == 1:
        return torch.from_numpy(cells).long()
    m = degree * n + 1
    g = torch.from_numpy(idx).long()[torch.from_numpy(cells).long()]
    p = torch.einsum("lv,cvd->cld", torch.from_numpy(_weights(degree)), g)
    return (p[..., 2] * m + p[..., 1]) * m + p[..., 0]


def _grid_points(idx, n, degree):
    """Grid index [nodes, 3] of every node."""
    if degree == 1:
        return idx
    m = degree * n + 1
    k = np.arange(m ** 3)
    return np.stack([k % m, (k // m) % m, k // (m * m)], axis=1)


def _boundary(idx, n, degree, bs):
    """Scalar boundary dofs and boundary values g = x + y + z (component c: plus c) on all scalar dofs."""
    p = _grid_points(idx, n, degree)
    nodes = np.nonzero(((p == 0) | (p == degree * n)).any(axis=1))[0]
    g = p.sum(axis=1) / float(degree * n)
    if bs > 1:
        nodes = (nodes[:, None] * bs + np.arange(bs)).ravel()
        g = (g[:, None] + np.arange(bs)).ravel()
    return nodes.astype(np.int32), g


def _fields(case, seed, ncells, nverts):
    """The case's coefficient arrays."""
    rng = np.random.default_rng([seed, 2])
    f = {}
    if case["element"] == "vp2":
        f["lam"], f["mu"] = rng.uniform(0.5, 2.0, ncells), rng.uniform(0.2, 1.0, ncells)
        f["load"] = rng.uniform(-1.0, 1.0, 3 * ncells)
        return f
    if case["coef"] == "dg0":
        f["k"] = 10.0 ** rng.uniform(-2.0, 2.0, ncells)
    elif case["coef"] == "p1":
        f["k"] = np.exp(rng.standard_normal(nverts))
    if case["op"] in ("system", "rhs", "solve"):
        f["load"] = rng.uniform(-1.0, 1.0, nverts if case["element"] == "p1" else ncells)
    return f


def _pinned(V, values):
    """A Function whose host array is page-locked."""
    f = fem.Function(V)
    t = torch.empty(len(values), dtype=torch.float64, pin_memory=True)
    f.x.array = t.numpy()
    f.x.array[:] = values
    f.keep = t
    return f


def _on_device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


class _State:
    """What a program keeps between calls; its meshes' device caches go with it."""

    def __init__(self, op):
        self.op = op
        self.meshes = []

    def __del__(self):
        for m in self.meshes:
            cufem.release_caches(m)


def _bilinear(case, V, mesh, f):
    pr = case["precision"]
    if case["element"] == "vp2":
        return fem.elasticity(V, _on_device(f["lam"]), _on_device(f["mu"]), precision=pr)
    if case["coef"] == "const":
        k = 1.5
    elif case["coef"] == "dg0":
        k = _on_device(f["k"])
    else:
        k = _pinned(fem.functionspace(mesh, ("P", 1)), f["k"])
    return fem.stiffness(V, k, precision=pr)


def _space(mesh, element):
    return fem.functionspace(mesh, ("P", DEGREE[element], (3,)) if element == "vp2" else ("P", DEGREE[element]))


def prepare(case, seed):
    s = _State(case["op"])
    s.asm = cufem.CUDAAssembler()
    if case["op"] == "graph":
        items = []
        for el, n, sd in _graph_items(case, seed):
            # (FP32 element tensors are offered from degree 2 on)
            c = _case(op="matrix", element=el, n=n, coef="dg0",
                      precision=case["precision"] if el == "p2" else "fp64")
            a, A, col, _, mesh, _ = _setup(s.asm, c, sd)
            s.meshes.append(mesh)
            items.append((a, A, col))
        s.items = items
        s.graph = cufem.AssemblyGraph(items).capture()
        return s
    s.a, s.A, s.col, s.L, mesh, f = _setup(s.asm, case, seed)
    s.meshes.append(mesh)
    s.fused = case["calls"] == "fused"
    if case["op"] == "batch":
        s.ks = _batch_fields(case, seed, mesh.num_cells)
        s.mats = [s.A] + [cufem.CUDAMatrix(s.A._ctx, s.A.sparsity) for _ in range(case["count"] - 1)]
    if s.L is not None:
        s.b = s.asm.create_vector(s.L)
    if case["op"] == "solve":
        s.asm.assemble_matrix(s.a, s.A, bcs=s.col)
        s.asm.assemble_rhs(s.L, s.a, s.col, vec=s.b)
    return s


def _graph_items(case, seed):
    """(element, n, seed) of the meshes: P1 and P2 in turn, n from 8 to the case's n."""
    rng = np.random.default_rng([case["n"], case["count"]])
    return [("p1" if q % 2 == 0 else "p2", int(rng.integers(8, case["n"] + 1)) if q > 1 else case["n"],
             seed * 100 + q) for q in range(case["count"])]


def _batch_fields(case, seed, ncells):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7 + 5)
    e = torch.rand((case["count"], ncells), generator=g, dtype=torch.float64, device="cuda")
    return 10.0 ** (4.0 * e - 2.0)


def _setup(asm, case, seed):
    n, el = case["n"], case["element"]
    x, cells, idx = _mesh(n, case["order"], el, seed)
    degree = DEGREE[el]
    grid = n if degree > 1 or case["order"] == "natural" else None
    mesh = fem.Mesh(x, cells, grid_n=grid)
    V = _space(mesh, el)
    f = _fields(case, seed, len(cells), len(x))
    if case["op"] == "ffcx":
        k = _pinned(fem.functionspace(mesh, ("P", 1)), f["k"])
        body = _ffcx_body(degree)
        a = cufem.form(fem.FFCxForm([fem.FFCxIntegral("cell", "tabulate_tensor_integral_reaction_diffusion_p%d"
                                                      % degree, body)], [V, V], [k], [0.75]))
    else:
        a = cufem.form(_bilinear(case, V, mesh, f))
    L = None
    if "load" in f:
        w = f["load"]
        if case["op"] in ("system", "rhs", "solve"):
            L = cufem.form(fem.load(V, _pinned(V, w) if el == "p1" else _on_device(w)))
    nodes, g = _boundary(idx, n, degree, V.bs)
    col = asm.pack_bcs([fem.dirichletbc(fem.Function(V, g), nodes)])
    A = None if case["op"] == "rhs" else asm.create_matrix(a)
    return a, A, col, L, mesh, f


def run(s):
    asm = s.asm
    if s.op in ("matrix", "ffcx"):
        asm.assemble_matrix(s.a, s.A, bcs=s.col)
        return s.A.values
    if s.op in ("system", "rhs"):
        if s.op == "system":
            asm.assemble_matrix(s.a, s.A, bcs=s.col)
        if s.fused:
            asm.assemble_rhs(s.L, s.a, s.col, vec=s.b)
        else:
            asm.assemble_vector(s.L, s.b)
            asm.apply_lifting(s.b, [s.a], [s.col])
            asm.set_bc(s.b, s.col, s.a.function_spaces[0])
        return s.b.vector if s.op == "rhs" else (s.A.values, s.b.vector)
    if s.op == "batch":
        asm.assemble_matrix_batch(s.a, s.ks, s.mats, bcs=s.col)
        return [m.values for m in s.mats]
    if s.op == "graph":
        s.graph.replay()
        return [A.values for _, A, _ in s.items]
    x, _, _ = asm.solve(s.A, s.b, rtol=1e-11)
    return x.vector


# ---------------------------------------------------------------------------
# least work
# ---------------------------------------------------------------------------
def _counts(case):
    """cells, vertices, scalar rows, nonzeros of the case's space."""
    n, el = case["n"], case["element"]
    C, N = 6 * n ** 3, (n + 1) ** 3
    E = 3 * n * (n + 1) ** 2 + 3 * n * n * (n + 1) + n ** 3
    F = (4 * C + 12 * n * n) // 2
    d = DEGREE[el]
    nnz = {1: N + 2 * E, 2: N + 7 * E + 12 * F + 6 * C, 3: N + 14 * E + 55 * F + 92 * C}[d]
    rows = (d * n + 1) ** 3
    return (C, N, 3 * rows, 9 * nnz) if el == "vp2" else (C, N, rows, nnz)


def work(case):
    if case["op"] == "graph":
        each = [work(_case(op="matrix", element=el, n=n, coef="dg0")) for el, n, _ in _graph_items(case, 0)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    C, N, rows, nnz = _counts(case)
    el, op = case["element"], case["op"]
    k = {"p1": 4, "p2": 10, "p3": 20, "vp2": 10}[el]
    bs = 3 if el == "vp2" else 1
    terms = {"p1": 3, "p2": 6, "p3": 6, "vp2": 9}[el]  # products of one entry of the element tensor
    if case["coef"] == "p1" and el == "p2":
        terms = 12
    coef = {"const": 0, "dg0": 8 * C * (2 if el == "vp2" else 1), "p1": 8 * N + 16 * C}[case["coef"]]
    mesh = 24 * N + 16 * C + (0 if el == "p1" else 4 * k * C) + rows  # coordinates, cells, dofmap, BC markers
    tensor = 2.0 * terms * bs * k * (bs * k + 1) / 2 * C
    matrix = {"bytes": 8 * nnz + mesh + coef, "flops": 60 * C + tensor}
    vector = {"bytes": 8 * rows + 9 * rows + mesh + coef + 8 * (N if el == "p1" else C * bs),
              "flops": 40.0 * C + 2 * k * bs * C}
    if op in ("matrix", "ffcx"):
        return matrix
    if op == "rhs":
        return vector
    if op == "system":
        return {"bytes": matrix["bytes"] + 17 * rows + 8 * (N if el == "p1" else C * bs),
                "flops": matrix["flops"] + 2 * k * bs * C}
    if op == "batch":
        return {"bytes": mesh + case["count"] * (8 * nnz + 8 * C), "flops": 60 * C + case["count"] * 2.0 * k * k * C}
    # solve: the matrix and the vectors once per iteration; Jacobi-PCG needs about 9 n iterations for P2 (5 n for
    # P1) at rtol 1e-11
    its = (9 if el == "p2" else 5) * case["n"]
    return {"bytes": its * (12.0 * nnz + 4 * rows + 96 * rows), "flops": its * (2.0 * nnz + 12 * rows)}


# ---------------------------------------------------------------------------
# the same results in 64 bits by plain torch and numpy
# ---------------------------------------------------------------------------
def _rule(m):
    """m^3-point rule on the reference tetrahedron, exact to degree 2m - 1 (Gauss-Jacobi on the collapsed cube)."""
    def jacobi(a):
        # points and weights on [0, 1] for the weight (1 - t)^a, from the three-term recurrence
        k = np.arange(m, dtype=float)
        ab = np.zeros(m)
        for i in range(m):
            ab[i] = -a * a / ((2 * i + a) * (2 * i + a + 2)) if a > 0 else 0.0
        k = np.arange(1, m, dtype=float)
        off = 2.0 / (2 * k + a) * np.sqrt(k * (k + a) * k * (k + a) / ((2 * k + a + 1) * (2 * k + a - 1)))
        t, v = np.linalg.eigh(np.diag(ab) + np.diag(off, 1) + np.diag(off, -1))
        return (1 + t) / 2, v[0] ** 2 / (a + 1)

    (t0, w0), (t1, w1), (t2, w2) = jacobi(0), jacobi(1), jacobi(2)
    pts, wts = [], []
    for z, wz in zip(t2, w2):
        for y, wy in zip(t1, w1):
            for x, wx in zip(t0, w0):
                pts.append([x * (1 - y) * (1 - z), y * (1 - z), z])
                wts.append(wx * wy * wz)
    return np.array(pts), np.array(wts)


def _tabulate(degree, pts):
    """Basis values [q, k] and reference gradients [q, 3, k] of the equispaced element."""
    e = [(i, j, k) for i in range(degree + 1) for j in range(degree + 1 - i) for k in range(degree + 1 - i - j)]

    def mono(X):
        return np.stack([X[:, 0] ** i * X[:, 1] ** j * X[:, 2] ** k for i, j, k in e], axis=1)

    def dmono(X, d):
        out = []
        for p in e:
            if p[d] == 0:
                out.append(np.zeros(len(X)))
                continue
            r = list(p)
            r[d] -= 1
            out.append(p[d] * X[:, 0] ** r[0] * X[:, 1] ** r[1] * X[:, 2] ** r[2])
        return np.stack(out, axis=1)

    nodes = _weights(degree)[:, 1:] / float(degree)
    c = np.linalg.inv(mono(nodes))
    return mono(pts) @ c, np.stack([dmono(pts, d) @ c for d in range(3)], axis=1)


_GRID_M = 4  # exact to degree 7: P3 stiffness (4), P2 with a P1 field (3), P3 load


def _geometry(x, cells):
    """K = J^-1 and |det J| of every cell."""
    X = x[cells]
    J = (X[:, 1:] - X[:, :1]).transpose(1, 2)
    return torch.linalg.inv(J), torch.linalg.det(J).abs()


def _element_matrices(case, f, x, cells, verts):
    """[C, k*bs, k*bs] element matrices; verts: the P1 field's cell dofs."""
    el, dev = case["element"], x.device
    degree = DEGREE[el]
    K, det = _geometry(x, cells)
    pts, wts = _rule(2 if case["op"] == "ffcx" else _GRID_M)
    phi, dphi = _tabulate(degree, pts)
    lam = np.column_stack([1 - pts.sum(axis=1), pts])
    w, phi, dphi, lam = (torch.from_numpy(v).to(dev) for v in (wts, phi, dphi, lam))
    if el == "vp2":
        R = torch.einsum("q,qsi,qtj->stij", w, dphi, dphi)
        KK = K @ K.transpose(1, 2)
        eye = torch.eye(3, dtype=torch.float64, device=dev)
        W = (f["lam"] * det)[:, None, None, None, None] * torch.einsum("cpa,cqb->cabpq", K, K)
        W = W + (f["mu"] * det)[:, None, None, None, None] * (torch.einsum("ab,cpq->cabpq", eye, KK)
                                                              + torch.einsum("cpb,cqa->cabpq", K, K))
        A = torch.einsum("cabpq,pqij->ciajb", W, R)
        return A.reshape(len(cells), 30, 30)
    G = det[:, None, None] * (K @ K.transpose(1, 2))
    if case["coef"] == "p1":
        R = torch.einsum("q,qm,qsi,qtj->mstij", w, lam, dphi, dphi)
        kG = f["k"][verts][:, :, None, None] * G[:, None]
        k = phi.shape[1]
        A = (kG.reshape(-1, 36) @ R.reshape(36, k * k)).reshape(-1, k, k)
    else:
        R = torch.einsum("q,qsi,qtj->stij", w, dphi, dphi)
        s = f["k"] if case["coef"] == "dg0" else torch.full((len(cells),), 1.5, dtype=torch.float64, device=dev)
        k = phi.shape[1]
        A = ((s[:, None, None] * G).reshape(-1, 9) @ R.reshape(9, k * k)).reshape(-1, k, k)
    if case["op"] == "ffcx":
        A = A + (0.75 * det)[:, None, None] * torch.einsum("q,qi,qj->ij", w, phi, phi)
    return A


def _element_vectors(case, f, x, cells):
    el = case["element"]
    _, det = _geometry(x, cells)
    pts, wts = _rule(_GRID_M)
    phi, _ = _tabulate(DEGREE[el], pts)
    w, phi = torch.from_numpy(wts).to(x.device), torch.from_numpy(phi).to(x.device)
    if el == "p1":
        return det[:, None] * (f["load"][cells] @ torch.einsum("q,qi,qj->ij", w, phi, phi))
    b = w @ phi
    if el == "vp2":
        return (det[:, None, None] * b[None, :, None] * f["load"].reshape(-1, 1, 3)).reshape(len(cells), -1)
    return (det * f["load"])[:, None] * b[None]


def _chunks(total, size):
    return [slice(i, min(total, i + size)) for i in range(0, total, size)]


def _exact_parts(case, seed, fields=None):
    """Device copies of the case's arrays."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, cells, idx = _mesh(case["n"], case["order"], case["element"], seed)
    f = _fields(case, seed, len(cells), len(x)) if fields is None else fields
    degree = DEGREE[case["element"]]
    bs = 3 if case["element"] == "vp2" else 1
    dofs = _dofs(cells, idx, case["n"], degree).to(dev)
    nodes, g = _boundary(idx, case["n"], degree, bs)
    nn = len(x) if degree == 1 else (degree * case["n"] + 1) ** 3
    f = {k: (torch.from_numpy(v) if isinstance(v, np.ndarray) else v).to(dev) for k, v in f.items()}
    mark = torch.zeros(nn * bs, dtype=torch.bool, device=dev)
    mark[torch.from_numpy(nodes).long().to(dev)] = True
    return {"x": torch.from_numpy(x).to(dev), "cells": torch.from_numpy(cells).long().to(dev), "f": f, "bs": bs,
            "dofs": dofs, "mark": mark, "g": torch.from_numpy(np.asarray(g, dtype=np.float64)).to(dev), "nn": nn}


def _slice_fields(case, f, sl):
    cellwise = {"lam", "mu"} | ({"k"} if case["coef"] == "dg0" else set())
    return {k: v[sl] if k in cellwise else v for k, v in f.items()}


def _pattern(p):
    """Block rows, block columns of the pattern and the place of every cell coupling in it."""
    d, nn = p["dofs"], p["nn"]
    k = d.shape[1]
    keys = (d[:, :, None] * nn + d[:, None, :]).reshape(-1)
    u, inv = torch.unique(keys, sorted=True, return_inverse=True)
    del keys
    return u // nn, u % nn, inv.reshape(-1, k * k)


def _exact_matrix(case, p, pattern=None):
    rows, cols, inv = _pattern(p) if pattern is None else pattern
    bs, mark, nb = p["bs"], p["mark"], len(rows)
    C, k = p["dofs"].shape
    vals = torch.zeros((nb, bs * bs), dtype=torch.float64, device=p["x"].device)
    for sl in _chunks(C, 200_000):
        E = _element_matrices(case, _slice_fields(case, p["f"], sl), p["x"], p["cells"][sl], p["cells"][sl])
        if bs == 1:
            vals.view(-1).index_add_(0, inv[sl].reshape(-1), E.reshape(-1))
        else:
            E = E.reshape(-1, k, bs, k, bs).permute(0, 1, 3, 2, 4).reshape(-1, bs * bs)
            vals.index_add_(0, inv[sl].reshape(-1), E)
    comp = torch.arange(bs, device=vals.device)
    r = rows[:, None, None] * bs + comp[None, :, None]
    c = cols[:, None, None] * bs + comp[None, None, :]
    v = vals.view(nb, bs, bs)
    v[mark[r] | mark[c]] = 0.0
    v[(r == c) & mark[r]] = 1.0
    if bs == 1:
        return v.reshape(-1)
    # scalar CSR order: row (I, a) lists its block columns' components in turn
    start = torch.searchsorted(rows, torch.arange(p["nn"] + 1, device=rows.device))
    length = (start[1:] - start[:-1])[rows]
    at = torch.arange(nb, device=rows.device) - start[rows]
    slot = (bs * bs * start[rows])[:, None, None] + comp[None, :, None] * (bs * length)[:, None, None] \
        + (bs * at)[:, None, None] + comp[None, None, :]
    out = torch.empty(nb * bs * bs, dtype=torch.float64, device=rows.device)
    out[slot.reshape(-1)] = v.reshape(-1)
    return out


def _exact_rhs(case, p):
    bs, mark, g = p["bs"], p["mark"], p["g"]
    C, k = p["dofs"].shape
    sd = (p["dofs"][:, :, None] * bs + torch.arange(bs, device=mark.device)).reshape(C, -1)
    b = torch.zeros(p["nn"] * bs, dtype=torch.float64, device=mark.device)
    f = p["f"]
    g0 = torch.where(mark, g, torch.zeros_like(g))
    for sl in _chunks(C, 200_000):
        fs = _slice_fields(case, f, sl)
        if case["element"] != "p1":
            fs["load"] = f["load"].reshape(C, -1)[sl].reshape(-1)
        b.index_add_(0, sd[sl].reshape(-1), _element_vectors(case, fs, p["x"], p["cells"][sl]).reshape(-1))
        touched = mark[sd[sl]].any(dim=1).nonzero()[:, 0] + sl.start
        if len(touched):
            ft = {q: (f[q][touched] if q in ("lam", "mu") or (q == "k" and case["coef"] == "dg0") else f[q]) for q in f}
            E = _element_matrices(case, ft, p["x"], p["cells"][touched], p["cells"][touched])
            b.index_add_(0, sd[touched].reshape(-1), -(E @ g0[sd[touched]][:, :, None]).reshape(-1))
    return torch.where(mark, g, b)


def exact(case, seed):
    op = case["op"]
    if op == "graph":
        return [_exact_matrix(c, _exact_parts(c, sd))
                for c, sd in ((_case(op="matrix", element=el, n=n, coef="dg0"), sd)
                              for el, n, sd in _graph_items(case, seed))]
    p = _exact_parts(case, seed)
    if op in ("matrix", "ffcx"):
        return _exact_matrix(case, p)
    if op == "system":
        return _exact_matrix(case, p), _exact_rhs(case, p)
    if op == "rhs":
        return _exact_rhs(case, p)
    if op == "batch":
        if not torch.cuda.is_available():
            return None
        pattern, out = _pattern(p), []
        for k in _batch_fields(case, seed, len(p["cells"])):
            p["f"] = {"k": k}
            out.append(_exact_matrix(case, p, pattern))
        return out
    # solve: conjugate gradients on the exact system, to rounding
    pattern = _pattern(p)
    vals, b = _exact_matrix(case, p, pattern), _exact_rhs(case, p)
    ptr = torch.searchsorted(pattern[0], torch.arange(p["nn"] + 1, device=b.device))
    A = torch.sparse_csr_tensor(ptr, pattern[1], vals, size=(p["nn"], p["nn"]))
    dinv = 1.0 / vals[pattern[0] == pattern[1]]
    x, r = torch.zeros_like(b), b.clone()
    z = dinv * r
    d, rz = z.clone(), torch.dot(r, z)
    for _ in range(4000):
        q = (A @ d[:, None])[:, 0]
        alpha = rz / torch.dot(d, q)
        x += alpha * d
        r -= alpha * q
        if float(torch.dot(r, r)) <= 1e-30 * float(torch.dot(b, b)):
            break
        z = dinv * r
        new = torch.dot(r, z)
        d = z + (new / rz) * d
        rz = new
    return x


# ---------------------------------------------------------------------------
# a form as FFCx writes it: inner(kappa grad u, grad v) dx + c u v dx, kappa a
# P1 field, c a constant, quadrature degree 3
# ---------------------------------------------------------------------------
def _ffcx_body(degree):
    pts, wts = _rule(2)
    phi, dphi = _tabulate(degree, pts)
    lam = np.column_stack([1 - pts.sum(axis=1), pts])
    k = phi.shape[1]

    def table(name, a):
        rows = ", ".join("{" + ", ".join(repr(float(v)) for v in r) + "}" for r in a)
        return "static const double %s[%d][%d] = {%s};\n" % (name, a.shape[0], a.shape[1], rows)

    body = "static const double weights[%d] = {%s};\n" % (len(wts), ", ".join(repr(float(v)) for v in wts))
    body += table("FE0", phi) + table("FE1", lam)
    for d in range(3):
        body += table("FE0_D%d" % d, dphi[:, d])
    return body + """
double J[3][3];
for (int r = 0; r < 3; ++r)
  for (int s = 0; s < 3; ++s) J[r][s] = coordinate_dofs[3 * (s + 1) + r] - coordinate_dofs[r];
const double c00 = J[1][1] * J[2][2] - J[1][2] * J[2][1];
const double c01 = J[1][2] * J[2][0] - J[1][0] * J[2][2];
const double c02 = J[1][0] * J[2][1] - J[1][1] * J[2][0];
const double detJ = J[0][0] * c00 + J[0][1] * c01 + J[0][2] * c02;
double K[3][3];
K[0][0] = c00 / detJ;
K[1][0] = c01 / detJ;
K[2][0] = c02 / detJ;
K[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) / detJ;
K[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) / detJ;
K[2][1] = (J[0][1] * J[2][0] - J[0][0] * J[2][1]) / detJ;
K[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) / detJ;
K[1][2] = (J[0][2] * J[1][0] - J[0][0] * J[1][2]) / detJ;
K[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) / detJ;
const double adet = fabs(detJ);
double G[3][3];
for (int s = 0; s < 3; ++s)
  for (int t = 0; t < 3; ++t) G[s][t] = K[s][0] * K[t][0] + K[s][1] * K[t][1] + K[s][2] * K[t][2];
for (int iq = 0; iq < NQ; ++iq) {
  double kappa = 0.0;
  for (int ic = 0; ic < 4; ++ic) kappa += w[ic] * FE1[iq][ic];
  const double fw = kappa * weights[iq] * adet;
  const double fm = c[0] * weights[iq] * adet;
  double t0[NB], t1[NB], t2[NB], t3[NB];
  for (int j = 0; j < NB; ++j) {
    const double d0 = FE0_D0[iq][j], d1 = FE0_D1[iq][j], d2 = FE0_D2[iq][j];
    t0[j] = fw * (G[0][0] * d0 + G[0][1] * d1 + G[0][2] * d2);
    t1[j] = fw * (G[1][0] * d0 + G[1][1] * d1 + G[1][2] * d2);
    t2[j] = fw * (G[2][0] * d0 + G[2][1] * d1 + G[2][2] * d2);
    t3[j] = fm * FE0[iq][j];
  }
  for (int i = 0; i < NB; ++i)
    for (int j = 0; j < NB; ++j)
      A[NB * i + j] += FE0_D0[iq][i] * t0[j] + FE0_D1[iq][i] * t1[j] + FE0_D2[iq][i] * t2[j] + FE0[iq][i] * t3[j];
}
""".replace("NQ", str(len(wts))).replace("NB", str(k))
