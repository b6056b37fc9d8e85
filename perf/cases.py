"""The work that users of feat3_b200 have it do, as cases that can be timed and checked.

Two layers are called, as their users call them:

* the operator layer (``feat3_b200.lafem``), which a FEAT3 build binds its containers to and
  through which its own multigrid templates run: matrix products with the defect and its norm,
  the ELL form, the transfers, and the vector work of an iteration;
* the solver layer (``feat3_b200.solver``): whole solves to a relative residual of 1e-8 on a
  hierarchy that the program has set up once, one application of the multigrid cycle as a
  preconditioner, and a solve followed by its adjoint gradient.

``exact`` computes every output again in 64 bits with plain torch: element matrices and lattice
stencils formed here, products by shifted arrays, and a multigrid-preconditioned CG that runs
until its residual stops falling.
"""
import itertools
import math

import numpy as np
import torch

from feat3_b200.lafem import DenseVector, SparseMatrixCSR, SparseMatrixELL, Transfer, UnitFilter
from feat3_b200.solver import MultiGrid

DT = {"f64": torch.float64, "f32": torch.float32}


# ------------------------------------------------------------------------------- the cases
def listed():
    return [
        # A defect and its norm on the smallest configured problem (2D Q1, 129 x 129), FEAT3's
        # default 64-bit Index: what one step of a stopping test costs when latency counts.
        dict(name="defect_2d_q1_small", kind="csr", dim=2, degree=1, nx=128, ny=128, nz=0, dtype="f64", index="u64",
             form="defect"),
        # The same on a 3D Q1 lattice of odd sides, 27 entries a row, larger than the L2: the
        # product that a FEAT3 program on CSR matrices spends its time in.
        dict(name="defect_3d_q1", kind="csr", dim=3, degree=1, nx=102, ny=100, nz=98, dtype="f64", index="u64",
             form="defect"),
        # The ELL container (C = 32) with rows of 9 to 25 entries (2D Q2) in FP32: ordinary size.
        dict(name="ell_2d_q2_f32", kind="ell", dim=2, degree=2, nx=150, ny=141, nz=0, dtype="f32", index="u32", C=32),
        # Prolongation and restriction between 129^3 and 65^3 as the reference stores them (P and R
        # in CSR), single precision.
        dict(name="transfer_3d_f32", kind="transfer", dim=3, nx=64, ny=64, nz=64, dtype="f32", index="u32"),
        # The vector work of one Jacobi-preconditioned CG iteration at 257^3, with the host reading
        # both dot products.
        dict(name="vectors_f64", kind="vectors", n=257 ** 3, dtype="f64"),
        # The default composition of the reference's Poisson application: 2D Q1, 129 x 129,
        # PCG with V(4,4), everything FP64: a small solve.
        dict(name="solve_2d_q1_f64", kind="solve", dim=2, degree=1, level=7, nu=4, precision="f64", format="sell",
             sigma=1, contrast=0.0),
        # A hierarchy that was assembled elsewhere and handed over as CSR matrices in a two-level
        # ordering (65^3, FP64, SELL-32-256).
        dict(name="solve_handed_3d_f64", kind="handed", dim=3, level=6, nu=2, precision="f64", sigma=256,
             contrast=1.0),
        # FP64 on assembled matrices at 257^3, varying coefficient: the drop-in form of the large
        # problem (a 5.5 GB finest matrix).
        dict(name="solve_3d_f64_sell", kind="solve", dim=3, degree=1, level=8, nu=2, precision="f64", format="sell",
             sigma=1, contrast=1.0),
        # Biquadratic elements, 1025 x 1025, FP16 matrix values inside an FP64 iteration.
        dict(name="solve_2d_q2_f16", kind="solve", dim=2, degree=2, level=9, nu=2, precision="f16", format="sell",
             sigma=1, contrast=1.0),
        # One cycle as a preconditioner of the caller's own iteration, FP32 on assembled matrices.
        dict(name="cycle_3d_f32_sell", kind="cycle", dim=3, degree=1, level=7, nu=2, precision="f32", format="sell",
             sigma=1, contrast=1.0),
        # Forward and backward: a solve and its adjoint gradient per coefficient, 513 x 513.
        dict(name="adjoint_2d_f32", kind="adjoint", dim=2, degree=1, level=9, nu=2, precision="f32", format="matfree",
             sigma=1, contrast=1.0),
        # The large solve: 16,974,593 unknowns, mixed precision on the matrix-free operator.
        dict(name="solve_3d_mixed_large", kind="solve", dim=3, degree=1, level=8, nu=2, precision="f32",
             format="matfree", sigma=1, contrast=1.0),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["csr", "csr", "ell", "transfer", "vectors", "solve", "solve", "solve", "handed", "cycle",
                       "adjoint"])
    dtype, index = rng.choice(["f64", "f64", "f32"]), rng.choice(["u32", "u64"])
    dim = rng.choice([2, 3])
    if kind in ("csr", "ell"):
        degree = rng.choice([1, 2]) if dim == 2 else 1
        n = log(1e3, 3e5) if kind == "ell" and dim == 2 else log(1e3, 1e5) if kind == "ell" else log(1e3, 1.5e6)
        side = max(2, n ** (1.0 / dim) / degree)
        c = [max(1, int(side * math.exp(rng.uniform(-0.4, 0.4)))) for _ in range(dim)] + [0]
        case = dict(kind=kind, dim=dim, degree=degree, nx=c[0], ny=c[1], nz=c[2] if dim == 3 else 0, dtype=dtype,
                    index=index)
        if kind == "ell":
            case["C"] = rng.choice([8, 16, 32, 32, 64])
        else:
            case["form"] = rng.choice(["defect", "defect", "product", "transposed"])
        return case
    if kind == "transfer":
        n = log(5e2, 3e5)
        c = [max(1, int(n ** (1.0 / dim) * math.exp(rng.uniform(-0.3, 0.3)))) for _ in range(dim)] + [0]
        return dict(kind=kind, dim=dim, nx=c[0], ny=c[1], nz=c[2] if dim == 3 else 0, dtype=dtype, index=index)
    if kind == "vectors":
        return dict(kind=kind, n=log(1e3, 2e7), dtype=dtype)
    # spread of log k over the cells; 0: k = 1
    contrast = round(rng.uniform(0.3, 1.2), 3) if rng.random() < 0.9 else 0.0
    if kind == "handed":
        return dict(kind=kind, dim=dim, level=rng.randint(4, 9) if dim == 2 else rng.randint(3, 6),
                    nu=rng.choice([2, 2, 3, 4]), precision=rng.choice(["f64", "f64", "f32", "f16"]),
                    sigma=rng.choice([1, 32, 256]), contrast=contrast)
    degree = 1 if dim == 3 or kind == "adjoint" else rng.choice([1, 1, 2])
    top = 10 if dim == 2 and degree == 1 else 9 if dim == 2 else 7
    level = rng.randint(5, min(top, 9) if kind == "adjoint" else top) if dim == 2 else rng.randint(4, top)
    fmt = rng.choice(["sell", "stencil", "matfree"])
    return dict(kind=kind, dim=dim, degree=degree, level=level, nu=rng.choice([2, 2, 3, 4]),
                precision=rng.choice(["f64", "f32", "f16"]) if fmt != "matfree" else rng.choice(["f64", "f32"]),
                format=fmt, sigma=rng.choice([1, 1, 256]), contrast=contrast)


# ------------------------------------------------------------------------------- lattices
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _normal(g, *shape):
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g)


def _basis_1d(degree):
    """mass and stiffness matrix of the 1D Lagrange element on the unit interval"""
    if degree == 1:
        return np.array([[2, 1], [1, 2]]) / 6.0, np.array([[1.0, -1], [-1, 1]])
    return (np.array([[4, 2, -1], [2, 16, 2], [-1, 2, 4]]) / 30.0,
            np.array([[7, -8, 1], [-8, 16, -8], [1, -8, 7]]) / 3.0)


def _element_matrix(dim, degree):
    """Laplace matrix of the unit cell, nodes with x fastest"""
    m, s = _basis_1d(degree)
    if dim == 2:
        return np.kron(m, s) + np.kron(s, m)
    return np.kron(m, np.kron(m, s)) + np.kron(m, np.kron(s, m)) + np.kron(s, np.kron(m, m))


def _stencil(dim, degree, k, scale=1.0):
    """{offset: array}: the lattice matrix of the cells' coefficients k (z, y, x order; offsets too)"""
    K = _element_matrix(dim, degree) * scale
    M = [degree * c + 1 for c in k.shape]
    local = list(itertools.product(range(degree + 1), repeat=dim))
    offs = list(itertools.product(range(-degree, degree + 1), repeat=dim))
    A = {o: torch.zeros(M, dtype=torch.float64, device=k.device) for o in offs}
    for i, a in enumerate(local):
        at = tuple(slice(a[d], a[d] + degree * (k.shape[d] - 1) + 1, degree) for d in range(dim))
        for j, b in enumerate(local):
            A[tuple(b[d] - a[d] for d in range(dim))][at] += K[i, j] * k
    return A


def _apply(A, x):
    dim = x.dim()
    pad = max(max(o) for o in A)
    xp = torch.nn.functional.pad(x, [pad] * (2 * dim))
    y = torch.zeros_like(x)
    for o, a in A.items():
        y.addcmul_(a, xp[tuple(slice(pad + o[d], pad + o[d] + x.shape[d]) for d in range(dim))])
    return y


def _csr(A):
    """row pointer, columns and values of the lattice matrix, structural zeros kept; degree 2: only
    the couplings that share a cell"""
    offs = sorted(A)
    any_a = A[offs[0]]
    M, dim, degree = any_a.shape, any_a.dim(), max(max(o) for o in offs)
    grid = torch.meshgrid(*[torch.arange(m, device="cuda") for m in M], indexing="ij")
    stride = [int(np.prod(M[d + 1:])) for d in range(dim)]
    row = sum(g * s for g, s in zip(grid, stride)).reshape(-1)
    ok, val = [], []
    for o in offs:
        there = torch.ones(M, dtype=torch.bool, device="cuda")
        for d in range(dim):
            to = grid[d] + o[d]
            there &= (to >= 0) & (to < M[d])
            if degree == 2:  # nodes between corners reach their own cell only
                there &= (abs(o[d]) < 2) | (grid[d] % 2 == 0)
        ok.append(there.reshape(-1))
        val.append(A[o].reshape(-1))
    ok, val = torch.stack(ok, 1), torch.stack(val, 1)
    shift = torch.tensor([sum(o[d] * stride[d] for d in range(dim)) for o in offs], device="cuda")
    col = (row[:, None] + shift[None, :])[ok]
    rp = torch.zeros(row.numel() + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(ok.sum(1), 0)
    return rp, col, val[ok]


def _boundary(M):
    b = torch.zeros(M, dtype=torch.bool, device="cuda")
    for d in range(len(M)):
        b.select(d, 0).fill_(True)
        b.select(d, M[d] - 1).fill_(True)
    return b


def _prol_1d(cells, degree):
    """nested interpolation from `cells` to 2 cells elements per side, one direction"""
    P = torch.zeros(2 * degree * cells + 1, degree * cells + 1, dtype=torch.float64)
    for i in range(P.shape[0]):
        e = min(i // (2 * degree), cells - 1)
        t = (i - 2 * degree * e) / (2.0 * degree)
        w = [1 - t, t] if degree == 1 else [(1 - t) * (1 - 2 * t), 4 * t * (1 - t), t * (2 * t - 1)]
        for a, v in enumerate(w):
            P[i, degree * e + a] = v
    return P.cuda()


def _along(mats, x):
    """x with a matrix applied along each of its directions"""
    for d, m in enumerate(mats):
        x = torch.movedim(torch.tensordot(m, x, dims=([1], [d])), 0, d).contiguous()
    return x


def _prol_csr(cells):
    """Q1 prolongation between lattices of cells and 2 cells as (rows, cols, values)"""
    dim = len(cells)
    Mf, Mc = [2 * c + 1 for c in cells], [c + 1 for c in cells]
    grid = torch.meshgrid(*[torch.arange(m, device="cuda") for m in Mf], indexing="ij")
    rows, cols, vals = [], [], []
    row = torch.arange(int(np.prod(Mf)), device="cuda").reshape(Mf)
    for b in itertools.product((0, 1), repeat=dim):
        w = torch.ones(Mf, dtype=torch.float64, device="cuda")
        c = torch.zeros(Mf, dtype=torch.int64, device="cuda")
        for d in range(dim):
            odd = grid[d] % 2 == 1
            w = w * torch.where(odd, 0.5, 0.0 if b[d] else 1.0)
            c = c * Mc[d] + (grid[d] + b[d]) // 2
        there = w > 0
        rows.append(row[there])
        cols.append(c[there])
        vals.append(w[there])
    return torch.cat(rows), torch.cat(cols), torch.cat(vals)


def _sorted_csr(rows, cols, vals, n):
    at = torch.argsort(rows * (int(cols.max()) + 1) + cols)
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return rp, cols[at], vals[at]


def _host(*tensors):
    return tuple(t.cpu().numpy() for t in tensors)


def _two_level_order(dim, level):
    """lattice index of each DOF when every refinement keeps the old vertices first and appends the
    new ones: edge points, then face points, then cell points"""
    c = torch.arange(2 ** level + 1, device="cuda")
    zeros = torch.full_like(c, level)  # trailing zero bits; 0 and 2^level are corners
    for b in range(level - 1, -1, -1):
        zeros = torch.where(c % (1 << (b + 1)) == (1 << b), b, zeros)
    grid = torch.meshgrid(*[zeros] * dim, indexing="ij")
    born = torch.stack(grid).amin(0)
    kind = sum((g == born).long() for g in grid)
    key = (level - born) * (dim + 1) + torch.where(born == level, 0, kind)
    return torch.argsort(key.reshape(-1), stable=True)


# ------------------------------------------------------------------------------- inputs
def _cells(case):
    return (case["ny"], case["nx"]) if case["dim"] == 2 else (case["nz"], case["ny"], case["nx"])


def _coefficient(shape, seed, contrast=1.0):
    """k = exp(g), g ~ N(0, contrast^2) per cell"""
    return torch.exp(contrast * _normal(_gen(seed, 1), *shape))


def _load(dim, degree, level, seed):
    """load vector of a source that is constant on each cell, zero on the boundary"""
    shape = (2 ** level,) * dim
    f = 0.5 + torch.rand(shape, dtype=torch.float64, device="cuda", generator=_gen(seed, 2))
    f = f * (0.5 ** level) ** dim
    w = {1: [0.5, 0.5], 2: [1 / 6, 4 / 6, 1 / 6]}[degree]
    M = [degree * c + 1 for c in shape]
    b = torch.zeros(M, dtype=torch.float64, device="cuda")
    for a in itertools.product(range(degree + 1), repeat=dim):
        at = tuple(slice(a[d], a[d] + degree * (shape[d] - 1) + 1, degree) for d in range(dim))
        b[at] += math.prod(w[i] for i in a) * f
    b[_boundary(M)] = 0.0
    return b


def _operator_inputs(case, seed):
    k = _coefficient(_cells(case), seed)
    A = _stencil(case["dim"], case["degree"], k)
    n = math.prod(next(iter(A.values())).shape)
    g = _gen(seed, 3)
    return A, _normal(g, n).to(DT[case["dtype"]]), _normal(g, n).to(DT[case["dtype"]])


def _vector_inputs(case, seed):
    g = _gen(seed, 4)
    v = {c: _normal(g, case["n"]).to(DT[case["dtype"]]) for c in "xrpq"}
    v["d"] = (0.5 + torch.rand(case["n"], dtype=torch.float64, device="cuda", generator=g)).to(DT[case["dtype"]])
    return v


def _transfer_inputs(case, seed):
    cells = _cells(case)
    g = _gen(seed, 5)
    nc, nf = math.prod(c + 1 for c in cells), math.prod(2 * c + 1 for c in cells)
    return cells, _normal(g, nc).to(DT[case["dtype"]]), _normal(g, nf).to(DT[case["dtype"]])


def _defect(case, seed):
    M = (case["degree"] * 2 ** case["level"] + 1,) * case["dim"]
    d = _normal(_gen(seed, 6), *M)
    d[_boundary(M)] = 0.0
    return d


def _target(case, seed):
    M = (2 ** case["level"] + 1,) * case["dim"]
    return 1e-2 * _normal(_gen(seed, 7), *M)


def _handed_levels(case, k):
    dim, levels = case["dim"], []
    for level in range(case["level"], 0, -1):
        shape = (2 ** level + 1,) * dim
        perm = _two_level_order(dim, level)
        inv = torch.empty_like(perm)
        inv[perm] = torch.arange(perm.numel(), device="cuda")
        rp, ci, va = _csr(_stencil(dim, 1, k, (0.5 ** level) ** (dim - 2)))
        rows = torch.repeat_interleave(torch.arange(perm.numel(), device="cuda"), rp[1:] - rp[:-1])
        A = _sorted_csr(inv[rows], inv[ci], va, perm.numel())
        d = {"A": _host(*A), "filter": _host(torch.sort(inv[_boundary(shape).reshape(-1)])[0])[0]}
        if levels:
            fine, fine_inv, fine_n = levels[-1], last_inv, last_inv.numel()
            r, c, v = _prol_csr([2 ** level] * dim)
            r, c = fine_inv[r], inv[c]
            fine["P"] = _host(*_sorted_csr(r, c, v, fine_n))
            fine["R"] = _host(*_sorted_csr(c, r, v, perm.numel()))
        levels.append(d)
        last_inv = inv
        k = _coarser(k)
    return levels


def _coarser(k):
    """mean over the 2^dim children of each coarser cell"""
    for d in range(k.dim()):
        k = 0.5 * (k[(slice(None),) * d + (slice(0, None, 2),)] + k[(slice(None),) * d + (slice(1, None, 2),)])
    return k


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("csr", "ell"):
        A, x, y = _operator_inputs(case, seed)
        M = next(iter(A.values())).shape
        rp, ci, va = _host(*_csr(A))
        dt = DT[case["dtype"]]
        if kind == "ell":
            mat = SparseMatrixELL(rp, ci, va, C=case["C"], dtype=dt, index=case["index"])
        else:
            mat = SparseMatrixCSR(rp, ci, va, dtype=dt, index=case["index"])
        bnd = _host(torch.nonzero(_boundary(M).reshape(-1)).reshape(-1))[0]
        return dict(case=case, A=mat, x=DenseVector(x), y=DenseVector(y), r=DenseVector.zeros(x.numel(), dt),
                    filter=UnitFilter(bnd, dtype=dt, index=case["index"]))
    if kind == "transfer":
        cells, c, f = _transfer_inputs(case, seed)
        r, q, v = _prol_csr(cells)
        dt = DT[case["dtype"]]
        P = SparseMatrixCSR(*_host(*_sorted_csr(r, q, v, f.numel())), columns=c.numel(), dtype=dt, index=case["index"])
        R = SparseMatrixCSR(*_host(*_sorted_csr(q, r, v, c.numel())), columns=f.numel(), dtype=dt, index=case["index"])
        return dict(case=case, T=Transfer(P, R), c=DenseVector(c), f=DenseVector(f),
                    pc=DenseVector.zeros(f.numel(), dt), rf=DenseVector.zeros(c.numel(), dt))
    if kind == "vectors":
        s = {n: DenseVector(t) for n, t in _vector_inputs(case, seed).items()}
        for n in ("x1", "r1", "z", "p1"):
            s[n] = DenseVector.zeros(case["n"], DT[case["dtype"]])
        s["case"] = case
        return s
    dim = case["dim"]
    if kind == "handed":
        k = _coefficient((2 ** case["level"],) * dim, seed, case["contrast"])
        mg = MultiGrid.from_csr(_handed_levels(case, k), sell_sigma=case["sigma"])
        mg.configure(nu=case["nu"], precision=case["precision"])
        rhs = _load(dim, 1, case["level"], seed).reshape(-1)[_two_level_order(dim, case["level"])]
        return dict(case=case, mg=mg, rhs=rhs.contiguous())
    k = None
    if case["contrast"] > 0:
        k = _coefficient((2 ** case["level"],) * dim, seed, case["contrast"]).reshape(-1)
    mg = MultiGrid.structured(dim, case["degree"], case["level"], 1, k, sell_sigma=case["sigma"])
    mg.configure(nu=case["nu"], precision=case["precision"], format=case["format"])
    s = dict(case=case, mg=mg)
    if kind == "cycle":
        s["d"] = _defect(case, seed).reshape(-1)
    else:
        s["rhs"] = _load(dim, case["degree"], case["level"], seed).reshape(-1)
    if kind == "adjoint":
        s["target"] = _target(case, seed).reshape(-1)
    return s


# ------------------------------------------------------------------------------- one pass
ALPHA, BETA = 0.37, 0.61  # step lengths of the vector case


def run(s):
    kind = s["case"]["kind"]
    if kind == "csr":
        form = s["case"]["form"]
        if form == "defect":
            r = s["filter"].filter_def(s["A"].apply(s["r"], s["x"], s["y"], -1.0))
            return {"r": r.t, "norm": r.norm2()}
        return {"r": s["A"].apply(s["r"], s["x"], transposed=form == "transposed").t}
    if kind == "ell":
        return {"r": s["A"].apply(s["r"], s["x"], s["y"], -1.0).t}
    if kind == "transfer":
        return {"prol": s["T"].prol(s["pc"], s["c"]).t, "rest": s["T"].rest(s["f"], s["rf"]).t}
    if kind == "vectors":
        s["x1"].axpy(s["p"], s["x"], ALPHA)
        s["r1"].axpy(s["q"], s["r"], -ALPHA)
        norm = s["r1"].norm2()
        s["z"].component_product(s["d"], s["r1"])
        rz = s["r1"].dot(s["z"])
        s["p1"].axpy(s["p"], s["z"], BETA)
        return {"x": s["x1"].t, "r": s["r1"].t, "z": s["z"].t, "p": s["p1"].t, "norm": norm, "rz": rz}
    if kind == "cycle":
        return {"cor": s["mg"].vcycle(s["d"])}
    u = s["mg"].solve(s["rhs"])["u"]
    if kind != "adjoint":
        return {"u": u}
    lam, grad, _ = s["mg"].adjoint_grad(u, s["target"])
    return {"u": u, "lambda": lam, "grad": grad}


# ------------------------------------------------------------------------------- bytes and operations
def _nnz(dim, degree, cells):
    per = [(3 * (c + 1) - 2) if degree == 1 else (5 * (c + 1) - 4 + 3 * c) for c in cells]
    return math.prod(per)


def _cycle_work(dim, degree, level, nu, value, vector, assembled):
    """bytes and operations of one V(nu, nu) cycle: per level 2 nu operator applications (the first
    step from zero is a scaling) and the defect, each reading the operator once, one vector and the
    right-hand side, and writing one vector; assembled operators are read at their value size
    without indices, matrix-free ones as one coefficient per cell"""
    by = fl = 0.0
    for l in range(level, 0, -1):
        cells = (2 ** l,) * dim
        n, nnz = math.prod(degree * c + 1 for c in cells), _nnz(dim, degree, cells)
        op = nnz * value if assembled else math.prod(cells) * vector
        by += 2 * nu * (op + 3 * n * vector)
        fl += 2 * nu * 2 * nnz
    return by, fl


def work(case):
    kind = case["kind"]
    if kind in ("csr", "ell", "transfer", "vectors"):
        sv = 8 if case["dtype"] == "f64" else 4
        if kind == "vectors":  # x p -> x1; r q -> r1; d -> z; p1 (r1 and z are read as they are made)
            return {"bytes": 9 * sv * case["n"], "flops": 11 * case["n"]}
        si, cells = 8 if case["index"] == "u64" else 4, _cells(case)
        if kind == "transfer":
            nc, nf = math.prod(c + 1 for c in cells), math.prod(2 * c + 1 for c in cells)
            nnz = math.prod((c + 1) + 2 * c for c in cells)
            return {"bytes": 2 * nnz * (sv + si) + (nc + nf) * (2 * sv + si), "flops": 4 * nnz}
        n, nnz = math.prod(case["degree"] * c + 1 for c in cells), _nnz(case["dim"], case["degree"], cells)
        vectors = 2 if kind == "csr" and case["form"] != "defect" else 3
        return {"bytes": nnz * (sv + si) + n * (vectors * sv + si), "flops": 2 * nnz}
    # whole solves: 8 iterations where the coefficient is constant, 18 where it varies (41 biquadratic),
    # each one cycle, one product of the outer iteration and its vectors
    dim, level, degree = case["dim"], case["level"], case.get("degree", 1)
    low = case["precision"] != "f64"
    value = {"f64": 8, "f32": 4, "f16": 2}[case["precision"]]
    assembled = case.get("format", "sell") != "matfree" or degree == 2
    by, fl = _cycle_work(dim, degree, level, case["nu"], value, 4 if low else 8, assembled)
    n, cells = (degree * 2 ** level + 1) ** dim, (2 ** level,) * dim
    nnz = _nnz(dim, degree, cells)
    if kind == "cycle":
        return {"bytes": by + 16 * n, "flops": fl}
    iters = 41 if degree == 2 else 18 if case["contrast"] > 0 else 8
    iters *= 2 if kind == "adjoint" else 1
    outer = (8 * nnz if assembled else 8 * math.prod(cells)) + 8 * 8 * n
    return {"bytes": iters * (by + outer) + 16 * n, "flops": iters * (fl + 2 * nnz + 10 * n)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("csr", "ell", "transfer", "vectors"):
        # rows of up to 27 products; measured 2e-16 and 9e-8 against 64-bit sums in another order
        return {"rel": 1e-15 if case["dtype"] == "f64" else 4e-7}
    if kind == "cycle":  # measured up to 2.5e-15, 2.3e-7 and 7e-4 (rounded matrix values)
        return {"rel": {"f64": 1e-14, "f32": 1e-6, "f16": 3e-3}[case["precision"]]}
    # stopped at a relative residual of 1e-8: measured up to 7e-10 from the solution, 1.4e-9 in the gradient
    return {"rel": 6e-9 if kind == "adjoint" else 4e-9}


# ------------------------------------------------------------------------------- 64-bit values
class _Exact:
    """geometric multigrid in 64 bits on the unit square or cube, homogeneous boundary"""

    def __init__(self, dim, degree, level, nu, k):
        self.nu, self.levels = nu, []
        for l in range(level, 0, -1):
            A = _stencil(dim, degree, k, (0.5 ** l) ** (dim - 2))
            M = next(iter(A.values())).shape
            inner = (~_boundary(M)).double()
            P = [_prol_1d(2 ** (l - 1), degree)] * dim if l > 1 else None
            self.levels.append((A, 0.5 * inner / A[(0,) * dim], inner, P))
            k = _coarser(k)
        A, _, inner, _ = self.levels[-1]
        n = inner.numel()
        eye = torch.eye(n, dtype=torch.float64, device="cuda").reshape(n, *inner.shape)
        dense = torch.stack([_apply(A, e * inner).mul(inner).reshape(-1) for e in eye], 1)
        keep = inner.reshape(-1) > 0
        self.inverse = torch.zeros_like(dense)
        self.inverse[torch.outer(keep, keep)] = torch.linalg.inv(dense[keep][:, keep]).reshape(-1)

    def defect(self, b, x, l=0):
        A, _, inner, _ = self.levels[l]
        return (b - _apply(A, x)) * inner

    def cycle(self, b, l=0):
        if l + 1 == len(self.levels):
            return (self.inverse @ b.reshape(-1)).reshape(b.shape)
        _, d, inner, P = self.levels[l]
        x = d * b
        for _ in range(self.nu - 1):
            x = x + d * self.defect(b, x, l)
        c = _along([p.t() for p in P], self.defect(b, x, l)) * self.levels[l + 1][2]
        x = x + _along(P, self.cycle(c, l + 1)) * inner
        for _ in range(self.nu):
            x = x + d * self.defect(b, x, l)
        return x

    def solve(self, b):
        """CG until the residual is 1e-14 of the first"""
        b = b * self.levels[0][2]
        x, r = torch.zeros_like(b), b
        z = self.cycle(r)
        p, rz, first = z, (r * z).sum(), r.norm()
        for _ in range(100):
            q = _apply(self.levels[0][0], p) * self.levels[0][2]
            alpha = rz / (p * q).sum()
            x, r = x + alpha * p, r - alpha * q
            if r.norm() <= 1e-14 * first:
                break
            z = self.cycle(r)
            last, rz = rz, (r * z).sum()
            p = z + rz / last * p
        return x


def exact(case, seed):
    kind = case["kind"]
    if kind in ("csr", "ell"):
        A, x, y = _operator_inputs(case, seed)
        low = case["dtype"] == "f32"
        A = {o: a.float().double() if low else a for o, a in A.items()}
        M = next(iter(A.values())).shape
        x, y = x.double().reshape(M), y.double().reshape(M)
        Ax = _apply(A, x)  # symmetric: the transposed product is the same
        if kind == "ell":
            return {"r": (y - Ax).reshape(-1)}
        if case["form"] != "defect":
            return {"r": Ax.reshape(-1)}
        r = (y - Ax) * (~_boundary(M)).double()
        return {"r": r.reshape(-1), "norm": float(r.norm())}
    if kind == "transfer":
        cells, c, f = _transfer_inputs(case, seed)
        P = [_prol_1d(n, 1) for n in cells]
        return {"prol": _along(P, c.double().reshape([n + 1 for n in cells])).reshape(-1),
                "rest": _along([p.t() for p in P], f.double().reshape([2 * n + 1 for n in cells])).reshape(-1)}
    if kind == "vectors":
        v = {n: t.double() for n, t in _vector_inputs(case, seed).items()}
        a, b = (float(torch.tensor(c, dtype=DT[case["dtype"]])) for c in (ALPHA, BETA))
        r = v["r"] - a * v["q"]
        z = v["d"] * r
        return {"x": v["x"] + a * v["p"], "r": r, "z": z, "p": z + b * v["p"], "norm": float(r.norm()),
                "rz": float((r * z).sum())}
    dim, degree, level = case["dim"], case.get("degree", 1), case["level"]
    k = _coefficient((2 ** level,) * dim, seed, case["contrast"])
    mg = _Exact(dim, degree, level, case["nu"], k)
    if kind == "cycle":
        return {"cor": mg.cycle(_defect(case, seed)).reshape(-1)}
    u = mg.solve(_load(dim, degree, level, seed))
    if kind == "handed":
        return {"u": u.reshape(-1)[_two_level_order(dim, level)]}
    if kind != "adjoint":
        return {"u": u.reshape(-1)}
    lam = mg.solve(u - _target(case, seed))
    K = _element_matrix(dim, 1) * (0.5 ** level) ** (dim - 2)
    corner = [tuple(slice(a, a + 2 ** level) for a in b) for b in itertools.product((0, 1), repeat=dim)]
    grad = torch.zeros_like(k)
    for i, a in enumerate(corner):
        for j, b in enumerate(corner):
            grad -= K[i, j] * lam[a] * u[b]
    return {"u": u.reshape(-1), "lambda": lam.reshape(-1), "grad": grad.reshape(-1)}
