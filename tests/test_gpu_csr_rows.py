"""CSR products over every width the kernel picks (1 to 32 threads per row, four entries of a thread
loaded at a time): rows shorter and longer than a group's step, empty rows, rows of very different
length, both index widths, with and without y, against SciPy in 64 bits."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

pytestmark = pytest.mark.gpu

LENGTHS = {
    "empty_and_1": lambda rng, n: rng.integers(0, 2, n),
    "1_to_8": lambda rng, n: rng.integers(1, 9, n),
    "9": lambda rng, n: np.full(n, 9),
    "13_to_20": lambda rng, n: rng.integers(13, 21, n),
    "27": lambda rng, n: np.full(n, 27),
    "33_to_60": lambda rng, n: rng.integers(33, 61, n),
    "125": lambda rng, n: np.full(n, 125),
    "4_to_7": lambda rng, n: rng.integers(4, 8, n),
    "long_rows": lambda rng, n: np.where((n - 1 - np.arange(n)) % 26 == 0, rng.integers(60, 69, n), rng.integers(0, 2, n)),
    "one_long": lambda rng, n: np.where(np.arange(n) == n // 2, 1500, rng.integers(0, 4, n)),
}


@pytest.mark.parametrize("index", ["u32", "u64"])
@pytest.mark.parametrize("dtype,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
@pytest.mark.parametrize("name", sorted(LENGTHS))
def test_rows(name, dtype, eps, index):
    from feat3_b200.lafem import DenseVector, SparseMatrixCSR
    rng = np.random.default_rng(3)
    n, m = 777, 2000
    rl = LENGTHS[name](rng, n)
    rp = np.concatenate([[0], np.cumsum(rl)])
    ci = np.concatenate([np.sort(rng.choice(m, k, replace=False)) for k in rl] + [np.zeros(0, np.int64)]).astype(np.int64)
    cast = (lambda a: a.astype(np.float32).astype(np.float64)) if dtype == torch.float32 else (lambda a: a)
    va, x, y = cast(rng.standard_normal(ci.size)), cast(rng.standard_normal(m)), cast(rng.standard_normal(n))
    S = sp.csr_matrix((va, ci, rp), shape=(n, m), copy=True)
    A = SparseMatrixCSR(rp, ci, va, columns=m, dtype=dtype, index=index)
    X, Y, R = (DenseVector(torch.tensor(v, dtype=dtype).cuda()) for v in (x, y, np.full(n, np.nan)))
    terms = sp.csr_matrix((abs(va), ci, rp), shape=(n, m)) @ abs(x)
    bound = (rl + 3) * eps * (terms + abs(y))  # one rounding per entry, three for a, b and the sum
    assert np.all(abs(A.apply(R, X).numpy() - S @ x) <= bound)
    assert np.all(abs(A.apply(R, X, Y, -1.0).numpy() - (y - S @ x)) <= bound)


@pytest.mark.parametrize("index", ["u32", "u64"])
@pytest.mark.parametrize("name", sorted(LENGTHS))
def test_terms_are_summed_in_groups(name, index):
    """FP32: the terms of a row are summed in 2, 4, 8, 16 or 32 groups (up to 6, 12, 32, 64 and more entries
    a row), each with one running sum, which are then added pairwise; a row of more than 32 entries per
    thread (up to four threads) in 32"""
    from feat3_b200.lafem import DenseVector, SparseMatrixCSR
    rng = np.random.default_rng(4)
    n, m = 777, 2000
    rl = LENGTHS[name](rng, n)
    rp = np.concatenate([[0], np.cumsum(rl)])
    ci = np.concatenate([np.sort(rng.choice(m, k, replace=False)) for k in rl] + [np.zeros(0, np.int64)]).astype(np.int64)
    va, x = rng.standard_normal(ci.size).astype(np.float32), rng.standard_normal(m).astype(np.float32)
    A = SparseMatrixCSR(rp, ci, va, columns=m, dtype=torch.float32, index=index)
    X, R = DenseVector(torch.tensor(x).cuda()), DenseVector(torch.full((n,), np.nan).cuda())
    out = A.apply(R, X).numpy()
    avg = ci.size / n
    g = 2 if avg <= 6 else 4 if avg <= 12 else 8 if avg <= 32 else 16 if avg <= 64 else 32
    ref = np.zeros(n, np.float32)
    for i in range(n):
        s = np.zeros(32 if rl[i] > 32 * g and g < 8 else g, np.float32)
        for k in range(rp[i], rp[i + 1]):  # one rounding (fused multiply-add): the FP64 product is exact
            s[(k - rp[i]) % s.size] = np.float32(float(va[k]) * float(x[ci[k]]) + float(s[(k - rp[i]) % s.size]))
        while s.size > 1:
            s = s[:s.size // 2] + s[s.size // 2:]
        ref[i] = s[0]
    # (the reference rounds twice, to 53 and to 24 bits: another last bit in 1 of 2^29 terms)
    assert np.count_nonzero(out != ref) <= 1


@pytest.mark.parametrize("index", ["u32", "u64"])
@pytest.mark.parametrize("length,rows,groups", [(3, 160000, 2), (6, 70000, 2), (9, 270000, 4), (16, 135000, 4), (27, 135000, 8),
                                                (40, 66000, 16)])
def test_many_rows(length, rows, groups, index):
    """row counts above which a row gets fewer threads (and several sums in each): the same groups,
    to the last bit in FP32 as above"""
    from feat3_b200.lafem import DenseVector, SparseMatrixCSR
    rng = np.random.default_rng(length)
    ci = rng.integers(0, rows, (rows, length))
    va = rng.standard_normal((rows, length)).astype(np.float32)
    x = rng.standard_normal(rows).astype(np.float32)
    A = SparseMatrixCSR(np.arange(rows + 1) * length, ci.ravel(), va.ravel(), columns=rows, dtype=torch.float32, index=index)
    X, R = DenseVector(torch.tensor(x).cuda()), DenseVector(torch.full((rows,), np.nan).cuda())
    s = np.zeros((rows, groups), np.float32)
    for j in range(length):
        t = va[:, j].astype(np.float64) * x[ci[:, j]] + s[:, j % groups]
        s[:, j % groups] = t.astype(np.float32)
    while s.shape[1] > 1:
        s = s[:, :s.shape[1] // 2] + s[:, s.shape[1] // 2:]
    assert np.count_nonzero(A.apply(R, X).numpy() != s[:, 0]) <= 1


@pytest.mark.parametrize("index", ["u32", "u64"])
@pytest.mark.parametrize("dtype,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
def test_many_short_rows_and_long_ones(dtype, eps, index):
    """one thread per row: rows around its limit of 32 entries and far above it"""
    from feat3_b200.lafem import DenseVector, SparseMatrixCSR
    rng = np.random.default_rng(2)
    n = 170000
    rl = rng.integers(0, 4, n)
    rl[rng.choice(n, 3000, replace=False)] = rng.integers(30, 36, 3000)
    rl[[5, 6, 7, n - 1]] = [3000, 32, 33, 700]
    rp = np.concatenate([[0], np.cumsum(rl)])
    ci = rng.integers(0, n, rp[-1])
    cast = (lambda a: a.astype(np.float32).astype(np.float64)) if dtype == torch.float32 else (lambda a: a)
    va, x = cast(rng.standard_normal(ci.size)), cast(rng.standard_normal(n))
    A = SparseMatrixCSR(rp, ci, va, columns=n, dtype=dtype, index=index)
    X, R = DenseVector(torch.tensor(x, dtype=dtype).cuda()), DenseVector(torch.full((n,), np.nan, dtype=dtype).cuda())
    S = sp.csr_matrix((va, ci, rp), shape=(n, n), copy=True)
    bound = (rl + 3) * eps * (sp.csr_matrix((abs(va), ci, rp), shape=(n, n)) @ abs(x))
    assert np.all(abs(A.apply(R, X).numpy() - S @ x) <= bound)


@pytest.mark.parametrize("dtype,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
@pytest.mark.parametrize("avg,empty", [(3, 0), (7, 0), (9, 0), (27, 0), (50, 0), (125, 0), (3, 200000), (9, 300000),
                                       (16, 200000), (27, 200000)])
def test_last_row_at_the_index_limit(avg, empty, dtype, eps):
    """32-bit row pointers up to 2^32 - 1: a lane's next position would lie behind the limit. The
    arrays start where the first of these rows does (their addresses are shifted by its position); the
    mean row length given and the number of (empty) rows before them pick the threads per row."""
    from feat3_b200 import _lib
    sfx = "f64" if dtype == torch.float64 else "f32"
    rng = np.random.default_rng(avg)
    m = 300
    for rl in ([1, 2, 0, 5], [40, 127, 0, 130], [300, 1], [7]):
        end = 2 ** 32 - 1
        ci = np.concatenate([np.sort(rng.choice(m, k, replace=False)) for k in rl])
        rl = [0] * empty + rl
        rp = end - sum(rl) + np.concatenate([[0], np.cumsum(rl)])
        nnz, n = sum(rl), len(rl)
        va = rng.standard_normal(nnz).astype(np.float32).astype(np.float64)
        x = rng.standard_normal(max(m, n)).astype(np.float32).astype(np.float64)
        S = sp.csr_matrix((va, ci, rp - rp[0]), shape=(n, m), copy=True)
        dev = lambda a, t: torch.tensor(a, dtype=t).cuda()
        V, X, Y, R = dev(va, dtype), dev(x, dtype), dev(np.zeros(m), dtype), dev(np.full(max(m, n), np.nan), dtype)
        C = torch.tensor(ci.astype(np.uint32).view(np.int32)).cuda()
        P = torch.tensor(rp.astype(np.uint32).view(np.int32)).cuda()
        first = int(rp[0])
        args = (V.data_ptr() - first * V.element_size(), C.data_ptr() - first * 4, P.data_ptr())
        st = torch.cuda.current_stream().cuda_stream
        _lib.call("fb_csr_apply_" + sfx, R.data_ptr(), 1.0, X.data_ptr(), 0.0, None, *args, n, m, avg * n, 0, st)
        bound = (np.array(rl) + 3) * eps * (abs(S) @ abs(x[:m]))
        assert np.all(abs(R[:n].double().cpu().numpy() - S @ x[:m]) <= bound)
        _lib.call("fb_csr_apply_" + sfx, R.data_ptr(), 1.0, X.data_ptr(), 0.0, None, *args, n, m, avg * n, 1, st)
        bound = (n + 3) * eps * (abs(S).T @ abs(x[:n]))
        assert np.all(abs(R[:m].double().cpu().numpy() - S.T @ x[:n]) <= bound)


@pytest.mark.parametrize("prec,eps", [("f64", 2.0 ** -53), ("f32", 2.0 ** -24)])
@pytest.mark.parametrize("long_p,long_r", [(0, 0), (33, 0), (200, 0), (0, 300), (200, 300)])
def test_transfers_with_long_rows(long_p, long_r, prec, eps):
    """one cycle on two handed-over levels whose prolongation or restriction has a row that is much
    longer than the mean, against the same in NumPy"""
    from feat3_b200.solver import MultiGrid
    rng = np.random.default_rng(8)
    n, nc = 3000, 700
    def diagonal_plus(m):
        B = sp.random(m, m, 4.0 / m, random_state=rng, format="csr")
        A = sp.csr_matrix(B + B.T + 8.0 * sp.identity(m))
        A.sort_indices()
        return A
    def transfer(rows, cols, k, row, length):
        T = sp.lil_matrix(sp.random(rows, cols, k / cols, random_state=rng))
        if length:
            T[row, np.sort(rng.choice(cols, length, replace=False))] = rng.uniform(0.1, 1.0, length)
        T = sp.csr_matrix(T)
        T.sort_indices()
        return T
    A, Ac = diagonal_plus(n), diagonal_plus(nc)
    P, R = transfer(n, nc, 2.0, n - 1, long_p), transfer(nc, n, 9.0, 17, long_r)
    csr = lambda M: (M.indptr, M.indices, M.data)
    none = np.zeros(0, np.int64)
    mg = MultiGrid.from_csr([{"A": csr(A), "P": csr(P), "R": csr(R), "filter": none}, {"A": csr(Ac), "filter": none}])
    mg.configure(nu=1, coarse="none", precision=prec)
    b = rng.standard_normal(n)
    w = 0.5 / A.diagonal()
    s = w * b
    c = R @ (b - A @ s)
    x = s + P @ c
    z = mg.vcycle(torch.tensor(b).cuda()).cpu().numpy()
    # roundings of every term on its way, as many as the longest rows have entries
    terms = lambda M: abs(M)
    at = abs(w * b) + terms(P) @ (terms(R) @ (abs(b) + terms(A) @ abs(s)))
    at = at + abs(w) * (abs(b) + terms(A) @ at)
    assert np.all(abs(z - (x + w * (b - A @ x))) <= (long_p + long_r + 40) * eps * at)
    mg.close()
