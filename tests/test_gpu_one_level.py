"""Hierarchies of one level with the direct coarse solver: a cycle is the product with the inverse of
the filtered matrix, whatever the cycle, the element type and the format; and a two-level hierarchy
below the dense small end's row limit, configured back and forth between the V- and the W-cycle."""
import numpy as np
import pytest
import scipy.sparse as sp
import torch

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

EPS = {"f64": 2.0 ** -53, "f32": 2.0 ** -24, "f16": 2.0 ** -24}  # (FP16 values, FP32 inverse)


def check(mg, A, filt, formats):
    """cycles and solves of the one-level hierarchy mg against the dense inverse"""
    n = A.shape[0]
    free = np.setdiff1d(np.arange(n), filt)
    F = A.toarray()[np.ix_(free, free)]
    inv = np.zeros((n, n))
    inv[np.ix_(free, free)] = np.linalg.inv(F)
    rng = np.random.default_rng(n)
    d = rng.uniform(0.5, 1.5, n)
    d[filt] = 0.0
    u = np.linalg.solve(F, d[free])
    cond = np.linalg.cond(F)
    dd = torch.tensor(d).cuda()
    for fmt in formats:
        for prec in ("f64", "f32", "f16"):
            for cyc in ("v", "f", "w"):
                mg.configure(nu=2, precision=prec, cycle=cyc, format=fmt, tol=1e-10)
                z = mg.vcycle(dd).cpu().numpy()
                # the rounding of the inverse, the vector and the result; two eliminations in FP64
                lim = 4 * EPS[prec] * (abs(inv) @ abs(d)) + 2 * n * EPS["f64"] * cond * np.linalg.norm(inv @ d)
                assert np.all(abs(z - inv @ d) <= lim), (fmt, prec, cyc)
                s = mg.solve(dd)
                assert s["status"] == "success", (fmt, prec, cyc)
                got = s["u"].cpu().numpy()
                # ||u - u*|| <= ||A^-1|| ||r|| <= cond 1e-10 ||u*||
                assert np.linalg.norm(got[free] - u) <= 1.1 * cond * 1e-10 * np.linalg.norm(u), (fmt, prec, cyc)
    mg.close()


@pytest.mark.parametrize("n,nfilt", [(1, 0), (2, 1), (5, 1), (8, 0), (31, 3), (130, 2)])
def test_handed_over(n, nfilt):
    from feat3_b200.solver import MultiGrid
    rng = np.random.default_rng(n)
    B = sp.random(n, n, min(1.0, 4.0 / n), random_state=rng, format="csr")
    A = sp.csr_matrix(B @ B.T + sp.identity(n))
    A.sort_indices()
    filt = np.sort(rng.choice(n, nfilt, replace=False))
    mg = MultiGrid.from_csr([{"A": (A.indptr, A.indices, A.data), "filter": filt}])
    check(mg, A, filt, ["sell"])


@pytest.mark.parametrize("dim,degree,level", [(2, 1, 1), (2, 1, 4), (2, 2, 3), (3, 1, 2), (3, 2, 2), (2, 1, 5)])
def test_structured(dim, degree, level):
    from feat3_b200.solver import MultiGrid
    k = np.exp(np.random.default_rng(9).standard_normal((1 << level) ** dim))
    H = po.Hierarchy(dim, degree, level, level, k)
    rp, ci, va = H.csr(level)
    A = sp.csr_matrix((va, ci, rp), shape=(len(rp) - 1,) * 2)
    mg = MultiGrid.structured(dim, degree, level, level, k)
    check(mg, A, H.filter(level), ["sell", "stencil", "matfree"])


def test_two_small_levels_between_v_and_w():
    """289 rows over 81: the operator's level has to lie above the coarsest one, so none is formed"""
    from feat3_b200.solver import MultiGrid
    k = np.exp(np.random.default_rng(9).standard_normal(16 ** 2))
    H = po.Hierarchy(2, 1, 4, 3, k)
    d = H.rhs("one")
    mg = MultiGrid.structured(2, 1, 4, 3, k)
    dd = torch.tensor(d).cuda()
    for cyc in ("v", "w", "v", "f", "v"):
        mg.configure(nu=2, cycle=cyc)
        z = mg.vcycle(dd).cpu().numpy()
        ref = H.vcycle(d, nu=2, cycle=cyc)
        assert np.linalg.norm(z - ref) <= 1e-13 * np.linalg.norm(ref), cyc
    mg.close()
