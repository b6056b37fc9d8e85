"""The small end of the V-cycle as one dense operator: one cycle against the oracle's, whose coarse
levels run step by step, for the smoothing counts, coarse solvers and element types the operator is
formed for, on hierarchies whose first level of at most 1,280 rows has one to five levels below it."""
import numpy as np
import pytest
import torch

from oracle import pyoracle as po

pytestmark = pytest.mark.gpu

# dim, degree, level, level_min, nu, coarse
CASES = [(2, 1, 6, 1, 1, "none"), (2, 1, 7, 1, 2, "direct"), (2, 1, 7, 2, 3, "smoother"), (2, 1, 6, 4, 2, "direct"), (3, 1, 5, 1, 2, "direct"),
         (3, 1, 4, 0, 2, "smoother"), (2, 2, 5, 1, 4, "direct"), (3, 2, 3, 1, 2, "none")]


def relerr(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def coefficient(dim, level):
    return np.exp(np.random.default_rng(5).standard_normal((1 << level) ** dim))


def dense_levels(H):
    """per level, finest first: the operator's level, the first below the finest with at most 1,280 rows"""
    n = [H.ndofs(l) for l in range(H.level, H.level_min - 1, -1)]
    at = next(i for i in range(1, len(n)) if n[i] <= 1280)
    assert at < len(n) - 1
    return [i == at for i in range(len(n))]


@pytest.mark.parametrize("case", CASES, ids=["d%dq%dL%d-%d-nu%d-%s" % c for c in CASES])
@pytest.mark.parametrize("fmt", ["sell", "stencil", "matfree"])
def test_cycle_matches_oracle(case, fmt):
    from feat3_b200.solver import MultiGrid
    dim, deg, lvl, lmin, nu, coarse = case
    k = coefficient(dim, lvl)
    H = po.Hierarchy(dim, deg, lvl, lmin, k)
    d = H.rhs("one") * np.random.default_rng(6).uniform(0.5, 1.5, H.ndofs())
    ref = H.vcycle(d, nu=nu, coarse=coarse)
    mg = MultiGrid.structured(dim, deg, lvl, lmin, k)
    dd = torch.tensor(d).cuda()
    first = None
    # FP64 to rounding; FP32 within 100 roundings of 2^-24 (some 50 dependent steps)
    for prec, tol in (("f64", 1e-13), ("f32", 6e-6), ("f64", 1e-13)):
        mg.configure(nu=nu, coarse=coarse, precision=prec, format=fmt)
        assert [mg.level_forms(l)[2] for l in range(mg.num_levels())] == dense_levels(H), prec
        out = mg.vcycle(dd).cpu().numpy()
        assert relerr(out, ref) <= tol, prec
        if prec == "f64":
            first = out if first is None else first
            np.testing.assert_array_equal(out, first)
    # the other cycles do not use the operator; the V-cycle after them does again
    mg.configure(nu=nu, coarse=coarse, format=fmt, cycle="w")
    assert not any(mg.level_forms(l)[2] for l in range(mg.num_levels()))
    mg.vcycle(dd)
    mg.configure(nu=nu, coarse=coarse, format=fmt)
    np.testing.assert_array_equal(mg.vcycle(dd).cpu().numpy(), first)
    assert not mg.vcycle(torch.zeros_like(dd)).any()
    mg.close()


@pytest.mark.parametrize("sigma", [1, 32])
def test_handed_hierarchy_matches_oracle(sigma):
    from feat3_b200.solver import MultiGrid
    H = po.Hierarchy(2, 2, 5, 1, coefficient(2, 5))
    levels = []
    for l in range(5, 0, -1):
        e = {"A": H.csr(l), "filter": H.filter(l)}
        if l > 1:
            e["P"], e["R"] = H.prol(l), H.rest(l)
        levels.append(e)
    d = H.rhs("one")
    mg = MultiGrid.from_csr(levels, sell_sigma=sigma).configure(nu=3)
    assert [mg.level_forms(l)[2] for l in range(mg.num_levels())] == dense_levels(H)
    assert relerr(mg.vcycle(torch.tensor(d).cuda()).cpu().numpy(), H.vcycle(d, nu=3)) <= 1e-13
    mg.close()


@pytest.mark.parametrize("case", CASES, ids=["d%dq%dL%d-%d-nu%d-%s" % c for c in CASES])
@pytest.mark.parametrize("fmt", ["sell", "stencil"])
def test_fp16_cycle(case, fmt):
    """FP16 values above the operator's level, which runs in FP32: against the oracle's cycle on
    unrounded values. The levels above it differ from it by the values' rounding, 2^-11 of each entry
    (two smoothings and a defect per level pass it on)."""
    from feat3_b200.solver import MultiGrid
    dim, deg, lvl, lmin, nu, coarse = case
    k = coefficient(dim, lvl)
    H = po.Hierarchy(dim, deg, lvl, lmin, k)
    d = H.rhs("one") * np.random.default_rng(6).uniform(0.5, 1.5, H.ndofs())
    mg = MultiGrid.structured(dim, deg, lvl, lmin, k)
    mg.configure(nu=nu, coarse=coarse, precision="f16", format=fmt)
    levels = dense_levels(H)
    assert [mg.level_forms(l)[2] for l in range(mg.num_levels())] == levels
    out = mg.vcycle(torch.tensor(d).cuda()).cpu().numpy()
    assert relerr(out, H.vcycle(d, nu=nu, coarse=coarse)) <= 2.0 ** -11 * 2 * (2 * nu + 1) * levels.index(True)
    mg.close()


TINY = [(2, 1, 7, 1, 2, "direct"), (2, 1, 6, 2, 3, "smoother"), (3, 1, 5, 1, 2, "direct"), (2, 2, 5, 1, 1, "none")]


@pytest.mark.parametrize("fmt", ["sell", "matfree"])
@pytest.mark.parametrize("case", TINY, ids=["d%dq%dL%d-%d-nu%d-%s" % c for c in TINY])
def test_tiny_and_non_finite_defects(case, fmt):
    """the operator holds no skip test: a cycle on a defect that could meet one runs level by level"""
    from feat3_b200.solver import MultiGrid
    dim, deg, lvl, lmin, nu, coarse = case
    k = coefficient(dim, lvl)
    H = po.Hierarchy(dim, deg, lvl, lmin, k)
    d = H.rhs("one") * np.random.default_rng(6).uniform(0.5, 1.5, H.ndofs())
    d /= np.linalg.norm(d)
    mg = MultiGrid.structured(dim, deg, lvl, lmin, k)
    for prec, eps, tol in (("f64", 2.0 ** -52, 1e-13), ("f32", 2.0 ** -23, 6e-6)):
        mg.configure(nu=nu, coarse=coarse, precision=prec, format=fmt)
        plain = mg.vcycle(torch.tensor(d).cuda()).cpu().numpy()
        for size in (1e-3, 0.3, 3.0, 30.0, 1e9):  # norms in units of the skip test's eps^2
            t = d * (size * eps ** 2)
            out = mg.vcycle(torch.tensor(t).cuda()).cpu().numpy()
            ref = H.vcycle(t, nu=nu, coarse=coarse, inner=prec)  # (zero where every smoother is left out)
            assert np.linalg.norm(out - ref) <= tol * np.linalg.norm(ref), (prec, size)
        np.testing.assert_array_equal(mg.vcycle(torch.tensor(d).cuda()).cpu().numpy(), plain)
        # iterations of a solve whose small levels meet the test (one eps^2 per point of a side)
        t = d * (H.ndofs() ** (1.0 / dim) * eps ** 2)
        out = mg.configure(nu=nu, coarse=coarse, precision=prec, format=fmt, max_iter=2).solve(torch.tensor(t).cuda())
        ref = H.solve(t, nu=nu, coarse=coarse, inner=prec, max_iter=2)
        np.testing.assert_allclose(out["hist"], ref["hist"], rtol=1e-4 if prec == "f32" else 1e-10)
        if coarse == "smoother":
            for bad in (np.inf, np.nan):
                t = d.copy()
                t[t.size // 2 + 3] = bad
                mg.configure(nu=nu, coarse=coarse, precision=prec, format=fmt)
                with np.errstate(invalid="ignore"):
                    ref = H.vcycle(t, nu=nu, coarse=coarse, inner=prec)
                np.testing.assert_array_equal(mg.vcycle(torch.tensor(t).cuda()).cpu().numpy(), ref)
    mg.close()


def test_operator_follows_the_configuration():
    """the operator is kept over configurations that do not change it and formed again for those that
    do, in each element type: every cycle against the oracle's"""
    from feat3_b200.solver import MultiGrid
    k = coefficient(2, 6)
    H = po.Hierarchy(2, 1, 6, 1, k)
    d = H.rhs("one")
    mg = MultiGrid.structured(2, 1, 6, 1, k)
    base = dict(nu=2, omega_jac=0.5, omega_rich=1.0, coarse="direct")
    runs = [{}, dict(tol=1e-4), dict(nu=3), dict(nu=3, precision="f32"), dict(precision="f32"), {}, dict(omega_jac=0.6),
            dict(omega_rich=0.9), dict(omega_rich=0.9, outer="richardson"), dict(coarse="none"), dict(cycle="w"),
            dict(coarse="none"), dict(precision="f16"), dict(precision="f32", omega_jac=0.6), dict(cgc="energy"), {},
            dict(format="matfree")]
    for run in runs:
        mg.configure(**{**base, **run})
        ref = H.vcycle(d, **{n: v for n, v in {**base, **run}.items() if n in (*base, "cycle", "cgc")})
        out = mg.vcycle(torch.tensor(d).cuda()).cpu().numpy()
        # FP16: values of 11 bits on the finest level
        assert relerr(out, ref) <= {"f64": 1e-13, "f32": 6e-6, "f16": 5e-3}[run.get("precision", "f64")], run
    mg.close()
