"""Vector kernels of the operator layer on aligned and unaligned vectors, in place and not, over sizes
around the 16-byte packs, the grid's step and the lengths from which 16-byte accesses are taken:
bitwise against torch for the single-operation kernels, within one rounding of the sum for axpy, and
the FP64-accumulated dot and norm."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 1023, 4099, 606208 * 2 + 5, 3000001, 5000003, 6250002,
                               10000001])
@pytest.mark.parametrize("dtype,eps", [(torch.float64, 2.0 ** -53), (torch.float32, 2.0 ** -24)])
def test_vectors(dtype, eps, n, shift):
    from feat3_b200.lafem import DenseVector
    g = torch.Generator("cuda").manual_seed(n + shift)
    x, y, r = (torch.randn(n + 4, dtype=dtype, device="cuda", generator=g)[s:s + n] for s in (shift, 0, shift))
    y = y + 3.0 * torch.sign(y)
    X, Y, R = DenseVector(x), DenseVector(y), DenseVector(r)
    assert torch.equal(R.component_product(X, Y).t, x * y)
    assert torch.equal(R.component_invert(Y, 0.5).t, 0.5 / y)
    assert torch.equal(R.scale(X, -2.5).t, -2.5 * x)
    a = 0.75  # exact in both types; a x + y with one or two roundings
    ref = a * x.double() + y.double()
    assert torch.all((R.axpy(X, Y, a).t.double() - ref).abs() <= 2 * eps * ((a * x.double()).abs() + y.double().abs()))
    assert torch.equal(DenseVector(x.clone()).axpy(X, Y, a).t, r)
    z = y.clone()  # in place
    Z = DenseVector(z)
    assert torch.equal(Z.axpy(X, Z, a).t, r)
    assert torch.equal(R.axpy(X, Y, 0.0).t, y)
    xd, yd = x.double(), y.double()
    # n additions in FP64 over at most n / 64 partials per thread and a tree: far below n eps
    bound = 2.0 ** -53 * 64 * (xd * yd).abs().sum().item()
    assert abs(X.dot(Y) - np.sum((xd * yd).cpu().numpy())) <= bound
    assert abs(X.norm2() - torch.linalg.vector_norm(xd).item()) <= 2.0 ** -53 * 64 * torch.linalg.vector_norm(xd).item()
    assert X.dot(Y) == X.dot(Y)
