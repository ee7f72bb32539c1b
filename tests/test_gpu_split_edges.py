"""The split-precision product (digits, tensor-core products, recombination) at
the ends of its range, against exact rational arithmetic: columns whose largest
element is subnormal, below 2^-959, near 2^1023; rows and columns of zeros;
elements 2^-60 .. 2^-64 below their column's largest; single-element products
that need every rounding case; results that underflow and overflow.

Bar, per element: half an ulp of the exact result, plus K 2^-56 rowmax colmax
for the digits' truncation and the dropped products; results below 2^-1021 may
flush to zero, and subnormal elements count as zero.
"""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
K, N = 128, 64


@pytest.fixture(scope="module")
def product():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H

    def run(X, Y):
        x = torch.from_numpy(np.ascontiguousarray(X.T)).cuda()
        y = torch.from_numpy(np.ascontiguousarray(Y.T)).cuda()
        c = torch.empty(N, K, dtype=torch.float64, device="cuda")
        H.check(H.lib().hqr_ozaki_product(K, x.data_ptr(), y.data_ptr(), c.data_ptr(), None), "hqr_ozaki_product")
        return c.cpu().numpy().T
    return run


def check(C, X, Y, rows):
    for r in rows:
        xr = [Fraction(float(v)) for v in X[r]]
        rmax = max(abs(v) for v in xr)
        for c in range(N):
            yc = [Fraction(float(v)) for v in Y[:, c]]
            exact = sum(a * b for a, b in zip(xr, yc) if a and b)
            cmax = max(abs(v) for v in yc)
            bar = K * Fraction(1, 2 ** 56) * rmax * cmax + abs(exact) * Fraction(1, 2 ** 53)
            bar += K * Fraction(1, 2 ** 1022) * (rmax + cmax) + Fraction(1, 2 ** 1021)
            got = float(C[r, c])
            if abs(exact) >= Fraction(2) ** 1024:
                assert np.isinf(got) and (got > 0) == (exact > 0), (r, c)
            else:
                assert abs(Fraction(got) - exact) <= bar, (r, c, got, float(exact))


@pytest.mark.parametrize("scale", [-1070, -1022, -1021, -960, -959, -500, 0, 900])
def test_column_scales(product, scale):
    rng = np.random.default_rng(scale + 2000)
    X, Y = rng.uniform(-1, 1, (K, K)), np.ldexp(rng.uniform(-1, 1, (K, N)), scale)
    X[:, 5] = 0.0
    X[9] = 0.0
    Y[:, 3] = 0.0
    check(product(X, Y), X, Y, [0, 9, 127])


def test_element_spreads(product):
    """Elements far below their column's (row's) largest, both signs, zeros and subnormals among them."""
    rng = np.random.default_rng(1)
    X = np.ldexp(rng.uniform(0.5, 1, (K, K)) * rng.choice([-1, 1], (K, K)), rng.integers(-70, 1, (K, K)))
    Y = np.ldexp(rng.uniform(0.5, 1, (K, N)) * rng.choice([-1, 1], (K, N)), rng.integers(-70, 1, (K, N)))
    X[:, 0], Y[0] = 1.0, -1.0
    X[:, 1], Y[1] = 0.0, -0.0
    X[:, 2], Y[2] = 5e-324, 1e-310
    check(product(X, Y), X, Y, [0, 64])


def test_rounding_and_range_ends(product):
    """One term per output: the product of two doubles, rounded once (or flushed, or infinite)."""
    rng = np.random.default_rng(2)
    X, Y = np.zeros((K, K)), np.zeros((K, N))
    X[np.arange(K), np.arange(K)] = rng.integers(2 ** 52, 2 ** 53, K) * np.where(np.arange(K) % 2, 1.0, -1.0)
    for c in range(N):
        Y[:, c] = rng.integers(2 ** 52, 2 ** 53, K)
    Y[:, 1] = 2.0 ** 52                    # exact
    Y[:, 2] = 3 * 2.0 ** 51 + 1            # ties and near ties
    Y[:, 3] = 2.0 ** 53 - 1
    Y = np.ldexp(Y, np.array([-104, 970, -1074, -1126][:4] * 16))
    X = np.ldexp(X, -52)
    check(product(X, Y), X, Y, [0, 1, 2, 3, 126, 127])
