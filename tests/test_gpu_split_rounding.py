"""The split-precision product's rounding, bit for bit.  With one term per output
and operands of at most 30 bits (31 for one of them) every digit pair that is
not zero is kept, so the exact product is rounded once, to nearest even:
ties, carries into the next power of two and both signs among them, for columns
in the middle of the range and for those whose digits take the general path.

At the low end of the range the columns have no subnormal elements and the rows
are large, so that every result is normal and nothing may flush.  Bar there:
K 2^-56 rowmax colmax for the digits that are dropped, and half an ulp.
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


def operands(seed):
    """Integers x (one per row) and y (K x N) of 27 to 30 bits and both signs; a quarter of the rows and
    columns hold pairs whose products are 2^58 - 1 and 2^60 - 1 (all ones: a carry) or odd multiples of
    a half unit in the last place (ties)."""
    rng = np.random.default_rng(seed)
    x = rng.integers(2 ** 26, 2 ** 30, K) * rng.choice([-1, 1], K)
    y = rng.integers(2 ** 26, 2 ** 30, (K, N)) * rng.choice([-1, 1], (K, N))
    x[0::8] = 2 ** 29 - 1
    y[:, 0::8] = 2 ** 29 + 1
    x[1::8] = -(2 ** 30 - 1)
    y[:, 1::8] = 2 ** 30 + 1
    x[2::8] = 2 ** 29 + 2 ** 3                # with y = 2^29 + odd: 59 bits, the lowest set bit is bit 3
    y[:, 2::8] = 2 ** 29 + 2 ** 2 * rng.integers(0, 2 ** 20, (K, N // 8)) * 2 + 2 ** 2
    return x, y


@pytest.mark.parametrize("ex,ey", [(0, 0), (-40, 100), (600, -1000), (-300, 700), (900, -1010)])
def test_one_term_is_rounded_once(product, ex, ey):
    x, y = operands(ex + ey + 5000)
    X = np.zeros((K, K))
    X[np.arange(K), np.arange(K)] = np.ldexp(x.astype(np.float64), ex)
    C = product(X, np.ldexp(y.astype(np.float64), ey))
    exact = [[int(a) * int(b) for b in row] for a, row in zip(x, y)]
    want = np.ldexp(np.array([[float(v) for v in row] for row in exact]), ex + ey)
    # the cases are there
    tie = carry = 0
    for row in exact:
        for v in row:
            drop = abs(v).bit_length() - 53
            tie += drop > 0 and abs(v) % 2 ** drop == 2 ** (drop - 1)
            carry += drop > 0 and abs(v) >> drop == 2 ** 53 - 1 and abs(v) % 2 ** drop > 2 ** (drop - 1)
    assert tie >= 100 and carry >= 100
    assert np.array_equal(C, want)


@pytest.mark.parametrize("scale", [-1021, -1020, -1000, -960, -959, -958])
def test_low_columns_with_normal_results(product, scale):
    rng = np.random.default_rng(3000 + scale)
    X = np.ldexp(rng.uniform(-1, 1, (K, K)), 900)
    Y = np.ldexp(rng.uniform(0.5, 1, (K, N)) * rng.choice([-1, 1], (K, N)), scale)
    C = product(X, Y)
    for r in (0, 31, 127):
        xr = [Fraction(float(v)) for v in X[r]]
        rmax = max(abs(v) for v in xr)
        for c in range(N):
            yc = [Fraction(float(v)) for v in Y[:, c]]
            exact = sum(a * b for a, b in zip(xr, yc))
            bar = K * Fraction(1, 2 ** 56) * rmax * max(abs(v) for v in yc) + abs(exact) * Fraction(1, 2 ** 53)
            assert abs(Fraction(float(C[r, c])) - exact) <= bar, (r, c)


def test_subnormal_columns_are_zero(product):
    rng = np.random.default_rng(9)
    X = np.ldexp(rng.uniform(-1, 1, (K, K)), 1000)
    Y = np.ldexp(rng.uniform(-1, 1, (K, N)), -1023)
    assert not product(X, Y).any()
