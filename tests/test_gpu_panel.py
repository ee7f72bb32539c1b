"""The FP64 panel column loop (GEQRT / TSQRT inner blocks) at its edges, against
the oracle: inner blocks of 8, 16, 24 and 32 columns, tiles whose V chunk fits
the staged buffer and tiles whose does not, one-tile and one-row-of-tiles
shapes; columns that are zero, repeated or tiny; and matrices scaled so far
that the general column loop takes over.

Bar: |gpu - oracle| <= 4 n eps ||A||_F elementwise for R and V (the reflectors'
scalars and sums round differently, each by an ulp or two), 4 n eps for TAU.
"""
import ctypes

import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    H.lib().hqr_set_error_mode(H.HQR_ERRORS_RETURN)
    return torch, H


def factor(env, A, M, N, NB, IB, precision=0):
    torch, H = env
    a = torch.from_numpy(A.copy()).cuda()
    tau = torch.zeros((M // NB) * (N // NB) * NB, dtype=torch.float64, device="cuda")
    plan = H.Plan(M, N, NB, IB, precision)
    H.check(H.lib().hqr_geqrf(plan.h, a.data_ptr(), tau.data_ptr(), None), "hqr_geqrf")
    plan.close()
    return a.cpu().numpy(), tau.cpu().numpy()


def compare(env, A2d, NB, IB):
    M, N = A2d.shape
    A = O.to_tiles(A2d, NB)
    ra, rtau = O.tile_qr(A, M, N, NB, IB)
    a, tau = factor(env, A, M, N, NB, IB)
    scale = np.abs(A2d).max() or 1.0
    n = max(M, N)
    assert np.abs(a - ra).max() / scale <= 4 * n * EPS * max(1.0, np.linalg.norm(A2d / scale))
    assert np.abs(tau - rtau).max() <= 4 * n * EPS


@pytest.mark.parametrize("M,N,NB,IB", [
    (16, 16, 16, 16), (32, 32, 32, 8), (64, 64, 64, 8), (96, 48, 48, 24), (192, 64, 64, 32), (64, 192, 64, 16),
    (128, 128, 128, 32), (256, 128, 128, 16), (288, 144, 144, 16), (288, 288, 144, 24), (512, 256, 256, 32),
    (512, 512, 512, 32),
])
def test_panel_shapes(env, M, N, NB, IB):
    compare(env, O.uniform_matrix(M, N, M + N + IB), NB, IB)


@pytest.mark.parametrize("what", ["zero_columns", "repeated_columns", "tiny_column", "tiny_alpha", "upper"])
def test_special_columns(env, what):
    NB, IB = 64, 16
    A = O.uniform_matrix(2 * NB, NB, 5)
    if what == "zero_columns":
        A[:, [0, 3, 17, 63]] = 0.0
    elif what == "repeated_columns":   # the second copy's remainder is rounding only: R alone is compared
        A[:, 9] = A[:, 8]
    elif what == "tiny_column":        # ||x||^2 below the plain range: LAPACK's rescaling
        A[:, 0] *= 1e-160
    elif what == "tiny_alpha":
        A[0, 0] = 1e-200
    else:                              # nothing below the diagonal: every tau is zero
        A = np.triu(A)
    if what == "repeated_columns":
        M, N = A.shape
        a, _ = factor(env, O.to_tiles(A, NB), M, N, NB, IB)
        R = np.triu(O.from_tiles(a, M, N, NB)[:N])
        assert np.linalg.norm(R.T @ R - A.T @ A) <= 4 * M * EPS * np.linalg.norm(A) ** 2
        return
    compare(env, A, NB, IB)


@pytest.mark.parametrize("scale", [1e-100, 1e100, 1e140, 1e152])
def test_scaled_matrices(env, scale):
    """A scaled by s has R scaled by s, V and TAU unchanged (1e140 and above: the general loop)."""
    M = N = 128
    A = O.uniform_matrix(M, N, 77)
    NB = 64
    a, tau = factor(env, O.to_tiles(A * scale, NB), M, N, NB, 16)
    b, tau1 = factor(env, O.to_tiles(A, NB), M, N, NB, 16)
    x, y = O.from_tiles(a, M, N, NB), O.from_tiles(b, M, N, NB)
    t = 4 * N * EPS * np.linalg.norm(A)
    assert np.abs(np.triu(x) / scale - np.triu(y)).max() <= t
    assert np.abs(np.tril(x, -1) - np.tril(y, -1)).max() <= t
    assert np.abs(tau - tau1).max() <= 4 * N * EPS


def test_not_finite_input_returns(env):
    """A NaN or an infinity spreads; the call still ends with the scheduler's ok."""
    M = N = 128
    for bad in (np.nan, np.inf):
        A = O.uniform_matrix(M, N, 3)
        A[5, 7] = bad
        a, _ = factor(env, O.to_tiles(A, 64), M, N, 64, 16)
        assert np.isnan(np.triu(O.from_tiles(a, M, N, 64))[:, 7:]).any()
