"""tile_kernel.h's column loops and applications where their work is cut: panels
wider than one column loop (33, 64, 100 columns), blocks that do not divide the
tile, more columns than one round of thread blocks, one-column and one-row
arguments, and T with values stored above its diagonal.

Bar: |gpu - oracle| <= 64 n eps max(1, ||inputs||_F), as test_gpu_tile_kernel.py.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def H():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    H.lib().hqr_set_error_mode(H.HQR_ERRORS_RETURN)
    return H


def P(a):
    return a.ctypes.data


def tol(n, *arrays):
    return 64 * n * EPS * max([1.0] + [float(np.linalg.norm(a)) for a in arrays])


@pytest.mark.parametrize("row,col", [(100, 100), (100, 99), (130, 64), (64, 33), (40, 1), (1, 1), (2, 2)])
def test_dgeqr2_widths(H, row, col):
    A0 = np.asfortranarray(np.random.default_rng(row + col).uniform(-1, 1, (row, col)))
    A, Ao = A0.copy(order="F"), A0.copy(order="F")
    t, to = np.full(col, 7.0), np.full(col, 7.0)
    Y, Yo = np.zeros((row, col), order="F"), np.zeros((row, col), order="F")
    H.lib().tile_sub_dgeqr2(row, col, P(A), row, P(t), P(Y), None)
    H.check(H.lib().hqr_last_error(), "tile_sub_dgeqr2")
    O.lib().orc_tk_sub_dgeqr2(row, col, O.ptr(Ao), row, O.ptr(to), O.ptr(Yo), O.ptr(np.zeros(3 * row * col)))
    b = tol(row, A0)
    assert np.abs(A - Ao).max() <= b and np.abs(t - to).max() <= b and np.abs(Y - Yo).max() <= b


@pytest.mark.parametrize("row,col", [(100, 70), (48, 33), (1, 1), (5, 64)])
def test_dtsqr2_widths(H, row, col):
    rng = np.random.default_rng(row * col)
    R0 = np.asfortranarray(np.triu(rng.uniform(-1, 1, (col, col))))
    A0 = np.asfortranarray(rng.uniform(-1, 1, (row, col)))
    R, Ro, A, Ao = R0.copy(order="F"), R0.copy(order="F"), A0.copy(order="F"), A0.copy(order="F")
    t, to = np.zeros(col), np.zeros(col)
    H.lib().tile_sub_dtsqr2(row, col, P(R), col, P(A), row, P(t), None)
    H.check(H.lib().hqr_last_error(), "tile_sub_dtsqr2")
    O.lib().orc_tk_sub_dtsqr2(row, col, O.ptr(Ro), col, O.ptr(Ao), row, O.ptr(to), O.ptr(np.zeros(3 * row * col)))
    b = tol(row + col, R0, A0)
    assert np.abs(np.triu(R) - np.triu(Ro)).max() <= b and np.abs(A - Ao).max() <= b and np.abs(t - to).max() <= b


@pytest.mark.parametrize("row,k,cols", [(33, 7, 1), (64, 64, 400), (300, 5, 3), (1, 1, 1)])
def test_dlarfb_and_dssrfb_columns(H, row, k, cols):
    """Against the formulas of the two applications (T lower), in numpy."""
    rng = np.random.default_rng(row + k + cols)
    F = np.asfortranarray
    Y = F(np.tril(rng.uniform(-1, 1, (row, k))) / row)
    T = F(rng.uniform(-1, 1, (k, k)))           # the strict upper part is not used
    A0 = F(rng.uniform(-1, 1, (row, cols)))
    A = A0.copy(order="F")
    H.lib().tile_sub_dlarfb(row, k, cols, P(Y), row, P(T), k, P(A), row, None)
    H.check(H.lib().hqr_last_error(), "tile_sub_dlarfb")
    assert np.abs(A - (A0 - Y @ (np.tril(T) @ (Y.T @ A0)))).max() <= tol(row, A0, T)
    V = F(rng.uniform(-1, 1, (row, k)) / row)
    C1, C2 = F(rng.uniform(-1, 1, (k, cols))), F(rng.uniform(-1, 1, (row, cols)))
    D1, D2 = C1.copy(order="F"), C2.copy(order="F")
    H.lib().tile_sub_dssrfb(k, row, k, cols, P(V), row, P(T), k, P(D1), k, P(D2), row, None)
    H.check(H.lib().hqr_last_error(), "tile_sub_dssrfb")
    W = np.tril(T) @ (C1 + V.T @ C2)
    b = tol(row + k, C1, C2, T)
    assert np.abs(D1 - (C1 - W)).max() <= b and np.abs(D2 - (C2 - V @ W)).max() <= b


def test_dlarft_reads_the_stored_upper_part(H):
    """The reference's recurrence sums T(c, r) for every c < i, the stored upper part included."""
    row, col = 50, 37
    rng = np.random.default_rng(9)
    Y = np.asfortranarray(rng.uniform(-1, 1, (row, col)) / row)
    tau = rng.uniform(0, 2, col)
    T = np.asfortranarray(np.triu(rng.uniform(-1, 1, (col, col)), 1))
    want = T.copy()
    G = Y.T @ Y
    for i in range(col):
        want[i, i] = tau[i]
    for i in range(1, col):
        want[i, :i] = [-tau[i] * (want[:i, r] @ G[i, :i]) for r in range(i)]
    H.lib().tile_sub_dlarft(row, col, P(Y), row, P(tau), P(T), col, None)
    H.check(H.lib().hqr_last_error(), "tile_sub_dlarft")
    assert np.abs(T - want).max() <= tol(row, want)
