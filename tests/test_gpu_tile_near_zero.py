"""tile_kernel.h panels with a column whose part below its head is nearly zero:
head = a - ||[a; x]|| is then exactly zero and V = x / 0, as in the reference,
but t = 2 / (head^2 + ||x||^2) is finite and with it R, TAU and the columns
right of it.  In the first columns and in later ones, on panels of one column
loop and on wider ones.

Bar: |gpu - oracle| <= 64 n eps max(1, ||inputs||_F), as test_gpu_tile_kernel.py,
on everything but the infinite column of V.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
TINY = [1e-9, 1e-30, 1e-120]


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


def ge_panel(row, col, c, tiny):
    """Columns < c on rows other than c and a set S; column c: 1 in row c, `tiny` on S, so that it
    reaches its own step as it is; the columns after it dense."""
    rng = np.random.default_rng(row + col + c)
    A = rng.uniform(-1, 1, (row, col))
    S = np.arange(row - 4, row)
    A[S, :c] = 0.0
    A[c, :c] = 0.0
    A[:, c] = 0.0
    A[S, c] = tiny * rng.uniform(0.5, 1, S.size)
    A[c, c] = 1.0
    return np.asfortranarray(A)


def ts_panel(row, col, c, tiny):
    rng = np.random.default_rng(row * col + c)
    R = np.triu(rng.uniform(0.5, 1, (col, col)))
    A = rng.uniform(-1, 1, (row, col))
    S = np.arange(row - 4, row)
    A[S, :c] = 0.0
    A[:, c] = 0.0
    A[S, c] = tiny * rng.uniform(0.5, 1, S.size)
    R[:c, c] = 0.0
    R[c, c] = 1.0
    return np.asfortranarray(R), np.asfortranarray(A)


def others(A, c):
    """A without column c below its diagonal (GE) / without column c (TS: A square or not, all rows)."""
    B = A.copy()
    B[:, c] = 0.0
    return B


@pytest.mark.parametrize("tiny", TINY)
@pytest.mark.parametrize("row,col,c", [(40, 24, 0), (40, 24, 9), (60, 33, 0), (120, 70, 3), (120, 70, 40), (120, 70, 69),
                                       (1000, 30, 0), (1000, 30, 28)])
def test_dgeqr2(H, row, col, c, tiny):
    A0 = ge_panel(row, col, c, tiny)
    A, Ao = A0.copy(order="F"), A0.copy(order="F")
    t, to = np.zeros(col), np.zeros(col)
    Y, Yo = np.zeros((row, col), order="F"), np.zeros((row, col), order="F")
    H.lib().tile_sub_dgeqr2(row, col, P(A), row, P(t), P(Y), None)
    H.check(H.lib().hqr_last_error(), "tile_sub_dgeqr2")
    O.lib().orc_tk_sub_dgeqr2(row, col, O.ptr(Ao), row, O.ptr(to), O.ptr(Yo), O.ptr(np.zeros(3 * row * col)))
    assert not np.isfinite(Ao[c + 1:, c]).all()          # the case is reached
    assert np.isfinite(others(Ao, c)).all()
    b = tol(row, A0)
    assert np.abs(others(A, c) - others(Ao, c)).max() <= b
    assert np.abs(A[:c + 1, c] - Ao[:c + 1, c]).max() <= b
    assert np.abs(others(Y, c) - others(Yo, c)).max() <= b and np.abs(t - to).max() <= b
    assert np.isinf(A[row - 4:, c]).all()


@pytest.mark.parametrize("tiny", TINY)
@pytest.mark.parametrize("row,col,c", [(24, 16, 0), (24, 16, 9), (60, 33, 0), (90, 70, 3), (90, 70, 40), (90, 70, 69),
                                       (1000, 30, 0), (1000, 30, 28)])
def test_dtsqr2(H, row, col, c, tiny):
    R0, A0 = ts_panel(row, col, c, tiny)
    R, Ro, A, Ao = R0.copy(order="F"), R0.copy(order="F"), A0.copy(order="F"), A0.copy(order="F")
    t, to = np.zeros(col), np.zeros(col)
    H.lib().tile_sub_dtsqr2(row, col, P(R), col, P(A), row, P(t), None)
    H.check(H.lib().hqr_last_error(), "tile_sub_dtsqr2")
    O.lib().orc_tk_sub_dtsqr2(row, col, O.ptr(Ro), col, O.ptr(Ao), row, O.ptr(to), O.ptr(np.zeros(3 * row * col)))
    assert not np.isfinite(Ao[:, c]).all() and np.isfinite(Ro).all() and np.isfinite(others(Ao, c)).all()
    b = tol(row + col, R0, A0)
    assert np.abs(np.triu(R) - np.triu(Ro)).max() <= b
    assert np.abs(others(A, c) - others(Ao, c)).max() <= b and np.abs(t - to).max() <= b
    assert np.isinf(A[row - 4:, c]).all()


@pytest.mark.parametrize("c", [0, 20, 50])
def test_one_block_drivers(H, c):
    """tile_dgeqrt / tile_dtsqrt with one block: R and the columns as above (T, of an infinite V, is not held)."""
    row, col, tiny = 96, 64, 1e-12
    A0 = ge_panel(row, col, c, tiny)
    A, Ao = A0.copy(order="F"), A0.copy(order="F")
    t, Y, T = np.zeros(col), np.zeros((row, col), order="F"), np.zeros((col, col), order="F")
    H.lib().tile_dgeqrt(row, col, col, P(A), row, P(t), P(Y), P(T), col, None)
    H.check(H.lib().hqr_last_error(), "tile_dgeqrt")
    O.lib().orc_tk_sub_dgeqr2(row, col, O.ptr(Ao), row, O.ptr(np.zeros(col)), O.ptr(np.zeros((row, col), order="F")),
                              O.ptr(np.zeros(3 * row * col)))
    assert np.abs(others(A, c) - others(Ao, c)).max() <= tol(row, A0)
    R0, B0 = ts_panel(row, col, c, tiny)
    R, Ro, B, Bo = R0.copy(order="F"), R0.copy(order="F"), B0.copy(order="F"), B0.copy(order="F")
    H.lib().tile_dtsqrt(row, col, col, P(R), col, P(B), row, P(t), P(T), col, None)
    H.check(H.lib().hqr_last_error(), "tile_dtsqrt")
    O.lib().orc_tk_sub_dtsqr2(row, col, O.ptr(Ro), col, O.ptr(Bo), row, O.ptr(np.zeros(col)),
                              O.ptr(np.zeros(3 * row * col)))
    assert np.abs(np.triu(R) - np.triu(Ro)).max() <= tol(row + col, R0, B0)
    assert np.abs(others(B, c) - others(Bo, c)).max() <= tol(row + col, R0, B0)


@pytest.mark.parametrize("e", [-500, -300, 300, 480])
def test_scaled_panels(H, e):
    """A scaled by 2^e: R scaled by it, V and TAU unchanged, as long as the squares stay in range; one
    column loop and three."""
    row, col = 100, 70
    A0 = np.asfortranarray(np.random.default_rng(5).uniform(-1, 1, (row, col)))
    out = []
    for s in (0, e):
        A = np.asfortranarray(np.ldexp(A0, s))
        t, Y = np.zeros(col), np.zeros((row, col), order="F")
        H.lib().tile_sub_dgeqr2(row, col, P(A), row, P(t), P(Y), None)
        H.check(H.lib().hqr_last_error(), "tile_sub_dgeqr2")
        out.append((np.ldexp(np.triu(A), -s), Y, t))
    b = tol(row, A0)
    for x, y in zip(*out):
        assert np.abs(x - y).max() <= b
