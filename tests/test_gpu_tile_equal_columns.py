"""tile_kernel.h panels with columns that are multiples of one another: what is left
of such a column is rounding errors, not zero, so its own reflector does not
divide by zero (the convention has no guard), and R is as good as ever.

The oracle's R is finite on all of these panels, but in general all the errors of
a column can be zero by chance; so at least three in four results are finite (with
one factor for a column's change it is about every second), and those have R^T
R within 8 (row + col) eps ||panel||_F^2 of the panel's Gram matrix, twice the
backward error bound of a Householder QR with 4 (row + col) eps.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
SHAPES = [(40, 40), (60, 30), (100, 70), (300, 33), (900, 40)]


@pytest.fixture(scope="module")
def H():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300
    return hybrid3_gb300


def panel(row, col, seed, equal):
    rng = np.random.default_rng(seed)
    A, R = rng.uniform(-1, 1, (row, col)), np.triu(rng.uniform(-1, 1, (col, col)))
    for M in (A, R):
        if equal == "first":
            M[:, 1] = M[:, 0]
        else:
            M[:, 9], M[:, col - 1] = 2 * M[:, 8], M[:, 4]
    return np.asfortranarray(A), np.asfortranarray(np.triu(R))


def hold(R, Ro, gram, row, col):
    assert np.isfinite(Ro).all()
    if not np.isfinite(R).all():
        return False
    bound = 8 * (row + col) * np.finfo(float).eps * np.trace(gram)
    assert np.linalg.norm(R.T @ R - gram) <= bound
    return True


@pytest.mark.parametrize("equal", ["first", "some"])
@pytest.mark.parametrize("row,col", SHAPES)
def test_equal_columns(H, row, col, equal):
    finite, p, work = 0, O.ptr, np.zeros(3 * row * col)
    for seed in range(8):
        A0, R0 = panel(row, col, seed, equal)
        for one_block in (False, True):
            A, Ao, t, T = A0.copy(order="F"), A0.copy(order="F"), np.zeros(col), np.zeros((col, col), order="F")
            Y, Yo = np.zeros((row, col), order="F"), np.zeros((row, col), order="F")
            if one_block:
                H.lib().tile_dgeqrt(row, col, col, p(A), row, p(t), p(Y), p(T), col, None)
            else:
                H.lib().tile_sub_dgeqr2(row, col, p(A), row, p(t), p(Y), None)
            H.check(H.lib().hqr_last_error(), "geqr2")
            O.lib().orc_tk_sub_dgeqr2(row, col, p(Ao), row, p(np.zeros(col)), p(Yo), p(work))
            finite += hold(np.triu(A)[:col], np.triu(Ao)[:col], A0.T @ A0, row, col)
            A, Ao, R, Ro = A0.copy(order="F"), A0.copy(order="F"), R0.copy(order="F"), R0.copy(order="F")
            if one_block:
                H.lib().tile_dtsqrt(row, col, col, p(R), col, p(A), row, p(t), p(T), col, None)
            else:
                H.lib().tile_sub_dtsqr2(row, col, p(R), col, p(A), row, p(t), None)
            H.check(H.lib().hqr_last_error(), "tsqr2")
            O.lib().orc_tk_sub_dtsqr2(row, col, p(Ro), col, p(Ao), row, p(np.zeros(col)), p(work))
            finite += hold(np.triu(R), np.triu(Ro), R0.T @ R0 + A0.T @ A0, row, col)
    assert finite >= 24   # of 32
