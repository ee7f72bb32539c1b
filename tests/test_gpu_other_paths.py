"""The kernels that take the sizes the faster ones do not: the triangular solves
of tile orders that 32 does not divide or above 256, and tile_kernel.h panels
that are taller than a column loop's shared memory (narrower loops, and column
by column through global memory).

Bars: test_gpu_columns.py's and test_gpu_tile_kernel.py's.
"""
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


@pytest.mark.parametrize("nrhs", [1, 9])
@pytest.mark.parametrize("NB", [16, 48, 80, 272, 320])
def test_least_squares_other_tile_orders(env, NB, nrhs):
    torch, H = env
    M, N = 3 * NB, 2 * NB
    rng = np.random.default_rng(nrhs + NB)
    A, B = rng.uniform(-1, 1, (M, N)), rng.uniform(-1, 1, (M, nrhs))
    want = np.linalg.lstsq(A, B, rcond=None)[0]
    plan = H.Plan(M, N, NB, 16)
    a = torch.from_numpy(O.to_tiles(A, NB)).cuda()
    b = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
    kappa = np.linalg.cond(A)
    bar = 100 * EPS * kappa * (1 + kappa * np.linalg.norm(B - A @ want) / (np.linalg.norm(A, 2) * np.linalg.norm(want)))
    for augmented in (False, True):
        x = torch.zeros(nrhs, N, dtype=torch.float64, device="cuda")
        plan.lstsq(a.data_ptr(), b.data_ptr(), nrhs, x.data_ptr(), augmented=augmented)
        assert np.linalg.norm(x.cpu().numpy().T - want) <= bar * np.linalg.norm(want)
    plan.close()


# 845 rows: the last that 32 columns fit; 27056: the last that one column fits
TALL = [(845, 40), (846, 40), (5000, 12), (14000, 3), (27056, 3), (27057, 3), (30000, 5)]


def P(a):
    return a.ctypes.data


def tol(n, *arrays):
    return 64 * n * EPS * max([1.0] + [float(np.linalg.norm(a)) for a in arrays])


@pytest.mark.parametrize("row,col", TALL)
def test_tall_dgeqr2(env, row, col):
    _, H = env
    A0 = np.asfortranarray(np.random.default_rng(row + col).uniform(-1, 1, (row, col)))
    A, Ao = A0.copy(order="F"), A0.copy(order="F")
    t, to = np.zeros(col), np.zeros(col)
    Y, Yo = np.zeros((row, col), order="F"), np.zeros((row, col), order="F")
    H.lib().tile_sub_dgeqr2(row, col, P(A), row, P(t), P(Y), None)
    H.check(H.lib().hqr_last_error(), "tile_sub_dgeqr2")
    O.lib().orc_tk_sub_dgeqr2(row, col, O.ptr(Ao), row, O.ptr(to), O.ptr(Yo), O.ptr(np.zeros(3 * row * col)))
    b = tol(row, A0)
    assert np.abs(A - Ao).max() <= b and np.abs(t - to).max() <= b and np.abs(Y - Yo).max() <= b


@pytest.mark.parametrize("row,col", TALL)
def test_tall_dtsqr2(env, row, col):
    _, H = env
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
