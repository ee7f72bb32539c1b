"""The triangular solves of the least-squares calls on factors with elements of
very different size.  A = [R; 0] with R upper triangular is its own
factorization (every tau is zero), and with powers of two in it each step of
the solve is exact: x is compared bit for bit.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    H.lib().hqr_set_error_mode(H.HQR_ERRORS_RETURN)
    return torch, H


def solve(env, R, b, NB, augmented):
    torch, H = env
    N = R.shape[0]
    M = N + NB
    A = np.zeros((M, N))
    A[:N] = R
    B = np.zeros((b.shape[1], M))
    B[:, :N] = b.T
    plan = H.Plan(M, N, NB, 32)
    dA, dB = torch.from_numpy(O.to_tiles(A, NB)).cuda(), torch.from_numpy(B).cuda()
    x = torch.zeros(b.shape[1], N, dtype=torch.float64, device="cuda")
    plan.lstsq(dA.data_ptr(), dB.data_ptr(), b.shape[1], x.data_ptr(), refine_steps=1 if augmented else 0,
               augmented=augmented)
    plan.close()
    return x.cpu().numpy().T


# (row, column, exponents of R(row, col), R(col, col) and the right-hand side's element `col`)
CASES = [(0, 1, 600, -600, -1000), (0, 1, -600, 600, 900), (3, 31, 700, -400, -700), (33, 60, -700, 400, 750),
         (2, 40, 600, -600, -1000), (62, 63, 500, -530, -900), (5, 9, 100, -100, 3), (5, 9, 0, 0, 0)]


@pytest.mark.parametrize("NB", [32, 64, 128])
@pytest.mark.parametrize("r,j,e_rj,e_jj,e_b", CASES)
def test_one_large_ratio(env, NB, r, j, e_rj, e_jj, e_b):
    """R = I but for one column: x_j = b_j / R_jj, x_r = b_r - R_rj x_j; the other right-hand side is zero."""
    N = 128
    R = np.eye(N)
    R[r, j], R[j, j] = np.ldexp(1.0, e_rj), np.ldexp(1.0, e_jj)
    b = np.zeros((N, 2))
    b[j, 0] = np.ldexp(1.0, e_b)
    want = np.zeros((N, 2))
    want[j, 0] = np.ldexp(1.0, e_b - e_jj)
    want[r, 0] = -np.ldexp(1.0, e_rj + e_b - e_jj)
    assert np.isfinite(want).all()
    assert np.array_equal(solve(env, R, b, NB, False), want)


@pytest.mark.parametrize("NB", [32, 64])
@pytest.mark.parametrize("r,j,e_rj,e_jj,e_b", CASES)
def test_one_large_ratio_augmented(env, NB, r, j, e_rj, e_jj, e_b):
    """The refinement's corrections are zero, R^-T of zeros among them."""
    N = 64
    R = np.eye(N)
    R[r, j], R[j, j] = np.ldexp(1.0, e_rj), np.ldexp(1.0, e_jj)
    b = np.zeros((N, 1))
    b[j, 0] = np.ldexp(1.0, e_b)
    got = solve(env, R, b, NB, True)
    assert got[j, 0] == np.ldexp(1.0, e_b - e_jj) and got[r, 0] == -np.ldexp(1.0, e_rj + e_b - e_jj)
    assert np.count_nonzero(got) == 2


@pytest.mark.parametrize("e_jj", [-1022, 1023])
def test_diagonal_near_the_ends(env, e_jj):
    """A diagonal element whose reciprocal is at or below the end of the normal numbers."""
    N = 64
    R = np.eye(N)
    R[7, 7] = np.ldexp(1.0, e_jj)
    b = np.zeros((N, 1))
    b[7, 0], b[8, 0] = np.ldexp(1.0, 1), 4.0
    got = solve(env, R, b, 64, False)
    assert got[8, 0] == 4.0 and np.count_nonzero(np.delete(got[:, 0], [7, 8])) == 0
    assert got[7, 0] == np.ldexp(1.0, 1 - e_jj)
