"""The FP64 panel column loop on columns of very different size, held column by
column: Householder QR commutes with a scaling of the columns, so with A = A0 D,
D powers of two, the reflectors of the leading columns are A0's and every
other column of R (in their rows) is A0's times its scale.

Bar: 4 n eps ||A0||_F of the column divided by its scale (test_gpu_panel.py's,
per column), plus what the FP64 range itself takes (n 2^-1074 / scale).
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps

# exponents of the leading columns' scale and of the others': products of the
# two that leave the range (both dots and factors), and pairs that do not
SCALES = [(-332, -731), (-399, -631), (-465, -615), (-465, -1000), (-100, -960), (0, -900), (332, -731), (440, -600),
          (440, -1000), (440, 440), (-300, 300), (-465, 440), (0, 0)]


@pytest.fixture(scope="module")
def env():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    H.lib().hqr_set_error_mode(H.HQR_ERRORS_RETURN)
    return torch, H


def scaled(A0, lead, e0, e1):
    """A0 with columns < lead scaled by 2^e0, the others by 2^e1; the scales."""
    e = np.where(np.arange(A0.shape[1]) < lead, e0, e1)
    return np.ldexp(A0, e[None, :]), e


def check(A0, lead, e, r):
    """Rows < lead of R (r: the factored matrix) against A0's, column by column."""
    M, N = A0.shape
    want = np.linalg.qr(A0[:, :lead], mode="complete")
    R0 = (want[0].T @ A0)[:lead]
    got = np.ldexp(np.triu(r)[:lead], -e[None, :])
    # the sign of each row is the reflector's: beta = -sign(alpha) ||.||
    sign = np.sign(np.diag(got[:, :lead])) * np.sign(np.diag(R0[:, :lead]))
    bar = 4 * max(M, N) * EPS * np.linalg.norm(A0) + np.ldexp(float(M), -1074 - e)
    assert (np.abs(got - sign[:, None] * R0).max(axis=0) <= bar).all()


def plan_factor(env, A, NB, IB, precision):
    torch, H = env
    M, N = A.shape
    a = torch.from_numpy(O.to_tiles(A, NB)).cuda()
    tau = torch.zeros((M // NB) * (N // NB) * NB, dtype=torch.float64, device="cuda")
    plan = H.Plan(M, N, NB, IB, precision)
    H.check(H.lib().hqr_geqrf(plan.h, a.data_ptr(), tau.data_ptr(), None), "hqr_geqrf")
    plan.close()
    return O.from_tiles(a.cpu().numpy(), M, N, NB)


@pytest.mark.parametrize("e0,e1", SCALES)
@pytest.mark.parametrize("M,N,NB,IB,lead", [
    (64, 64, 64, 16, 8), (64, 64, 64, 32, 19), (192, 64, 64, 32, 8), (96, 96, 48, 24, 23), (32, 32, 32, 8, 1),
    (512, 256, 256, 32, 30),
])
def test_columns_of_different_size(env, M, N, NB, IB, lead, e0, e1):
    A0 = O.uniform_matrix(M, N, M + N + IB)
    A, e = scaled(A0, lead, e0, e1)
    check(A0, lead, e, plan_factor(env, A, NB, IB, 0))


@pytest.mark.parametrize("e0,e1", SCALES)
def test_batch(env, e0, e1):
    torch, H = env
    shapes = [(64, 32, 32, 8), (128, 128, 128, 16)]
    A0 = [O.uniform_matrix(M, N, M) for M, N, _, _ in shapes]
    A = [scaled(a, 5, e0, e1) for a in A0]
    dA = [torch.from_numpy(O.to_tiles(a, s[2])).cuda() for (a, _), s in zip(A, shapes)]
    dT = [torch.zeros((M // NB) * (N // NB) * NB, dtype=torch.float64, device="cuda") for M, N, NB, _ in shapes]
    batch = H.Batch(*zip(*shapes))
    batch.geqrf([t.data_ptr() for t in dA], [t.data_ptr() for t in dT])
    for a0, (_, e), d, (M, N, NB, _) in zip(A0, A, dA, shapes):
        check(a0, 5, e, O.from_tiles(d.cpu().numpy(), M, N, NB))
    batch.close()


@pytest.mark.parametrize("e0,e1", [s for s in SCALES if s not in ((440, 440), (-465, 440))])
def test_split_panel(env, e0, e1):
    """The panel of the split precision: the columns of its first inner block."""
    _, H = env
    A0 = O.uniform_matrix(256, 128, 11)
    A, e = scaled(A0, 6, e0, e1)
    r = plan_factor(env, A, 128, 32, H.HQR_PREC_OZAKI)
    check(A0[:, :16], 6, e[:16], r[:, :16])


def test_zero_and_padded_columns(env):
    """Columns that are zero, or zero but for rows another column has as zeros: nothing to lift."""
    M = N = 64
    A0 = O.uniform_matrix(M, N, 3)
    A0[:, 20:40] = 0.0
    A0[:32, 5], A0[32:, 6] = 0.0, 0.0
    ra, _ = O.tile_qr(O.to_tiles(A0, 64), M, N, 64, 32)
    got = plan_factor(env, A0, 64, 32, 0)
    assert np.abs(got - O.from_tiles(ra, M, N, 64)).max() <= 4 * N * EPS * np.linalg.norm(A0)
