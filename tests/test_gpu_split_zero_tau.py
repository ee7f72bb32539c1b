"""The triangular factors T behind the split-precision updates, where reflectors
are missing: columns of zeros (tau = 0) at and beside the edges of the blocks of
16, 32 and 64 columns that T is built from, whole blocks of them, and tile rows
of zeros (every tau of the tile is 0).

Bar: 8 m eps ||.||_F elementwise for Q R - A, for Q^T A below its diagonal and for
Q Q^T C - C.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps
NB = 128


@pytest.mark.parametrize("zero,zero_rows", [
    ([], 0), ([0], 0), ([127], 1), ([15, 16, 17, 31, 32, 33], 0), ([63, 64, 65, 127, 128, 191, 192], 2),
    (list(range(16, 32)), 0), (list(range(64, 128)), 1), (list(range(1, 128)), 0), (list(range(0, 256, 2)), 0),
])
def test_zero_columns(zero, zero_rows):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    L = H.lib()
    M, N = 4 * NB, 2 * NB
    A2d = O.uniform_matrix(M, N, 40 + len(zero))
    A2d[:, zero] = 0.0
    if zero_rows:
        A2d[M - zero_rows * NB:] = 0.0
    plan = H.Plan(M, N, NB, 32, H.HQR_PREC_OZAKI)
    a = torch.from_numpy(O.to_tiles(A2d, NB)).cuda()
    tau = torch.zeros((M // NB) * (N // NB) * NB, dtype=torch.float64, device="cuda")
    H.check(L.hqr_geqrf(plan.h, a.data_ptr(), tau.data_ptr(), None), "hqr_geqrf")
    taus = tau.cpu().numpy().reshape(N // NB, M // NB, NB)
    for j in zero:
        assert (taus[j // NB, :, j % NB] == 0).all()
    R2d = np.triu(O.from_tiles(a.cpu().numpy(), M, N, NB))

    def apply(x2d, fn):
        c = torch.from_numpy(O.to_tiles(x2d, NB)).cuda()
        H.check(fn(plan.h, a.data_ptr(), tau.data_ptr(), c.data_ptr(), x2d.shape[1] // NB, 1, None), "apply")
        return O.from_tiles(c.cpu().numpy(), M, x2d.shape[1], NB)
    bar = 8 * M * EPS
    assert np.abs(apply(R2d, L.hqr_ormqr_n) - A2d).max() <= bar * np.linalg.norm(A2d)
    assert np.abs(np.tril(apply(A2d, L.hqr_ormqr_t), -1)).max() <= bar * np.linalg.norm(A2d)
    C2d = O.uniform_matrix(M, NB, 17)
    assert np.abs(apply(apply(C2d, L.hqr_ormqr_t), L.hqr_ormqr_n) - C2d).max() <= bar * np.linalg.norm(C2d)
    plan.close()
