"""FP64 update tasks narrower than a tile's nominal column block, and panel
blocks whose trailing updates are tasks: where the rules that choose them turn
(one tile, one tile row, few tiles, a tile column with few right-hand sides,
few and many panel tiles), the results are the oracle's and the statistics count what they did before.

Bar: n eps ||.||_F elementwise, as test_gpu_qr.py.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("M,N,NB,IB", [
    (64, 64, 64, 16), (128, 128, 64, 64), (192, 64, 64, 16), (64, 192, 64, 16), (480, 288, 96, 32), (288, 288, 48, 24),
    (640, 640, 128, 32), (1024, 512, 256, 32), (512, 512, 512, 32), (1280, 1280, 32, 8), (1536, 1536, 64, 16),
    # parts of a block's trailing update: 24 columns in three, 32 in four up to two panel tiles an SM, in two beyond
    (144, 96, 48, 24), (96, 96, 32, 32), (64 * 152, 128, 64, 32), (64 * 153, 128, 64, 32), (64 * 160, 128, 64, 32),
])
def test_factor_and_apply(M, N, NB, IB):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    L = H.lib()
    A2d = O.uniform_matrix(M, N, M + 3 * N + NB)
    A = O.to_tiles(A2d, NB)
    ra, rtau = O.tile_qr(A, M, N, NB, IB)
    plan = H.Plan(M, N, NB, IB)
    a = torch.from_numpy(A.copy()).cuda()
    tau = torch.zeros((M // NB) * (N // NB) * NB, dtype=torch.float64, device="cuda")
    H.check(L.hqr_geqrf(plan.h, a.data_ptr(), tau.data_ptr(), None), "hqr_geqrf")
    count = plan.stats()["count"]
    t = max(M, N) * EPS * np.linalg.norm(A2d)
    assert np.abs(a.cpu().numpy() - ra).max() <= t
    assert np.abs(tau.cpu().numpy() - rtau).max() <= t
    steps, MT, NT, nblk = min(M, N) // NB, M // NB, N // NB, NB // min(IB, 32)
    panels = sum(MT - i for i in range(steps))
    assert count[0] == steps * nblk and count[1] == (panels - steps) * nblk
    C2d = O.uniform_matrix(M, NB, 17)
    C = O.to_tiles(C2d, NB)
    want = O.dormqr(ra, rtau, C, M, N, NB, 1)
    c = torch.from_numpy(C.copy()).cuda()
    H.check(L.hqr_ormqr_t(plan.h, a.data_ptr(), tau.data_ptr(), c.data_ptr(), 1, 1, None), "hqr_ormqr_t")
    assert np.abs(c.cpu().numpy() - want).max() <= 4 * max(M, N) * EPS * np.linalg.norm(C2d)
    H.check(L.hqr_ormqr_n(plan.h, a.data_ptr(), tau.data_ptr(), c.data_ptr(), 1, 1, None), "hqr_ormqr_n")
    assert np.abs(c.cpu().numpy() - C).max() <= 8 * max(M, N) * EPS * np.linalg.norm(C2d)
    plan.close()


@pytest.mark.parametrize("nrhs", [1, 8, 17, 64, 65])
@pytest.mark.parametrize("NB", [64, 96, 256])
def test_least_squares_columns(nrhs, NB):
    """Few right-hand sides in a tile column: only their column blocks are tasks; both triangular solves."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    M, N = 3 * NB, 2 * NB
    rng = np.random.default_rng(nrhs + NB)
    A, B = rng.uniform(-1, 1, (M, N)), rng.uniform(-1, 1, (M, nrhs))
    want = np.linalg.lstsq(A, B, rcond=None)[0]
    plan = H.Plan(M, N, NB, 32)
    a = torch.from_numpy(O.to_tiles(A, NB)).cuda()
    b = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
    kappa = np.linalg.cond(A)
    bar = 100 * EPS * kappa * (1 + kappa * np.linalg.norm(B - A @ want) / (np.linalg.norm(A, 2) * np.linalg.norm(want)))
    for augmented in (False, True):
        x = torch.zeros(nrhs, N, dtype=torch.float64, device="cuda")
        plan.lstsq(a.data_ptr(), b.data_ptr(), nrhs, x.data_ptr(), augmented=augmented)
        assert np.linalg.norm(x.cpu().numpy().T - want) <= bar * np.linalg.norm(want)
    plan.close()
