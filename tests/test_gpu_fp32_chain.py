"""FP32-class factorizations whose panel chain sets the pace: FP32 panel blocks
take half the time of the split precision's FP64 ones and the products fewer
digits, so the factorization takes no longer than the split one's.

Bar: 1.05 times, the spread of the fastest of four runs.  The results: ||R^T R -
A^T A|| within 1e-3 of ||A||^2, the class's precision at these sizes.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
NB = 128


@pytest.mark.parametrize("MT,NT", [(2, 2), (12, 12), (30, 6), (10, 40), (100, 3), (64, 8), (256, 4), (48, 48)])
def test_no_longer_than_the_split_precision(MT, NT):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    L, M, N = H.lib(), MT * NB, NT * NB
    s = torch.cuda.current_stream()
    a0 = torch.empty(M * N, dtype=torch.float64, device="cuda")
    H.check(L.hqr_fill_uniform(M, N, NB, 7, a0.data_ptr(), s.cuda_stream), "hqr_fill_uniform")
    tau = torch.zeros(MT * N, dtype=torch.float64, device="cuda")
    times = []
    for precision in (H.HQR_PREC_FP32, H.HQR_PREC_OZAKI):
        plan, best = H.Plan(M, N, NB, 32, precision), float("inf")
        for _ in range(4):
            a = a0.clone()
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            H.check(L.hqr_geqrf_async(plan.h, a.data_ptr(), tau.data_ptr(), s.cuda_stream), "hqr_geqrf_async")
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        H.check(L.hqr_plan_status(plan.h, s.cuda_stream), "hqr_plan_status")
        plan.close()
        times.append(best)
        if precision == H.HQR_PREC_FP32:
            A = torch.from_numpy(O.from_tiles(a0.cpu().numpy(), M, N, NB)).cuda()
            R = torch.triu(torch.from_numpy(O.from_tiles(a.cpu().numpy(), M, N, NB)).cuda())[:min(M, N)]
            err = torch.linalg.norm(R.T @ R - A.T @ A) / torch.linalg.norm(A) ** 2
            assert float(err) <= 1e-3
    assert times[0] <= 1.05 * times[1], times
