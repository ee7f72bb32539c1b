"""The width of the update tasks of Q generation and Q^T C: Q generation has fewer
updates than Q^T C on as many columns, and the same chain of them, so it takes
no longer, also where the rule for the width sits between chain and work.

Bar: 1.05 times, the spread of the fastest of four runs.
"""
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("MT,NB,IB", [(4, 512, 32), (3, 512, 32), (20, 32, 8), (14, 32, 8), (12, 48, 24), (6, 64, 16),
                                      (6, 128, 32), (4, 256, 32)])
def test_q_generation_takes_no_longer_than_an_application(MT, NB, IB):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    L, n = H.lib(), MT * NB
    s = torch.cuda.current_stream()
    a = torch.from_numpy(O.to_tiles(O.uniform_matrix(n, n, 5), NB)).cuda()
    tau = torch.zeros(MT * n, dtype=torch.float64, device="cuda")
    plan = H.Plan(n, n, NB, IB)
    H.check(L.hqr_geqrf(plan.h, a.data_ptr(), tau.data_ptr(), s.cuda_stream), "hqr_geqrf")

    def fastest(call):
        best = float("inf")
        for _ in range(4):
            c, ry = torch.ones_like(a), a.clone()
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            call(c.data_ptr(), ry.data_ptr())
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best

    q = fastest(lambda c, ry: H.check(L.hqr_make_q_async(plan.h, c, ry, tau.data_ptr(), 1, s.cuda_stream), "make_q"))
    t = fastest(lambda c, ry: H.check(L.hqr_ormqr_t_async(plan.h, ry, tau.data_ptr(), c, MT, 1, s.cuda_stream), "qt"))
    H.check(L.hqr_plan_status(plan.h, s.cuda_stream), "hqr_plan_status")
    plan.close()
    assert q <= 1.05 * t, (q, t)
