"""Q^T C with one reflector tile of order 512: its chain is one task long, so the
tasks are narrowed only while all of them fit the SMs at once.

Bar: 3 and 4 tile columns are then one wave of tasks of 16 columns, and 1 is one
of 8, each of which reads all of V: at most 1.6 times the time.  Two waves of
the narrow tasks are about twice it.
"""
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
NB = 512


@pytest.mark.parametrize("CT", [3, 4])
def test_one_wave(CT):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    L, s = H.lib(), torch.cuda.current_stream()
    a = torch.from_numpy(O.to_tiles(O.uniform_matrix(NB, NB, 5), NB)).cuda()
    tau = torch.zeros(NB, dtype=torch.float64, device="cuda")
    plan = H.Plan(NB, NB, NB, 64)
    H.check(L.hqr_geqrf(plan.h, a.data_ptr(), tau.data_ptr(), s.cuda_stream), "hqr_geqrf")
    best = {}
    for ct in (1, CT):
        c = torch.ones(NB * NB * ct, dtype=torch.float64, device="cuda")
        best[ct] = float("inf")
        for _ in range(5):
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            H.check(L.hqr_ormqr_t_async(plan.h, a.data_ptr(), tau.data_ptr(), c.data_ptr(), ct, 1, s.cuda_stream), "qt")
            e1.record()
            torch.cuda.synchronize()
            best[ct] = min(best[ct], e0.elapsed_time(e1))
    H.check(L.hqr_plan_status(plan.h, s.cuda_stream), "hqr_plan_status")
    plan.close()
    assert best[CT] <= 1.6 * best[1], best


def test_one_wave_a_link():
    """Two tiles down a column, the same bar: 192 narrow tasks a tile would be two waves for each."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    L, s = H.lib(), torch.cuda.current_stream()
    a = torch.from_numpy(O.to_tiles(O.uniform_matrix(2 * NB, NB, 5), NB)).cuda()
    tau = torch.zeros(2 * NB, dtype=torch.float64, device="cuda")
    plan = H.Plan(2 * NB, NB, NB, 64)
    H.check(L.hqr_geqrf(plan.h, a.data_ptr(), tau.data_ptr(), s.cuda_stream), "hqr_geqrf")
    best = {}
    for ct in (1, 3):
        c = torch.ones(2 * NB * NB * ct, dtype=torch.float64, device="cuda")
        best[ct] = float("inf")
        for _ in range(5):
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            H.check(L.hqr_ormqr_t_async(plan.h, a.data_ptr(), tau.data_ptr(), c.data_ptr(), ct, 1, s.cuda_stream), "qt")
            e1.record()
            torch.cuda.synchronize()
            best[ct] = min(best[ct], e0.elapsed_time(e1))
    H.check(L.hqr_plan_status(plan.h, s.cuda_stream), "hqr_plan_status")
    plan.close()
    assert best[3] <= 1.6 * best[1], best
