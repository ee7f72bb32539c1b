"""hqr_geqrf_noalloc and plans launch the same kernel: a small tile's call must
not lower the shared memory that a larger tile's launches were given.

Bar: bit for bit the factorization before it.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NB,IB", [(256, 32), (512, 32)])
def test_small_noalloc_between_larger_plans(NB, IB):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    L = H.lib()
    H.lib().hqr_set_error_mode(H.HQR_ERRORS_RETURN)
    A = torch.from_numpy(O.to_tiles(O.uniform_matrix(2 * NB, NB, 5), NB)).cuda()
    small = torch.from_numpy(O.to_tiles(O.uniform_matrix(64, 32, 6), 32)).cuda()
    tau, stau = torch.zeros(2 * NB, dtype=torch.float64, device="cuda"), torch.zeros(64, dtype=torch.float64, device="cuda")
    plan = H.Plan(2 * NB, NB, NB, IB)
    out = []
    for _ in range(2):
        a = A.clone()
        torch.cuda.synchronize()
        H.check(L.hqr_geqrf(plan.h, a.data_ptr(), tau.data_ptr(), None), "hqr_geqrf")
        out.append(a.cpu().numpy())
        s = small.clone()
        torch.cuda.synchronize()
        H.check(L.hqr_geqrf_noalloc(64, 32, 32, 8, s.data_ptr(), stau.data_ptr(), None), "hqr_geqrf_noalloc")
    plan.close()
    assert np.array_equal(*out)
