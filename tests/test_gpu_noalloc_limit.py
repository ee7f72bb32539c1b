"""hqr_geqrf_noalloc at the end of its fixed scratch: the largest square matrix
of a tile order that it takes (found by asking; larger ones are refused) is
factored as hqr_geqrf factors it, bit for bit, twice over what the first call
left there.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NB,IB,rows", [(32, 8, 1), (64, 16, 1), (128, 32, 1), (256, 32, 1), (64, 32, 20)])
def test_largest_matrix(NB, IB, rows):
    """rows: tile rows for each tile column."""
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    L = H.lib()
    L.hqr_set_error_mode(H.HQR_ERRORS_RETURN)
    NT = int((64 * 2**20 / 8 / rows) ** 0.5) // NB + 1   # one tile column more than T alone could fill
    big = torch.zeros(rows * NT * NT * NB * NB, dtype=torch.float64, device="cuda")
    big_tau = torch.zeros(rows * NT * NT * NB, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    refused = 0
    while True:
        M, N = rows * NT * NB, NT * NB
        rc = L.hqr_geqrf_noalloc(M, N, NB, IB, big.data_ptr(), big_tau.data_ptr(), None)
        if rc != H.HQR_ERR_UNSUPPORTED:
            break
        refused += 1
        NT -= 1
    assert rc == H.HQR_OK and refused >= 1
    A = torch.from_numpy(O.to_tiles(O.uniform_matrix(M, N, NB + rows), NB)).cuda()
    plan = H.Plan(M, N, NB, IB)
    want, wtau = A.clone(), torch.zeros(rows * NT * NT * NB, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    H.check(L.hqr_geqrf(plan.h, want.data_ptr(), wtau.data_ptr(), None), "hqr_geqrf")
    plan.close()
    for _ in range(2):
        a, tau = A.clone(), torch.zeros_like(wtau)
        torch.cuda.synchronize()
        H.check(L.hqr_geqrf_noalloc(M, N, NB, IB, a.data_ptr(), tau.data_ptr(), None), "hqr_geqrf_noalloc")
        assert np.array_equal(a.cpu().numpy(), want.cpu().numpy())
        assert np.array_equal(tau.cpu().numpy(), wtau.cpu().numpy())
