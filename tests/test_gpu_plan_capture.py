"""After a factorization on a plan, its Q generation and the applications to up
to N columns enqueue kernels and memsets only: they need no more scheduler
tables than the factorization reserved, so they can be captured into a CUDA
graph by their first call.  Where the applications' tasks are narrower than the
factorization's (few tile columns, a domain tree) as elsewhere.

Bar: 4 n eps ||C||_F elementwise against the same calls outside a graph.
"""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("M,N,NB,IB,CT,tree,prec", [
    (512, 512, 32, 32, 9, 0, 0), (800, 704, 32, 32, 13, 0, 0), (256, 256, 64, 16, 4, 0, 0),
    (768, 192, 64, 32, 3, 4, 0), (512, 512, 128, 32, 4, 2, 0), (1024, 256, 128, 32, 2, 2, 1), (512, 512, 128, 32, 4, 0, 1),
])
def test_apply_and_make_q_in_a_graph(M, N, NB, IB, CT, tree, prec):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    L = H.lib()
    A = torch.from_numpy(O.to_tiles(O.uniform_matrix(M, N, 3), NB)).cuda()
    C0 = torch.from_numpy(O.to_tiles(O.uniform_matrix(M, CT * NB, 4), NB)).cuda()
    tau = torch.zeros((M // NB) * (N // NB) * NB, dtype=torch.float64, device="cuda")
    c, q, ry = C0.clone(), torch.zeros(M * N, dtype=torch.float64, device="cuda"), torch.zeros_like(A)
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    plan = H.Plan(M, N, NB, IB, prec)
    if tree:
        plan.set_tree(tree)

    def calls():
        H.check(L.hqr_ormqr_t_async(plan.h, A.data_ptr(), tau.data_ptr(), c.data_ptr(), CT, 1, s.cuda_stream),
                "hqr_ormqr_t_async")
        if not (prec and not tree):   # (a split plan's operands of H are allocated by their first use)
            H.check(L.hqr_make_q_async(plan.h, q.data_ptr(), ry.data_ptr(), tau.data_ptr(), 1, s.cuda_stream),
                    "hqr_make_q_async")

    H.check(L.hqr_geqrf(plan.h, A.data_ptr(), tau.data_ptr(), s.cuda_stream), "hqr_geqrf")
    ry.copy_(A)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        calls()
    g.replay()
    torch.cuda.synchronize()
    H.check(L.hqr_plan_status(plan.h, s.cuda_stream), "hqr_plan_status")
    got_c, got_q = c.clone(), q.clone()
    c.copy_(C0)
    q.zero_()
    ry.copy_(A)
    torch.cuda.synchronize()
    calls()
    H.check(L.hqr_plan_status(plan.h, s.cuda_stream), "hqr_plan_status")
    bar = 4 * max(M, N) * EPS * float(C0.norm())
    assert float((got_c - c).abs().max()) <= bar
    assert float((got_q - q).abs().max()) <= bar
    plan.close()
