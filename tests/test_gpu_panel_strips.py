"""A panel block that applies itself to the rest of its tile does so in the
tile's nominal column blocks, whatever the width of the update tasks.  On tall
matrices of few tile columns, where the update tasks are narrow and the first
steps' panel blocks are whole, a panel block takes as long as in a batch of the
same matrix, whose update tasks have the nominal width.

Bar: 1.25 times.  The last step's panel blocks, half of them at most, apply
themselves in tasks of parts of their columns, a third more work: (1 + 4/3) / 2
= 1.17, and 7 % for the spread of two runs.
"""
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("MT,NB,IB", [(2000, 64, 16), (700, 128, 16), (700, 128, 32)])
def test_whole_panel_blocks_keep_their_strips(MT, NB, IB):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import hybrid3_gb300 as H
    M, N = MT * NB, 2 * NB
    a0 = torch.from_numpy(O.uniform_matrix(M * 2, NB, 1).ravel().copy()).cuda()
    tau = torch.zeros(MT * 2 * NB, dtype=torch.float64, device="cuda")
    plan, batch = H.Plan(M, N, NB, IB), H.Batch([M], [N], [NB], [IB], ctas_per_sm=1)
    each = []
    for p in (plan, batch):
        for _ in range(2):
            a = a0.clone()
            torch.cuda.synchronize()
            if p is plan:
                H.check(H.lib().hqr_geqrf(plan.h, a.data_ptr(), tau.data_ptr(), None), "hqr_geqrf")
            else:
                batch.geqrf([a.data_ptr()], [tau.data_ptr()])
        st = p.stats()
        each.append(st["cycles"][1] / st["count"][1])
        p.close()
    assert each[0] <= 1.25 * each[1], each
