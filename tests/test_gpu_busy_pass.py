"""The voxel pass that also runs the next iteration's kNN/E-step, on a plan for far more
supervoxels than the frame has, so that most of its blocks own none, while other streams keep the
SMs busy: such a block may find a place only after the others have ended the frame.  It has to
leave the pass's work counters as the rest do; every later call on the plan depends on them."""
import numpy as np
import pytest

import _fixtures as F

pytestmark = pytest.mark.gpu
CALLS = 150


@pytest.mark.parametrize("iters,tol", [(20, 1e-4), (3, -1.0)])
def test_idle_blocks_on_a_busy_device_leave_the_work_counters(cuda_ok, iters, tol):
    import torch
    from tgmm_b200 import _lib as L
    from tgmm_b200 import engine as E
    f = F.frame("moved")
    df, start, prm = E.to_device(f), E.gauss_to_device(f.gauss), F.params(iters, tol=tol)

    def plan(fused):
        p = E.Plan(f.n_vox, 2000, f.n_gauss)
        p.set_knn_group(8)
        p.set_knn_fusion(fused)
        return p

    def buffers():
        return start.clone(), torch.empty(5 * f.n_sv, device="cuda"), torch.empty(5 * f.n_sv, dtype=torch.int32,
                                                                                 device="cuda")

    apart = plan(False)
    gm, rnk, ind = buffers()
    stats = apart.run_device(df, gm, rnk, ind, prm)
    want = E.gauss_from_device(gm), rnk.cpu().numpy(), ind.cpu().numpy()
    apart.close()

    plans, streams = [plan(True), plan(True)], [torch.cuda.Stream(), torch.cuda.Stream()]
    busy = torch.cuda.Stream()
    a = torch.randn(4096, 4096, device="cuda", dtype=torch.bfloat16)
    c = torch.empty_like(a)
    outs = [[buffers() for _ in range(CALLS)] for _ in plans]
    torch.cuda.synchronize()
    for i in range(CALLS):
        with torch.cuda.stream(busy):
            for _ in range(4):
                torch.mm(a, a, out=c)
        for p, st, o in zip(plans, streams, outs):
            p.run_device(df, *o[i], prm, stats=False, stream=st)
    torch.cuda.synchronize()
    for p, o in zip(plans, outs):
        for gm, rnk, ind in o:
            assert L.records_equal(E.gauss_from_device(gm), want[0])
            assert np.array_equal(rnk.cpu().numpy(), want[1]) and np.array_equal(ind.cpu().numpy(), want[2])
        gm, rnk, ind = buffers()
        got = p.run_device(df, gm, rnk, ind, prm)
        assert {k: v for k, v in got.items() if k != "knn_searches"} == {
            k: v for k, v in stats.items() if k != "knn_searches"}
        p.close()
