"""The captured EM with a tolerance: the first iterations unconditionally, the later ones in nested
conditional graph nodes of growing length.  Bit for bit the kernel-by-kernel form for iteration
limits at and around the nodes' ends, and for frames that converge inside each of them."""
import numpy as np
import pytest

import _fixtures as F

pytestmark = pytest.mark.gpu


def _run(name, iters, tol):
    import torch
    from tgmm_b200 import engine as E
    f = F.frame(name)
    df, gm = E.to_device(f), E.gauss_to_device(f.gauss)
    rnk = torch.empty(5 * f.n_sv, device="cuda")
    ind = torch.empty(5 * f.n_sv, dtype=torch.int32, device="cuda")
    plan = E.Plan(f.n_vox, f.n_sv, f.n_gauss)
    out = []
    for _ in range(2):
        gm.copy_(E.gauss_to_device(f.gauss))
        st = plan.run_device(df, gm, rnk, ind, F.params(iters, tol=tol))
        out.append((E.gauss_from_device(gm), rnk.cpu().numpy(), ind.cpu().numpy(), st))
    plan.close()
    return out


@pytest.mark.parametrize("name,iters,tol", [("small", 1, 0.0), ("small", 3, 1e-30), ("small", 4, 1e-30),
                                            ("moved", 5, 1e-30), ("moved", 8, 1e-30), ("moved", 9, 0.0),
                                            ("hard", 40, 0.0), ("small", 400, 1e-6), ("hard", 400, 1e-9)])
def test_nested_conditional_iterations_change_no_bit(cuda_ok, monkeypatch, name, iters, tol):
    from tgmm_b200 import _lib as L
    graph = _run(name, iters, tol)
    monkeypatch.setenv("TGMM_NO_GRAPH", "1")
    eager = _run(name, iters, tol)
    for a in graph:
        assert L.records_equal(a[0], eager[0][0])
        assert np.array_equal(a[1], eager[0][1]) and np.array_equal(a[2], eager[0][2])
        assert a[3] == eager[0][3]
