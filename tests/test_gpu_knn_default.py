"""An untouched plan takes its kNN/E-step's width and arrangement from its capacity in
supervoxels: at each side of the rule's lines a call gives the bits of the eight-lane kernel of
its own, with a fixed iteration count and with a tolerance (knn_searches counts the work of the
path taken, the two search forms keeping lists of different lengths)."""
import numpy as np
import pytest

import _fixtures as F
from tgmm_b200 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,tol,fp64", [("tiny", -1.0, False), ("c1", -1.0, False), ("moved", -1.0, False),
                                           ("hard", 0.0, False), ("moved", 1e-6, False), ("moved", -1.0, True)])
@pytest.mark.parametrize("capacity", [0, 1000, 1001, 3000, 3001, 6000, 6001])
def test_default_width_gives_the_same_bits(cuda_ok, name, tol, fp64, capacity):
    from tgmm_b200 import engine as E
    f = F.frame(name)
    df = E.to_device(f)
    prm = F.params(12, tol)
    if fp64:
        prm.ll_precision = L.TGMM_LLPREC_FP64
    out = []
    for by_hand in (False, True):
        plan = E.Plan(f.n_vox, max(capacity, f.n_sv), f.n_gauss)
        try:
            if by_hand:
                plan.set_knn_group(8)
                plan.set_knn_fusion(False)
                assert plan.tuning() == {"knn_lanes": 8, "knn_fused": False}
            out.append(plan.run_host(df, f.gauss, prm))
        finally:
            plan.close()
    a, b = out
    assert L.records_equal(a["gauss"], b["gauss"])
    for k in a:
        if k not in ("gauss", "knn_searches"):
            assert np.array_equal(a[k], b[k]), k
