"""The FP64 log-likelihood, which takes a supervoxel in four parts: voxels of zero density inside
and outside the reference's kept window, whole strides of them, on supervoxel sizes around its
tiles (256 voxels) and the window (1024), at the FP64 mode's 1e-9 against the oracle; a batch
beside the frames alone, bit for bit."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_ll_stream import SIZES, _frame, _run

pytestmark = pytest.mark.gpu


def _zeros(f, kind, rng):
    """Moves voxels far from every Gaussian: their density is zero."""
    x = f.query.reshape(3, -1)
    if kind == "spread":
        far = rng.choice(x.shape[1], 200, replace=False)
    else:
        far = []
        for s, n in enumerate(SIZES):
            a = int(f.label_ptr[s])
            if kind == "window":  # the kept window's last fifth
                far += range(a + n - n // 5, a + n)
            elif kind == "strides" and n > 1024:  # whole strides of 1024, and some but their first
                far += [i for t in range(0, 40) for i in range(a + t, a + n, 1024)]
                far += [i for t in range(60, 90) for i in range(a + t + 1024, a + n, 1024)]
            elif kind == "all" and s % 5 == 0:
                far += range(a, a + n)
    x[:, np.array(sorted(set(far)), np.int64)] += 4000
    return f


# (supervoxels that are far as a whole ("all") stretch their Gaussians until hundreds of densities
# are subnormal, where one unit of rounding is a large part of the value: the oracle is no measure
# there, and they are compared with themselves in a batch only)
@pytest.mark.parametrize("kind", ["spread", "window", "strides"])
@pytest.mark.parametrize("w4dof", [1, 0])
def test_zero_densities_in_four_parts(cuda_ok, kind, w4dof):
    from tgmm_b200 import _lib as L
    f = _zeros(_frame(14.0, 0, 3 + w4dof, general=not w4dof), kind, np.random.default_rng(8))
    st = _run([f], w4dof=w4dof, ll_precision=L.TGMM_LLPREC_FP64)[0]
    for mode, got in ((O.LL_TRUE, st["ll_true"]), (O.LL_AS_REFERENCE, st["ll_as_reference"])):
        want = O.em_run(f.query, f.img, f.centroids, f.label_ptr, f.gauss,
                        O.params(max_iter=3, tol=-1.0, w4dof=w4dof, ll_mode=mode))["ll_hist"][-1]
        assert abs(got - want) <= 1e-9 * abs(want), (mode, got, want)


def test_batch_and_alone_are_the_same_bits_in_fp64(cuda_ok):
    from tgmm_b200 import _lib as L
    rng = np.random.default_rng(4)
    frames = [_zeros(_frame(s, 0, i), k, rng) for i, (s, k) in enumerate([(3.0, "window"), (14.0, "strides"),
                                                                          (60.0, "all")])]
    batch = _run(frames, ll_precision=L.TGMM_LLPREC_FP64)
    for f, b in zip(frames, batch):
        a = _run([f], ll_precision=L.TGMM_LLPREC_FP64)[0]
        assert (a["ll_true"], a["ll_as_reference"]) == (b["ll_true"], b["ll_as_reference"])
