"""The FP32 log-likelihood pass at its edges, against the FP64 oracle at the mixed mode's 1e-6
relative: supervoxel sizes around its units (128 voxels), blocks (512) and the reference's kept
window (1024), empty ones, Gaussians crowded, near and far apart (one to five candidates kept),
both covariance forms, voxels of zero density inside and outside the kept window, a fixed
Gaussian whose precision is indefinite, and a batch beside the frames alone (bit for bit)."""
import numpy as np
import pytest

import _fixtures as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu
SIZES = [0, 1, 31, 32, 127, 128, 129, 255, 257, 511, 512, 513, 640, 1023, 1024, 1025, 1151, 1152, 1153, 1537, 2100, 3]


def _frame(spread, outliers, seed, general=False):
    from tgmm_b200 import _lib as L
    from tgmm_b200 import synth
    rng = np.random.default_rng(seed)
    S = len(SIZES)
    centre = rng.uniform(0, spread * S ** (1 / 3), size=(S, 3)) + 40
    lp = np.concatenate([[0], np.cumsum(SIZES)]).astype(np.int64)
    sv = np.repeat(np.arange(S), SIZES)
    x = np.round(centre[sv] + rng.normal(0, 3, size=(sv.size, 3)))
    if outliers:  # far from every Gaussian: a density of zero
        x[rng.choice(sv.size, outliers, replace=False)] += 4000
    img = rng.uniform(0.05, 1, sv.size).astype(np.float32)
    g = np.zeros(S, L.GAUSS_DTYPE)
    n = rng.uniform(60, 400, S)
    g["m_k"] = centre + rng.normal(0, 1, (S, 3))
    g["m_o"] = g["m_k"]
    for k in ("beta_k", "nu_k", "alpha_k"):
        g[k] = n
    for k in ("beta_o", "nu_o", "alpha_o"):
        g[k] = 0.3 * n + 4
    W = np.zeros((S, 6))
    W[:, 0], W[:, 3], W[:, 5] = rng.uniform(0.06, 0.2, (3, S))
    W[:, 1] = 0.02 * rng.uniform(-1, 1, S)
    if general:
        W[:, 2], W[:, 4] = 0.02 * rng.uniform(-1, 1, (2, S))
    g["W_k"], g["W_o"] = W / n[:, None], W / g["nu_o"][:, None]
    cent = np.ascontiguousarray(centre.T.astype(np.float32).reshape(-1))
    return synth.Frame(np.ascontiguousarray(x.T.astype(np.float32).reshape(-1)), img, cent, lp,
                       np.arange(S, dtype=np.int32), 1.0, gauss=g)


def _run(frames, **kw):
    import torch
    from tgmm_b200 import engine as E
    dfs, gms = [E.to_device(f) for f in frames], [E.gauss_to_device(f.gauss) for f in frames]
    rnk = [torch.empty(5 * f.n_sv, device="cuda") for f in frames]
    ind = [torch.empty(5 * f.n_sv, dtype=torch.int32, device="cuda") for f in frames]
    plan = E.Plan(sum(f.n_vox for f in frames), sum(f.n_sv for f in frames), sum(f.n_gauss for f in frames),
                  max_frames=len(frames))
    st = plan.run_batch(dfs, gms, rnk, ind, F.params(3, **kw))
    plan.close()
    return st


@pytest.mark.parametrize("spread", [3.0, 14.0, 60.0])
@pytest.mark.parametrize("w4dof", [1, 0])
@pytest.mark.parametrize("outliers", [0, 60])
def test_log_likelihood_at_the_edges(cuda_ok, spread, w4dof, outliers):
    f = _frame(spread, outliers, int(spread) + outliers + w4dof, general=not w4dof)
    st = _run([f], w4dof=w4dof)[0]
    for mode, got in ((O.LL_TRUE, st["ll_true"]), (O.LL_AS_REFERENCE, st["ll_as_reference"])):
        want = O.em_run(f.query, f.img, f.centroids, f.label_ptr, f.gauss,
                        O.params(max_iter=3, tol=-1.0, w4dof=w4dof, ll_mode=mode))["ll_hist"][-1]
        assert abs(got - want) <= 1e-6 * abs(want), (mode, got, want)


def test_indefinite_precision_of_a_fixed_gaussian(cuda_ok):
    """Two negative eigenvalues: a positive determinant, no Cholesky factor."""
    f = _frame(60.0, 0, 5)
    f.gauss["fixed"][5] = 1
    W = f.gauss["W_k"][5]
    f.gauss["W_k"][5] = [-W[0] * 1e-3, 0, 0, -W[3] * 1e-3, 0, W[5]]
    st = _run([f])[0]
    want = O.em_run(f.query, f.img, f.centroids, f.label_ptr, f.gauss, O.params(max_iter=3, tol=-1.0))["ll_hist"][-1]
    assert abs(st["ll"] - want) <= 1e-6 * abs(want), (st["ll"], want)


def test_batch_and_alone_are_the_same_bits(cuda_ok):
    frames = [_frame(3.0, 9, 1), _frame(14.0, 0, 2), _frame(60.0, 30, 3)]
    batch = _run(frames)
    for f, b in zip(frames, batch):
        a = _run([f])[0]
        assert (a["ll_true"], a["ll_as_reference"]) == (b["ll_true"], b["ll_as_reference"])
