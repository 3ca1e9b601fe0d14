"""The two forms of the standalone kNN's query kernel (a group of lanes per query, a warp per 32
queries) on the layouts where they can go wrong, bit for bit against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_knn_k import SCALE, gpu_knn_k

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["rows", "scattered", "clumped", "lattice", "far", "nonfinite"])
@pytest.mark.parametrize("nq,k", [(31, 1), (99999, 5), (100000, 11), (100033, 5)])
def test_knn_both_query_forms_on_every_layout(cuda_ok, kind, nq, k):
    """The group form (fewer than 100,000 queries) and the warp form, on queries that lie in
    rows as a supervoxel's voxels do, scattered, clumped beyond what a search keeps, on a
    lattice (equal distances), outside the references, and with NaN and infinite coordinates;
    bit for bit against the oracle on a sample of the queries."""
    rng = np.random.default_rng(nq + 7 * k)
    nref = 900
    r = rng.uniform(0, 200, size=(3, nref)).astype(np.float32)
    own = np.arange(nq) * nref // nq
    q = np.round(r[:, own] + rng.normal(0, 4, size=(3, nq))).astype(np.float32)
    if kind == "scattered":
        q = rng.uniform(-20, 220, size=(3, nq)).astype(np.float32)
    elif kind == "clumped":
        r[:, :400] = r[:, :1] + rng.normal(0, 0.05, size=(3, 400)).astype(np.float32)
        r[:, 400:440] = r[:, :1]
    elif kind == "lattice":
        r, q = np.round(r / 8) * 8, np.round(q / 4) * 4
    elif kind == "far":
        q = q + np.float32(5000)
    elif kind == "nonfinite":
        q[rng.integers(0, 3, 40), rng.integers(0, nq, 40)] = np.nan
        q[0, rng.integers(0, nq, 5)] = np.inf
        r[0, :3] = np.nan
    q, r = np.ascontiguousarray(q.reshape(-1)), np.ascontiguousarray(r.reshape(-1))
    gi, gd = gpu_knn_k(q, r, k)
    pick = np.unique(np.concatenate([np.arange(0, nq, max(1, nq // 1500)), np.arange(nq - min(nq, 40), nq)]))
    if kind == "nonfinite":
        pick = np.unique(np.concatenate([pick, np.flatnonzero(~np.isfinite(q.reshape(3, nq)).all(0))]))
    qs = np.ascontiguousarray(q.reshape(3, nq)[:, pick].reshape(-1))
    oi, od = O.knn_topk(qs, r, k, SCALE)
    np.testing.assert_array_equal(gi.reshape(k, nq)[:, pick], oi.reshape(k, -1))
    np.testing.assert_array_equal(gd.reshape(k, nq)[:, pick], od.reshape(k, -1))
