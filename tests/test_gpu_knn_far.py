"""The standalone kNN where a query's neighbours lie many cells away: references in one corner of
the queries' box, in a few spots of one slice and at one end of a line along each axis, with some
queries whose coordinates are NaN or infinite; both query forms, bit for bit against the oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_knn_k import SCALE, gpu_knn_k

pytestmark = pytest.mark.gpu


def layout(kind, nq, nref, rng):
    """(queries, references), each 3 x n."""
    q, r = rng.uniform(0, 1000, (3, nq)), rng.uniform(0, 1000, (3, nref))
    if kind == "corner":
        r = r * 0.04
    elif kind == "slice":  # one plane: references in eight spots
        q[2], r[2] = 3, 3
        r[:2] = rng.uniform(0, 1000, (2, 8))[:, rng.integers(0, 8, nref)] + rng.normal(0, 4, (2, nref))
    else:  # a line along one axis, references on its first twentieth
        a = "xyz".index(kind[-1])
        for p in (q, r):
            for d in range(3):
                if d != a:
                    p[d] = 7
            p[a] *= 20
        r[a] *= 0.05
    q = np.round(q, 1)
    odd = rng.choice(nq, 60, replace=False)
    q[rng.integers(0, 3, 60), odd] = np.tile([np.nan, np.inf, -np.inf], 20)
    return q.astype(np.float32), np.round(r, 1).astype(np.float32), odd


@pytest.mark.parametrize("kind", ["corner", "slice", "line x", "line y", "line z"])
@pytest.mark.parametrize("nq,nref,k", [(20000, 20000, 1), (20000, 20000, 11), (20000, 60000, 5), (100033, 20000, 5),
                                       (100033, 60000, 11)])
def test_knn_of_far_queries(cuda_ok, kind, nq, nref, k):
    rng = np.random.default_rng(nq + nref + k)
    q, r, odd = layout(kind, nq, nref, rng)
    gi, gd = gpu_knn_k(np.ascontiguousarray(q.reshape(-1)), np.ascontiguousarray(r.reshape(-1)), k)
    pick = np.unique(np.concatenate([rng.choice(nq, 400, replace=False), odd, [0, nq - 1]]))
    oi, od = O.knn_topk(np.ascontiguousarray(q[:, pick].reshape(-1)), np.ascontiguousarray(r.reshape(-1)), k, SCALE)
    np.testing.assert_array_equal(gi.reshape(k, nq)[:, pick], oi.reshape(k, -1))
    np.testing.assert_array_equal(gd.reshape(k, nq)[:, pick], od.reshape(k, -1))
