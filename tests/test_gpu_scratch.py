"""Scratch of the standalone calls: small requests come from the library's own pool, larger ones
and captured streams from the default pool.  The same results on either side of the line, from
several threads on streams of their own, and from a captured graph."""
import threading

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _inputs(nq, nref, seed):
    import torch
    rng = np.random.default_rng(seed)
    q = rng.uniform(0, 300, 3 * nq).astype(np.float32)
    r = rng.uniform(0, 300, 3 * nref).astype(np.float32)
    return torch.from_numpy(q).cuda(), torch.from_numpy(r).cuda(), O.knn(q, r)


def test_knn_around_the_pool_line_from_threads_on_their_own_streams(cuda_ok):
    import torch
    from tgmm_b200 import engine as E
    jobs = [_inputs(700, n, i) for i, n in enumerate((5, 300, 26000, 26500, 40000))]
    torch.cuda.synchronize()
    bad = []

    def work(n):
        st = torch.cuda.Stream()
        for rep in range(6):
            q, r, want = jobs[(n + rep) % len(jobs)]
            with torch.cuda.stream(st):
                got = E.knn(q, r, stream=st)
                st.synchronize()
            if not np.array_equal(got.cpu().numpy(), want):
                bad.append((n, rep))

    threads = [threading.Thread(target=work, args=(n,)) for n in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_knn_in_a_captured_graph(cuda_ok):
    import torch
    from tgmm_b200 import engine as E
    q, r, want = _inputs(900, 500, 9)
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=st):
        got = E.knn(q, r, stream=st)
    for _ in range(2):
        got.fill_(-1)
        g.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(got.cpu().numpy(), want)
