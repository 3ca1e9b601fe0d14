"""The trim's flood where its forms meet: boxes of 31, 32 and 33 voxels along x, supervoxels one
and two voxels from the x and y borders and on them, one-voxel rows, long winding paths, islands
above the threshold, all five neighbourhoods; the volume and the list form bit for bit the host
oracle's arrays."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
DIMS = (96, 80, 24)


def _volume(seed):
    """Box-shaped supervoxels with bright winding paths on a dim ground."""
    rng = np.random.default_rng(seed)
    X, Y, Z = DIMS
    lab = np.zeros((Z, Y, X), np.uint32)
    raw = rng.integers(100, 130, size=(Z, Y, X)).astype(np.uint16)
    boxes = [(0, 31, 0, 9, 0, 6), (1, 32, 10, 9, 0, 6), (2, 33, 20, 9, 0, 6), (X - 31, 31, 0, 9, 0, 6),
             (X - 33, 32, 10, 9, 0, 6), (X - 35, 33, 20, 9, 0, 6), (40, 20, 0, 12, 8, 9), (40, 20, 1 + 12, 12, 8, 9),
             (40, 20, Y - 13, 12, 8, 9), (62, 1, 30, 30, 8, 10), (5, 30, 32, 1, 2, 20), (8, 25, 40, 25, 0, 20),
             (64, 30, 36, 30, 7, 12), (3, 60, 68, 6, 1, 5)]
    n = 0
    for x, w, y, h, z, d in boxes:
        sl = (slice(z, z + d), slice(y, y + h), slice(x, x + w))
        part = lab[sl]
        if part.any():
            continue
        n += 1
        lab[sl] = np.where(rng.random(part.shape) < 0.92, n, 0)
        r = raw[sl]
        r[:] = rng.integers(200, 320, size=r.shape)
        p = [d // 2, h // 2, w // 2]
        for _ in range(w * h * d // 3):  # a winding bright path
            a = rng.integers(0, 3)
            p[a] = int(np.clip(p[a] + rng.choice([-1, 1]), 0, r.shape[a] - 1))
            r[tuple(p)] = rng.integers(600, 1200)
        r[rng.random(r.shape) < 0.03] = 900  # islands
    return np.ascontiguousarray(raw), np.ascontiguousarray(lab), n


@pytest.mark.parametrize("conn", [4, 6, 8, 26, 74])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_flood_forms_match_the_host_build(cuda_ok, seed, conn):
    import torch
    from tgmm_b200 import engine as E
    raw, lab, n = _volume(seed)
    rc, want = O.frame_build(raw, lab, n, O.frame_params(conn=conn, min_size=20))
    assert rc == 0
    b = E.FrameBuilder(DIMS, n, conn3d=conn, min_nuclei_size=20)
    rd = torch.from_numpy(raw.reshape(-1).view(np.int16)).cuda()
    ld = torch.from_numpy(lab.reshape(-1).view(np.int32)).cuda()
    lin = np.concatenate([np.flatnonzero(lab.reshape(-1) == k + 1) for k in range(n)])
    ptr = np.concatenate([[0], np.cumsum([(lab == k + 1).sum() for k in range(n)])]).astype(np.int64)
    lists = (torch.from_numpy(lin.astype(np.int32)).cuda(),
             torch.from_numpy(raw.reshape(-1)[lin].view(np.int16)).cuda(), torch.from_numpy(ptr).cuda())
    for got, thr in (b.build(rd, ld), b.build_lists(*lists)):
        out = [t.cpu().numpy() for t in (got.query, got.img, got.centroids, got.label_ptr)]
        for key, g in zip(("query", "img", "cent", "lptr"), out):
            np.testing.assert_array_equal(g, want[key], err_msg=key)
        np.testing.assert_array_equal(thr, want["thr"])
