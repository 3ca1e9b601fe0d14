"""The trim's flood where a supervoxel's box exceeds shared memory (65536 voxels) and the reached
bits lie in the workspace: in a workspace that holds anything, in repeated builds, and for pixel
lists that hold the same voxels, each of which is trimmed as if it were alone."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
X, Y = 70, 66


def _part(rng, depth):
    """A supervoxel of a box of 60 x 56 x depth: bright paths and islands on a dim ground."""
    shape = (depth, 56, 60)
    own = rng.random(shape) < 0.9
    own[0, 0, 0] = own[-1, -1, -1] = True
    raw = rng.integers(200, 320, size=shape).astype(np.uint16)
    p = [depth // 2, 28, 30]
    for _ in range(own.size // 6):
        a = rng.integers(0, 3)
        p[a] = int(np.clip(p[a] + rng.choice([-1, 1]), 0, shape[a] - 1))
        raw[tuple(p)] = rng.integers(600, 1200)
    raw[rng.random(shape) < 0.03] = 900
    raw[depth // 2, 24:33, 26:35] = 700  # around the brightest voxel: every form keeps the part
    raw[depth // 2, 28, 30] = 2000
    own[depth // 2, 24:33, 26:35] = True
    return own, raw


def _volume(parts, z0):
    """The parts at depths z0 of a volume, labelled in order (they must not overlap)."""
    depth = max(z + own.shape[0] for z, (own, _) in zip(z0, parts)) + 2
    lab, raw = np.zeros((depth, Y, X), np.uint32), np.full((depth, Y, X), 90, np.uint16)
    for i, (z, (own, r)) in enumerate(zip(z0, parts)):
        sl = slice(z, z + own.shape[0]), slice(4, 60), slice(5, 65)
        assert not lab[sl].any()
        lab[sl] = np.where(own, i + 1, 0)
        raw[sl] = np.where(own, r, raw[sl])
    return raw, lab


def _lists(parts, z0):
    """The same supervoxels as pixel lists; here they may overlap."""
    lin, val = [], []
    for z, (own, r) in zip(z0, parts):
        k, j, i = np.nonzero(own)
        lin.append(((k + z) * Y + j + 4) * X + i + 5)
        val.append(r[own])
    return np.concatenate(lin), np.concatenate(val), np.concatenate([[0], np.cumsum([x.size for x in lin])])


def _builder(depth, n, conn):
    from tgmm_b200 import engine as E
    return E.FrameBuilder((X, Y, depth), n, conn3d=conn, max_nuclei_size=10 ** 6, min_nuclei_size=20)


def _oracle(raw, lab, n, conn):
    rc, want = O.frame_build(raw, lab, n, O.frame_params(max_size=10 ** 6, conn=conn, min_size=20))
    assert rc == 0
    return want


def _arrays(f):
    return {k: t.cpu().numpy() for k, t in (("query", f.query), ("img", f.img), ("cent", f.centroids),
                                            ("lptr", f.label_ptr))}


def _device_lists(lin, val, ptr):
    import torch
    return (torch.from_numpy(lin.astype(np.int32)).cuda(), torch.from_numpy(val.view(np.int16).copy()).cuda(),
            torch.from_numpy(ptr.astype(np.int64)).cuda())


@pytest.mark.parametrize("conn", [4, 6, 8, 26, 74])
def test_big_boxes_in_a_workspace_that_holds_anything(cuda_ok, conn):
    import torch
    z0 = (1, 25, 52)
    b = None
    for seed in (1, 2):
        rng = np.random.default_rng(seed)
        parts = [_part(rng, d) for d in (24, 21, 20)]
        raw, lab = _volume(parts, z0)
        if b is None:
            b = _builder(raw.shape[0], 3, conn)
        want = _oracle(raw, lab, 3, conn)
        lists = _device_lists(*_lists(parts, z0))
        b.build_lists(*lists)  # allocates the lists' workspace
        for fill in (0xFF, 0x00, 0xA5):
            b.workspace.fill_(fill)
            b.list_ws.fill_(fill)
            rd = torch.from_numpy(raw.reshape(-1).view(np.int16)).cuda()
            ld = torch.from_numpy(lab.reshape(-1).view(np.int32)).cuda()
            for build in (lambda: b.build(rd, ld), lambda: b.build_lists(*lists)):
                for _ in range(2):
                    f, thr = build()
                    got = _arrays(f)
                    for key in got:
                        np.testing.assert_array_equal(got[key], want[key], err_msg=key)
                    np.testing.assert_array_equal(thr, want["thr"])


@pytest.mark.parametrize("conn", [6, 74])
@pytest.mark.parametrize("shift", [0, 1, 11])
def test_lists_that_hold_the_same_voxels_are_trimmed_each_alone(cuda_ok, shift, conn):
    rng = np.random.default_rng(40 + shift)
    parts = [_part(rng, 22), _part(rng, 23), _part(rng, 22)]
    # apart in the oracle's volume; `shift` voxels deeper than one another in the lists
    apart, over = (1, 30, 60), (1, 1 + shift, 1 + 2 * shift)
    want = _oracle(*_volume(parts, apart), 3, conn)
    lin, val, ptr = _lists(parts, over)
    depth = 100
    b = _builder(depth, 3, conn)
    n = int(ptr[-1])
    assert n <= X * Y * depth
    f, thr = b.build_lists(*_device_lists(lin, val, ptr))
    got = _arrays(f)
    np.testing.assert_array_equal(thr, want["thr"])
    np.testing.assert_array_equal(got["lptr"], want["lptr"])
    np.testing.assert_array_equal(got["img"], want["img"])
    lp, N = want["lptr"], want["n_vox"]
    q, wq = got["query"].reshape(3, N), want["query"].reshape(3, N).copy()
    for s in range(3):
        wq[2, lp[s]:lp[s + 1]] += over[s] - apart[s]
        # the centroid alone, where the list says the supervoxel lies
        alone = _oracle(*_volume([parts[s]], (over[s],)), 1, conn)
        np.testing.assert_array_equal(got["cent"].reshape(3, 3)[:, s], alone["cent"])
    np.testing.assert_array_equal(q, wq)
