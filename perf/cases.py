"""The timed workloads: the calls a tracking program makes of this framework, over the sizes it
makes them at.

Every case is a dict of plain values.  `prepare` makes what such a program holds before the call
(device arrays, Gaussian records, plans and builders it keeps), `run` is one pass through the
public entry points, `exact` the same results in 64 bits from plain torch.  Volumes, nuclei and
Gaussians come from the seeded generator of the benchmark (`tgmm_b200.synth`): a case's `shape`
fixes where its nuclei lie, so that every seed gives arrays of the same sizes, and the seed draws
the intensities and the Gaussians' starting positions.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from tgmm_b200 import _lib as L
from tgmm_b200 import engine as E
from tgmm_b200 import synth

SCALE = (1.0, 1.0, 2.0)  # kNN and regularisation scale of every configuration
DEV = "cuda"


def listed():
    return [
        # the smallest EM call there is in use: a cropped region with a dozen nuclei, where the
        # launches and their gaps are the whole call
        dict(name="em_tiny", kind="em", x=64, y=64, z=32, nuclei=12, axes="3-6", shape=7, iters=20, tol=-1.0,
             w4dof=True, ll="reference", fp64=False, stats=True, tune=False),
        # the small configuration through the reference's ownership model: Gaussians on the host,
        # results back on the host, one synchronous call
        dict(name="em_host_small", kind="em_host", x=256, y=256, z=64, nuclei=300, axes="3-6", shape=1, iters=20,
             tol=-1.0),
        # one time point of a tracked series: the frame's voxel runs expanded on the device, the
        # EM with the reference's convergence test, the posterior made the next prior
        dict(name="track_step", kind="track", x=1024, y=1024, z=256, nuclei=5000, axes="4-8", shape=17, iters=20,
             tol=1e-6),
        # the headline: one 1-Gvoxel frame, 20 iterations, inputs and Gaussians resident
        dict(name="em_frame_large", kind="em", x=2048, y=1024, z=512, nuclei=20000, axes="4-8", shape=2000, iters=20,
             tol=-1.0, w4dof=True, ll="reference", fp64=False, stats=False, tune=True),
        # the batched form: uneven volumes in one call
        dict(name="em_batch", kind="batch", volumes=16, side=256, depth=96, shape=7, iters=20, tol=-1.0),
        # the options for validation runs: full covariance, every voxel in the likelihood, FP64 terms
        dict(name="em_general_fp64", kind="em", x=511, y=509, z=127, nuclei=2000, axes="4-8", shape=5, iters=10,
             tol=-1.0, w4dof=False, ll="true", fp64=True, stats=True, tune=False),
        # frame preparation from the raw image and the label volume of the segmentation
        dict(name="build_volume", kind="build", x=1024, y=1024, z=512, nuclei=10000, axes="4-8", shape=11, conn=6,
             lists=False),
        # the same from the segmentation's pixel lists, at the 1-Gvoxel frame
        dict(name="build_lists", kind="build", x=2048, y=1024, z=512, nuclei=20000, axes="4-8", shape=2000, conn=6,
             lists=True),
        # the tracking graph: each supervoxel's nearest supervoxels in the next time point
        dict(name="knn_graph", kind="knn_k", queries=20019, refs=20007, k=10),
        # the five nearest Gaussians of every foreground voxel
        dict(name="knn_voxels", kind="knn", queries=1426921, refs=2000),
        # the split round's test: local log-likelihood around each division candidate
        dict(name="local_ll", kind="local", x=1024, y=1024, z=256, nuclei=5000, axes="4-8", shape=17, lists=400),
        # compact voxels expanded into the EM's arrays, the upload path of a large frame
        dict(name="expand_compact", kind="expand", x=2048, y=1024, z=512, voxels=14471738),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, nuclei, per):
    """Volume sides for `nuclei` nuclei at `per` voxels each, uneven and often odd."""
    vol = nuclei * per
    z = max(24, int(round((vol / rng.uniform(6, 20)) ** (1 / 3))))
    y = max(48, int(round(math.sqrt(vol / z) * rng.uniform(0.7, 1.1))))
    x = max(48, int(round(vol / z / y)))
    return x, y, z


def draw(rng):
    kind = rng.choice(["em", "em", "em_host", "track", "batch", "build", "knn_k", "knn", "local", "expand"])
    axes = rng.choice(["3-6", "4-8"])
    shape = rng.randint(0, 1 << 20)
    per = int(rng.uniform(9000, 54000))
    if kind == "em":
        fp64 = rng.random() < 0.25
        n = _log(rng, 12, 4000 if fp64 else 16000)
        x, y, z = _box(rng, n, per)
        return dict(kind=kind, x=x, y=y, z=z, nuclei=n, axes=axes, shape=shape,
                    iters=rng.randint(5, 20), tol=-1.0, w4dof=rng.random() < 0.7, ll=rng.choice(["reference", "true"]),
                    fp64=fp64, stats=rng.random() < 0.5, tune=rng.random() < 0.3)
    if kind in ("em_host", "track"):
        n = _log(rng, 12, 3000 if kind == "em_host" else 12000)
        x, y, z = _box(rng, n, per)
        return dict(kind=kind, x=x, y=y, z=z, nuclei=n, axes=axes, shape=shape,
                    iters=rng.randint(10, 20), tol=-1.0 if kind == "em_host" else 1e-6)
    if kind == "batch":
        return dict(kind=kind, volumes=rng.randint(2, 24), side=_log(rng, 96, 256), depth=rng.randint(48, 96),
                    shape=shape, iters=rng.randint(5, 20), tol=-1.0)
    if kind == "build":
        n = _log(rng, 50, 10000)
        x, y, z = _box(rng, n, per)
        return dict(kind=kind, x=x, y=y, z=z, nuclei=n, axes=axes, shape=shape,
                    conn=rng.choice([6, 6, 26, 74]), lists=rng.random() < 0.5)
    if kind == "knn_k":
        return dict(kind=kind, queries=_log(rng, 300, 60000), refs=_log(rng, 300, 60000), k=rng.choice([1, 5, 10, 11]))
    if kind == "knn":
        return dict(kind=kind, queries=_log(rng, 1000, 1400000), refs=_log(rng, 100, 20000))
    if kind == "local":
        n = _log(rng, 100, 6000)
        x, y, z = _box(rng, n, per)
        return dict(kind=kind, x=x, y=y, z=z, nuclei=n, axes=axes, shape=shape,
                    lists=max(1, int(n * rng.uniform(0.01, 0.3))))
    return dict(kind="expand", x=rng.randint(200, 2048), y=rng.randint(200, 1024), z=rng.randint(100, 512),
                voxels=_log(rng, 20000, 4000000))


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _spec(c, dims=None, nuclei=None):
    lo, hi = (3.0, 6.0) if c.get("axes", "4-8") == "3-6" else (4.0, 8.0)
    return synth.VolumeSpec(dims=dims or (c["x"], c["y"], c["z"]), n_nuclei=nuclei or c["nuclei"], axis_min=lo,
                            axis_max=hi)


def _params(c):
    return synth.em_params(iters=c["iters"], tol=c["tol"], w4dof=1 if c.get("w4dof", True) else 0,
                           ll_mode=L.TGMM_LL_TRUE if c.get("ll") == "true" else L.TGMM_LL_AS_REFERENCE,
                           ll_precision=L.TGMM_LLPREC_FP64 if c.get("fp64") else L.TGMM_LLPREC_MIXED)


def _batch_shapes(c):
    """The batch's volumes: sides in [side/2, side], depths in [depth/2, depth], one nucleus per
    ~3000 voxels, at least 12."""
    r = np.random.default_rng(c["shape"])
    out = []
    for _ in range(c["volumes"]):
        X, Y = (int(v) for v in r.integers(c["side"] // 2, c["side"] + 1, 2))
        Z = int(r.integers(c["depth"] // 2, c["depth"] + 1))
        out.append(((X, Y, Z), max(12, round(X * Y * Z / 3000))))
    return out


def _redraw(f, seed):
    """The frame with its raw values drawn anew (Poisson-like spread, above the threshold) and what
    follows from them: rescaled intensities and intensity-weighted centroids."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    thr, N, S = int(f.spec.threshold), f.n_vox, f.n_sv
    raw = torch.from_numpy(f.raw.astype(np.int32)).to(DEV).float()
    raw = (raw + raw.sqrt() * torch.randn(N, device=DEV, generator=g)).round().long().clamp(thr + 1, 2000)
    w = raw - thr
    den = int(w.max())
    q = torch.from_numpy(f.query).to(DEV).view(3, N).long()
    sv = torch.repeat_interleave(torch.arange(S, device=DEV), torch.from_numpy(f.label_ptr).to(DEV).diff())
    tot = torch.zeros(S, dtype=torch.long, device=DEV).index_add_(0, sv, w).double()
    cent = torch.stack([torch.zeros(S, dtype=torch.long, device=DEV).index_add_(0, sv, w * q[d]).double() / tot
                        for d in range(3)])
    f.img, f.centroids = (w.double() / den).float().cpu().numpy(), cent.float().view(-1).cpu().numpy()
    f.raw, f.max_fg = raw.to(torch.int32).cpu().numpy().astype(np.uint16), float(den + thr)
    return f


def _frame(c, seed, shape=None, dims=None, nuclei=None, gaussians=True):
    shape = c["shape"] if shape is None else shape
    spec = _spec(c, dims, nuclei)
    f = synth.make_frame(spec, synth.random_nuclei(spec, shape), shape)
    if gaussians:
        synth.init_gaussians(f, seed)
    synth.release(f)
    return _redraw(f, seed)


def _batch_frames(c, seed):
    return [_frame(c, seed + i, c["shape"] + i, d, n) for i, (d, n) in enumerate(_batch_shapes(c))]


def _track_frames(c, seed):
    """Gaussians of one time point (as its priors stand) and the voxels of the next, whose nuclei
    have moved and divided."""
    spec = _spec(c)
    nuc = synth.random_nuclei(spec, c["shape"])
    f0 = synth.make_frame(spec, nuc, c["shape"])
    synth.init_gaussians(f0, seed)
    synth.release(f0)
    f1 = synth.make_frame(spec, synth.evolve_nuclei(nuc, spec, np.random.default_rng(c["shape"])), c["shape"] + 1)
    synth.release(f1)
    return f0.gauss, _redraw(f1, seed)


def _build_inputs(c, seed):
    """A segmented volume on the GPU: each supervoxel's linear indices and raw values."""
    f = _frame(c, seed, gaussians=False)
    X, Y, Z = f.spec.dims
    q = torch.from_numpy(f.query).to(DEV).view(3, f.n_vox).long()
    lin = q[0] + X * (q[1] + Y * q[2])
    val = torch.from_numpy(f.raw.view(np.int16)).to(DEV)
    ptr = torch.from_numpy(np.ascontiguousarray(f.label_ptr, np.int64)).to(DEV)
    return lin, val, ptr, f.n_sv


def _points(c, seed):
    """kNN inputs: references spread over a volume of the usual density; queries are the moved
    references (a graph's next time point) or voxels around them."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    nr, nq = c["refs"], c["queries"]
    side = (nr * 30000.0) ** (1 / 3)
    ext = torch.tensor([1.6 * side, 1.25 * side, side / 2], device=DEV)
    ref = torch.rand(nr, 3, device=DEV, generator=g) * ext
    own = torch.arange(nq, device=DEV) * nr // nq  # a reference's queries sit together
    q = ref[own] + torch.randn(nq, 3, device=DEV, generator=g) * (1.5 if c["kind"] == "knn_k" else 4.0)
    if c["kind"] == "knn":
        q = torch.round(q)
    return q.clamp_min(0).t().contiguous().view(-1), ref


def _local_inputs(c, seed):
    f = _frame(c, seed)
    df = E.to_device(f)
    gm = E.gauss_to_device(f.gauss)
    cent = df.centroids.view(3, -1).t()
    mean = _fields(gm)["m"].float()
    ind = _nearest(cent, mean, 5)[1].t().contiguous().view(-1).to(torch.int32)
    r = np.random.default_rng(seed)
    order = np.argsort(f.sv_nucleus, kind="stable")
    start = np.searchsorted(f.sv_nucleus[order], f.gauss_nucleus)
    end = np.searchsorted(f.sv_nucleus[order], f.gauss_nucleus, side="right")
    pick = r.permutation(f.n_gauss)[:c["lists"]]
    return df, ind, gm, [[int(s) for s in order[start[k]:end[k]]] for k in pick]


def _em_state(c, frames, gauss, max_frames=1):
    dfs = [E.to_device(f, n_gauss=g.shape[0]) for f, g in zip(frames, gauss)]
    K, S = [g.shape[0] for g in gauss], [f.n_sv for f in frames]
    gm0 = torch.cat([E.gauss_to_device(g) for g in gauss])
    s = dict(dfs=dfs, gm0=gm0, gm=gm0.clone(), rnk=torch.empty(5 * sum(S), device=DEV),
             ind=torch.empty(5 * sum(S), dtype=torch.int32, device=DEV), params=_params(c),
             plan=E.Plan(sum(f.n_vox for f in frames), sum(S), sum(K), max_frames=max_frames))
    s["gms"] = list(s["gm"].split([288 * k for k in K]))
    s["rnks"], s["inds"] = list(s["rnk"].split([5 * n for n in S])), list(s["ind"].split([5 * n for n in S]))
    return s


def prepare(case, seed):
    c, kind = case, case["kind"]
    s = dict(kind=kind, stats=bool(c.get("stats", True)))
    if kind == "em":
        f = _frame(c, seed)
        s.update(_em_state(c, [f], [f.gauss]))
        if c["tune"]:
            s["plan"].autotune(s["dfs"], s["gms"], s["rnks"], s["inds"], s["params"], reps=2)
    elif kind == "em_host":
        f = _frame(c, seed)
        s.update(_em_state(c, [f], [f.gauss]), gauss=f.gauss)
    elif kind == "batch":
        fs = _batch_frames(c, seed)
        s.update(_em_state(c, fs, [f.gauss for f in fs], max_frames=len(fs)))
        s["plan"].autotune(s["dfs"], s["gms"], s["rnks"], s["inds"], s["params"], reps=2)
    elif kind == "track":
        gauss, f = _track_frames(c, seed)
        s.update(_em_state(c, [f], [gauss]))
        rp, rs, rl, raw, dims, off, den = f.runs()
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)  # noqa: E731
        s["codes"] = (t(rp), t(rs.view(np.int32)), t(rl.view(np.int16)), t(raw.view(np.int16)), dims, off, den)
    elif kind == "build":
        lin, val, ptr, n = _build_inputs(c, seed)
        dims = (c["x"], c["y"], c["z"])
        b = s["builder"] = E.FrameBuilder(dims, n, conn3d=c["conn"], max_vox=lin.numel())
        for t in (b.query, b.img, b.cent, b.lptr, b.thr):
            t.zero_()
        s["lists"] = c["lists"]
        if c["lists"]:
            s["args"] = (lin.to(torch.int32), val, ptr)
        else:
            nvol = dims[0] * dims[1] * dims[2]
            g = torch.Generator(device=DEV).manual_seed(seed)
            raw = torch.randint(100, 130, (nvol,), device=DEV, generator=g, dtype=torch.int16)
            raw[lin] = val
            lab = torch.zeros(nvol, dtype=torch.int32, device=DEV)
            lab[lin] = torch.repeat_interleave(torch.arange(1, n + 1, device=DEV, dtype=torch.int32), ptr.diff())
            s["args"] = (raw, lab)
    elif kind in ("knn", "knn_k"):
        q, ref = _points(c, seed)
        s["q"], s["ref"] = q, (ref.contiguous().view(-1) if kind == "knn" else ref.t().contiguous().view(-1))
        if kind == "knn_k":
            s["k"], nq = c["k"], c["queries"]
            s["ind"] = torch.empty(c["k"] * nq, dtype=torch.int32, device=DEV)
            s["dist"] = torch.empty(c["k"] * nq, device=DEV)
    elif kind == "local":
        s["args"] = _local_inputs(c, seed)
    elif kind == "expand":
        lin, raw, q, im = _expand_inputs(c, seed)
        s["args"] = (lin, raw, (c["x"], c["y"], c["z"]), 150.0, 1087.0, q, im)
    return s


def _expand_inputs(c, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    n, nvol = c["voxels"], c["x"] * c["y"] * c["z"]
    lin = torch.randint(0, nvol, (n,), device=DEV, generator=g).sort()[0]
    raw = torch.randint(151, 1238, (n,), device=DEV, generator=g, dtype=torch.int32)
    lin = torch.where(lin >= 2 ** 31, lin - 2 ** 32, lin).to(torch.int32)
    return lin, raw.to(torch.int16), torch.empty(3 * n, device=DEV), torch.empty(n, device=DEV)


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def _fields(gm):
    """The named fields of device Gaussian records."""
    d, i = gm.view(torch.float64).view(-1, 36), gm.view(torch.int32).view(-1, 72)
    return dict(beta=d[:, 0], nu=d[:, 1], alpha=d[:, 2], m=d[:, 3:6], W=d[:, 6:12], eld=d[:, 12], elr=d[:, 13],
                beta_o=d[:, 15], nu_o=d[:, 16], alpha_o=d[:, 17], m_o=d[:, 18:21], W_o=d[:, 21:27],
                sv=i[:, 55:71], n_sv=i[:, 71])


def _stat(st):
    return dict(ll=st["ll"], total_alpha=st["total_alpha"], iterations=st["iterations"], converged=st["converged"],
                n_dead=st["n_dead"])


def run(state):
    s, kind = state, state["kind"]
    if kind in ("em", "batch", "track"):
        s["gm"].copy_(s["gm0"])  # the EM updates its records in place
        if kind == "track":
            rp, rs, rl, raw, dims, off, den = s["codes"]
            df = s["dfs"][0]
            E.expand_runs(rp, rs, rl, raw, df.label_ptr, dims, off, den, df.query, df.img)
        out = {}
        if kind == "batch":
            s["plan"].run_batch(s["dfs"], s["gms"], s["rnks"], s["inds"], s["params"], stats=False)
        else:
            st = s["plan"].run_device(s["dfs"][0], s["gm"], s["rnk"], s["ind"], s["params"], stats=s["stats"])
            out = _stat(st) if st else {}
        if kind == "track":
            E.update_priors(s["gm"], s["dfs"][0].n_gauss)
            out.update(query=df.query, img=df.img)
        return dict(out, rnk=s["rnk"], ind=s["ind"], **_fields(s["gm"]))
    if kind == "em_host":
        o = s["plan"].run_host(s["dfs"][0], s["gauss"], s["params"])
        g = o["gauss"]
        names = dict(beta="beta_k", nu="nu_k", alpha="alpha_k", m="m_k", W="W_k", eld="eLD", elr="eLR",
                     beta_o="beta_o", nu_o="nu_o", alpha_o="alpha_o", m_o="m_o", W_o="W_o", sv="supervoxelIdx",
                     n_sv="supervoxelNum")
        return dict(_stat(o), rnk=o["rnk"], ind=o["ind"], **{k: g[v] for k, v in names.items()})
    if kind == "build":
        b = s["builder"]
        f, _ = (b.build_lists if s["lists"] else b.build)(*s["args"], read_thr=False)
        return dict(n_vox=f.n_vox, n_sv=f.n_sv, query=b.query, img=b.img, centroids=b.cent, label_ptr=b.lptr,
                    thr=b.thr)  # the builder's buffers: zero past the sizes in front
    if kind == "knn":
        return dict(ind=E.knn(s["q"], s["ref"], SCALE))
    if kind == "knn_k":
        sc = (C.c_float * 3)(*SCALE)
        L.check(L.gmem().tgmm_knn_k(s["q"].data_ptr(), s["q"].numel() // 3, s["ref"].data_ptr(), s["ref"].numel() // 3,
                                    s["k"], sc, s["ind"].data_ptr(), s["dist"].data_ptr(),
                                    torch.cuda.current_stream().cuda_stream), "tgmm_knn_k")
        return dict(ind=s["ind"], dist=s["dist"])
    if kind == "local":
        return dict(ll=E.local_likelihood(*s["args"]))
    E.expand_frame(*s["args"])
    return dict(query=s["args"][5], img=s["args"][6])


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    per = 304.0 if c.get("axes") == "3-6" else 718.0  # foreground voxels a nucleus, on these volumes
    if kind in ("em", "em_host", "track", "batch"):
        K = sum(n for _, n in _batch_shapes(c)) if kind == "batch" else c["nuclei"]
        N = K * (650.0 if kind == "batch" else per)
        iters = 4 if kind == "track" else c["iters"]
        # voxels in once; centroids, CSR, records in and out; candidates and responsibilities out.
        # per voxel and iteration: five quadratic forms and a log of five exponentials
        b = 16 * N + K * (20 + 2 * 288 + 40)
        if kind == "track":  # about 3 bytes a voxel of codes in, the float arrays out, read by the EM
            b += 19 * N
        return dict(bytes=b, flops=100 * N * iters)
    if kind == "build":
        n = c["nuclei"] * per
        vol = c["x"] * c["y"] * c["z"]
        return dict(bytes=(6 * n if c["lists"] else 4 * vol + 2 * n) + 16 * n / 4, flops=0)
    if kind == "knn":
        return dict(bytes=c["queries"] * 32 + c["refs"] * 12, flops=0)
    if kind == "knn_k":
        return dict(bytes=c["queries"] * (12 + 8 * c["k"]) + c["refs"] * 12, flops=0)
    if kind == "local":
        return dict(bytes=c["lists"] * (16 * per + 5 * 120), flops=c["lists"] * per * 5 * 20)
    return dict(bytes=c["voxels"] * 22, flops=0)


# ---------------------------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------------------------
def _nearest(q, ref, k):
    """The k nearest references of each query row: (squared scaled distances, indices), nearest first."""
    s = torch.tensor(SCALE, dtype=torch.float64, device=DEV)
    a, b = q.double() * s, ref.double() * s
    d, i = [], []
    step = max(1, int(4e8) // max(1, b.shape[0]))
    for r in range(0, a.shape[0], step):
        x = a[r:r + step]
        t = sum((x[:, None, e] - b[None, :, e]) ** 2 for e in range(3))
        v, j = t.topk(min(k, b.shape[0]), dim=1, largest=False, sorted=True)
        d.append(v)
        i.append(j)
    return torch.cat(d), torch.cat(i)


def _sym(w):
    return w[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].view(-1, 3, 3)


def _upper(m):
    return torch.stack([m[:, 0, 0], m[:, 0, 1], m[:, 0, 2], m[:, 1, 1], m[:, 1, 2], m[:, 2, 2]], 1)


def _maha(W, d):
    return torch.einsum("ni,nij,nj->n", d, _sym(W), d)


def _segments(x, sv, n):
    return torch.zeros((n,) + x.shape[1:], dtype=torch.float64, device=DEV).index_add_(0, sv, x)


def _exact_em(c, frame, gauss):
    """The EM of one frame in 64 bits: E-step over supervoxels, Dirichlet / Normal-Wishart update,
    regularisation, dead rule, log-likelihood test."""
    p = _params(c)
    N, S = frame.n_vox, frame.n_sv
    x = torch.from_numpy(frame.query).to(DEV).view(3, N).t().double()
    I = torch.from_numpy(frame.img).to(DEV).double()
    cent = torch.from_numpy(frame.centroids).to(DEV).view(3, S).t()
    lp = torch.from_numpy(frame.label_ptr).to(DEV)
    sv = torch.repeat_interleave(torch.arange(S, device=DEV), lp.diff())
    n = lp.diff().double()
    kept = torch.ones(N, dtype=torch.bool, device=DEV) if p.ll_mode == L.TGMM_LL_TRUE else \
        torch.arange(N, device=DEV) >= lp[1:][sv] - 1024
    e = x - cent.double()[sv]
    outer = torch.stack([e[:, 0] ** 2, e[:, 0] * e[:, 1], e[:, 0] * e[:, 2], e[:, 1] ** 2, e[:, 1] * e[:, 2],
                         e[:, 2] ** 2], 1)
    G1, G2 = _segments(e, sv, S), _segments(outer, sv, S)
    H0, H1, H2 = _segments(I, sv, S), _segments(e * I[:, None], sv, S), _segments(outer * I[:, None], sv, S)
    ia, ib = [0, 0, 0, 1, 1, 2], [0, 1, 2, 1, 2, 2]
    g = {k: v.clone() for k, v in _fields(E.gauss_to_device(gauss)).items()}
    fixed = torch.from_numpy(np.ascontiguousarray(gauss["fixed"])).to(DEV) != 0
    rs = [float(v) for v in p.reg_scale]
    rs = torch.tensor(rs if any(rs) else [float(v) for v in p.scale], dtype=torch.float64, device=DEV)
    hist, it, done = [-1.0, -10.0, -100.0, -1000.0], 0, False
    while it < p.max_iter_em and not done:
        it += 1
        dead = g["m_o"][:, 0] < -1e31
        A = g["alpha"].sum()
        eld = 3 * math.log(2.0) + torch.linalg.det(_sym(g["W"])).log() + sum(
            torch.digamma(0.5 * (g["nu"] + 1.0 - i)) for i in range(3))
        eld = torch.where(dead, -1e32, eld)
        elr = torch.where(dead, -1e32, torch.digamma(g["alpha"]) - torch.digamma(A))
        g["eld"], g["elr"] = eld, elr
        cand = _nearest(cent, g["m"].float(), 5)[1]
        lik = []
        for j in range(5):
            k = cand[:, j]
            u = g["m"][k] - cent.double()
            D = torch.stack([G2[:, q] - G1[:, ia[q]] * u[:, ib[q]] - u[:, ia[q]] * G1[:, ib[q]] +
                             n * u[:, ia[q]] * u[:, ib[q]] for q in range(6)], 1)
            w = torch.tensor([1., 2., 2., 1., 2., 1.], dtype=torch.float64, device=DEV)
            t = -0.5 * (3 * n / g["beta"][k] + g["nu"][k] * (g["W"][k] * D * w).sum(1)) + n * (elr[k] + 0.5 * eld[k])
            lik.append(torch.where(dead[k] & (n > 0), -math.inf, t))
        lik = torch.stack(lik, 1)
        rnk = 1.0 / (lik[:, None, :] - lik[:, :, None]).exp().sum(2)
        r = torch.where(rnk > 1e-3, rnk, 0.0)
        K = g["nu"].shape[0]
        N0 = torch.zeros(K, dtype=torch.float64, device=DEV)
        N1, N2 = torch.zeros(K, 3, dtype=torch.float64, device=DEV), torch.zeros(K, 6, dtype=torch.float64, device=DEV)
        for j in range(5):
            k = cand[:, j]
            d = cent.double() - g["m_o"][k].clamp_min(-1e4)
            rj = r[:, j]
            N0.index_add_(0, k, rj * H0)
            N1.index_add_(0, k, rj[:, None] * (H1 + H0[:, None] * d))
            N2.index_add_(0, k, rj[:, None] * (H2 + H1[:, ia] * d[:, ib] + d[:, ia] * H1[:, ib] +
                                               H0[:, None] * d[:, ia] * d[:, ib]))
        live = ~dead & ~fixed
        has = N0 > 0
        inv = torch.where(has, 1.0 / N0.clamp_min(1e-300), 0.0)
        xb = torch.where(has[:, None], g["m_o"] + N1 * inv[:, None], 0.0)
        Sk = N2 - N1[:, ia] * N1[:, ib] * inv[:, None]
        bo = g["beta_o"]
        beta, nu, alpha = bo + N0, g["nu_o"] + N0, (g["alpha_o"] + N0).clamp_min(0.0)
        m = (bo[:, None] * g["m_o"] + N0[:, None] * xb) / beta[:, None]
        Wo = g["W_o"].clone()
        Wo[:, 5] = torch.where(live & (Wo[:, 5] < 1e-8), 0.5 * (Wo[:, 0] + Wo[:, 3]), Wo[:, 5])
        safe = torch.where(live[:, None], Wo, torch.tensor([1., 0, 0, 1, 0, 1], dtype=torch.float64, device=DEV))
        dx = torch.where(live[:, None], xb - g["m_o"], 0.0)
        Wi = _upper(torch.linalg.inv(_sym(safe))) + Sk + (N0 * bo / beta)[:, None] * dx[:, ia] * dx[:, ib]
        Wi = torch.where(live[:, None], Wi, torch.tensor([1., 0, 0, 1, 0, 1], dtype=torch.float64, device=DEV))
        W = _upper(torch.linalg.inv(_sym(Wi))) / (rs[ia] * rs[ib])
        if p.w4dof:
            W[:, 2] = W[:, 4] = 0.0
        ev, V = torch.linalg.eigh(_sym(W).cpu())
        ev, V = ev.to(DEV), V.to(DEV)
        ev = torch.minimum(torch.maximum(ev, (p.lambda_min / nu)[:, None]), (p.lambda_max / nu)[:, None])
        ev = torch.minimum(ev, p.max_excentricity * ev[:, :1])
        W = _upper(torch.einsum("kia,ka,kja->kij", V, ev, V)) * (rs[ia] * rs[ib])
        for name, new in (("beta", beta), ("nu", nu), ("alpha", alpha), ("m", m), ("W", W)):
            g[name] = torch.where(live.view((-1,) + (1,) * (new.dim() - 1)), new, g[name])
        g["W_o"] = Wo
        A = g["alpha"].sum()
        kill = torch.isnan(g["W"]).any(1) | torch.isnan(eld) | ((g["alpha"] / A < 1e-5) & live)
        g["alpha"] = torch.where(kill, 0.0, g["alpha"])
        for name in ("m", "m_o"):
            g[name] = torch.where(kill[:, None], -1e32, g[name])
        g["W"] = torch.where(kill[:, None], torch.tensor([1., 0, 0, 1, 0, 1], dtype=torch.float64, device=DEV), g["W"])
        A = g["alpha"].sum()
        wt = (torch.linalg.det(_sym(g["W"])) * g["nu"] ** 3).sqrt() / (2 * math.pi) ** 1.5 * g["alpha"] / A
        dens = torch.zeros(N, dtype=torch.float64, device=DEV)
        for j in range(5):
            k = cand[:, j][sv]
            dens += wt[k] * (-0.5 * g["nu"][k] * _maha(g["W"][k], x - g["m"][k].clamp_min(-1e4))).exp()
        ok = kept & (dens > 0)
        hist = [float(torch.where(ok, I * dens.clamp_min(1e-320).log(), 0.0).sum())] + hist[:3]
        done = not all(abs(hist[0] - h) / abs(h) > p.tol_likelihood for h in hist[1:])
    out = {k: g[k] for k in ("beta", "nu", "alpha", "m", "W", "eld", "elr", "beta_o", "nu_o", "alpha_o", "m_o", "W_o")}
    return dict(out, rnk=rnk.t().contiguous().view(-1), ll=hist[0], total_alpha=float(A))


def _exact_priors(o):
    """The posterior as the next time point's prior."""
    nk = o["nu"] - o["nu_o"]
    nu_o = nk.clamp_min(3.0)
    return dict(o, m_o=o["m"], beta_o=(0.01 * nk).clamp_min(1e-5), nu_o=nu_o,
                W_o=o["W"] * (o["nu"] / nu_o)[:, None], alpha_o=torch.full_like(nk, o["total_alpha"] * 1e-5 * 0.8),
                nu=o["nu"] * 2, W=o["W"] / 2)


def _exact_build(c, seed):
    """Trimming, size filter, erase order, centroids and rescaled intensities, over all
    supervoxels at once; the thresholds as the rule states them, in 32-bit floats."""
    lin, val, ptr, n = _build_inputs(c, seed)
    X, Y, Z = c["x"], c["y"], c["z"]
    N, cnt = lin.numel(), ptr.diff()
    sv = torch.repeat_interleave(torch.arange(n, device=DEV), cnt)
    v = val.long() & 0xffff
    srt = v[torch.argsort(sv * 65536 + v)]
    at = lambda k: srt[ptr[:-1] + k].float()  # noqa: E731
    k2 = ((torch.tensor(1.0, device=DEV) - torch.tensor(0.4, device=DEV)) * cnt.float()).long()
    lo, hi = at(torch.zeros_like(cnt)), at(cnt - 1)
    mm = torch.tensor(255.0, device=DEV) / (hi - lo)
    bins = ((v.float() - lo[sv]) * mm[sv]).nan_to_num(0).long().clamp(0, 255)
    h = torch.bincount(sv * 256 + bins, minlength=256 * n).view(n, 256).float()
    wb = h.cumsum(1)
    bin_ = torch.arange(256, device=DEV)
    sb = (h * bin_).cumsum(1)
    wf = cnt[:, None].float() - wb
    d = sb / wb - (sb[:, -1:] - sb) / wf
    var = torch.where((wb > 0) & (wf > 0), wb * wf * d * d, 0.0)
    best = torch.where(var == var.max(1, keepdim=True)[0], bin_, 256).min(1)[0]  # the first of equals
    t3 = torch.where(torch.isfinite(mm), best.float() / mm + lo, torch.tensor(-1.0, device=DEV))
    thr = torch.maximum(torch.maximum(at((cnt - 3000).clamp_min(0)), at(torch.minimum(k2, cnt - 1))), t3).long()
    cand = v > thr[sv]
    entry = torch.full((X * Y * Z,), -1, dtype=torch.int32, device=DEV)
    entry[lin] = torch.arange(N, device=DEV, dtype=torch.int32)
    r = 2 if c["conn"] == 74 else 1
    offs = [dx + X * (dy + Y * dz) for dz in (-1, 0, 1) for dy in range(-r, r + 1) for dx in range(-r, r + 1)
            if (dx or dy or dz) and (c["conn"] != 6 or abs(dx) + abs(dy) + abs(dz) == 1)]
    first = torch.full((n,), N, device=DEV).scatter_reduce(
        0, sv, torch.where(v == hi[sv].long(), torch.arange(N, device=DEV), N), "amin")
    reach = torch.zeros(N, dtype=torch.bool, device=DEV)
    reach[first] = True
    reach &= cand
    front = reach.nonzero().view(-1)
    while front.numel():  # breadth first from each supervoxel's brightest voxel
        new = []
        for o in offs:
            t = lin[front] + o
            ok = (t >= 0) & (t < X * Y * Z)
            j = entry[t[ok]].long()
            f = front[ok][j >= 0]
            j = j[j >= 0]
            j = j[(sv[j] == sv[f]) & cand[j] & ~reach[j]]
            reach[j] = True
            new.append(j)
        front = torch.cat(new).unique()
    kept = torch.zeros(n, dtype=torch.long, device=DEV).index_add_(0, sv, reach.long())
    order, small = list(range(n)), (kept < 50).nonzero().view(-1).tolist()
    for i in reversed(small):  # each erased supervoxel trades places with the last one left
        order[i], order[-1] = order[-1], order[i]
        order.pop()
    order = torch.tensor(order, device=DEV)
    rank = torch.full((n,), -1, device=DEV)
    rank[order] = torch.arange(order.numel(), device=DEV)
    keep = reach & (rank[sv] >= 0)
    key = rank[sv[keep]] * (X * Y * Z) + lin[keep]
    idx = keep.nonzero().view(-1)[torch.argsort(key)]
    l, w = lin[idx], v[idx].double()
    q = torch.stack([l % X, (l // X) % Y, l // (X * Y)]).double()
    S, s = order.numel(), rank[sv[idx]]
    cent = torch.zeros(3, S, dtype=torch.float64, device=DEV).index_add_(1, s, q * w) / _segments(w, s, S)
    sub = w - thr[sv[idx]]
    top, low = max(float(sub.max()), 0.0), min(float(sub.min()), 0.0)
    pad = lambda a, size: torch.nn.functional.pad(a, (0, size - a.numel()))  # noqa: E731
    return dict(query=pad(q.view(-1), 3 * N), img=pad((sub - low) / (top - low), N),
                centroids=pad(cent.view(-1), 3 * n))


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("em", "em_host"):
        f = _frame(c, seed)
        o = _exact_em(c, f, f.gauss)
        if not c.get("stats", True):
            o.pop("ll"), o.pop("total_alpha")
        return o
    if kind == "track":
        gauss, f = _track_frames(c, seed)
        o = _exact_priors(_exact_em(c, f, gauss))
        thr = float(np.float32(f.spec.threshold))
        img = (torch.from_numpy(f.raw.astype(np.float64)) - thr) / (float(f.max_fg) - thr)
        return dict(o, query=torch.from_numpy(f.query).double(), img=img)
    if kind == "batch":
        outs = [_exact_em(c, f, f.gauss) for f in _batch_frames(c, seed)]
        return {k: torch.cat([o[k] for o in outs]) for k in outs[0] if k not in ("ll", "total_alpha")}
    if kind == "build":
        return _exact_build(c, seed)
    if kind == "knn":
        return None  # indices alone
    if kind == "knn_k":
        q, ref = _points(c, seed)
        d = _nearest(q.view(3, -1).t(), ref, c["k"])[0]
        return dict(dist=d.t().contiguous().view(-1))
    if kind == "local":
        df, ind, gm, lists = _local_inputs(c, seed)
        g, S = _fields(gm), df.n_sv
        A = g["alpha"].sum()
        wt = (torch.linalg.det(_sym(g["W"])) * g["nu"] ** 3).sqrt() / (2 * math.pi) ** 1.5 * g["alpha"] / A
        x, lp = df.query.view(3, -1).t().double(), df.label_ptr.tolist()
        cand = ind.view(5, S).long()
        out = []
        for one in lists:
            t = 0.0
            for s in one:
                a, b = max(lp[s], lp[s + 1] - 1024), lp[s + 1]
                dens = sum(wt[k] * (-0.5 * g["nu"][k] * _maha(g["W"][k].expand(b - a, 6), x[a:b] - g["m"][k])).exp()
                           for k in cand[:, s])
                ok = dens > 0
                t = t + (df.img[a:b].double()[ok] * dens[ok].log()).sum()
            out.append(float(t))
        return dict(ll=np.array(out))
    lin, raw, _, _ = _expand_inputs(c, seed)
    l = lin.long() & 0xffffffff
    q = torch.stack([l % c["x"], (l // c["x"]) % c["y"], l // (c["x"] * c["y"])]).double().view(-1)
    return dict(query=q, img=((raw.long() & 0xffff).double() - 150.0) / 1087.0)
