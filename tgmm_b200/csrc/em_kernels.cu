// em_kernels.cu -- the sm_100a kernels of the supervoxel VI-EM.
//
// One EM call is:  build_maps, import (+ frame tail), moments,
//                  then per iteration: knn_estep, mstep_update, kill_prep (+ frame tail),
//                  ll_pass (+ convergence test);  finally assign, export.
// Every kernel loops over the whole batch (one or many frames); frames that have
// converged are skipped through their FrameState::done flag, so a captured graph of
// max_iter iterations serves any batch.  No kernel uses float atomics: per-frame sums
// are fixed-order sums of frame-aligned chunk partials, the M-step visits each
// Gaussian's (supervoxel, slot) pairs in ascending position order, and results are
// bit-identical whether a frame runs alone or inside a batch.
#include <float.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <cstddef>
#include <type_traits>

#include "tgmm_internal.cuh"

namespace tgmm {

namespace {

constexpr float kInfF = __builtin_huge_valf();
constexpr double kInf = __builtin_huge_val();

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;  // identical in every lane: each butterfly level adds commutative pairs
}

__device__ __forceinline__ int warp_sum_i(int v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Fixed-order sum of the partials [base, base+n) by one warp: lane l adds l, l+32, ...
// in order, then a butterfly.  Every warp that calls it with the same data gets the
// same bits.
__device__ __forceinline__ double warp_sum_range(const double* a, int base, int n) {
  const int lane = threadIdx.x & 31;
  double s = 0.0;
  int i = lane;
  for (; i + 96 < n; i += 128) {  // four loads in flight, added in the same order
    const double a0 = a[base + i], a1 = a[base + i + 32], a2 = a[base + i + 64], a3 = a[base + i + 96];
    s += a0;
    s += a1;
    s += a2;
    s += a3;
  }
  for (; i < n; i += 32) s += a[base + i];
  return warp_sum(s);
}

// Block (kN threads) fixed-order sum; result valid in thread 0.
template <int kN>
__device__ __forceinline__ double block_sum_n(double v, double* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < kN / 32; i++) t += sh[i];
  return t;
}

// A chunk's alpha (fixed-order sum, kGChunk threads) and dead count, in one reduction,
// written to the chunk's partials by thread 0.
__device__ __forceinline__ void chunk_partials(double alpha, int dead, double* shd, int* shi, double* alpha_part,
                                               int32_t* dead_part, int c) {
  const double wa = warp_sum(alpha);
  const int wd = warp_sum_i(dead);
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    shd[w] = wa;
    shi[w] = wd;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double at = 0.0;
    int nd = 0;
    for (int i = 0; i < kGChunk / 32; i++) {
      at += shd[i];
      nd += shi[i];
    }
    alpha_part[c] = at;
    dead_part[c] = nd;
  }
}

// ---------------------------------------------------------------------------
// kNN primitives.  Distance (FP32, the reference's formula and rounding):
//   a = (q0 - r0) * s0;  d = a*a;  b = (q1 - r1) * s1;  d = fma(b, b, d);  c = ...; d = fma(c, c, d)
// Order: (d, index) ascending, NaN as +inf -> ties go to the lower index.
// ---------------------------------------------------------------------------
// The N nearest found so far, sorted in (d, index) order; unused slots hold (+inf, INT_MAX).
template <int N>
struct TopN {
  float d[N];
  int i[N];
};
using Top5 = TopN<kJ>;

template <int N>
__device__ __forceinline__ void topn_init(TopN<N>& t) {
#pragma unroll
  for (int j = 0; j < N; j++) {
    t.d[j] = kInfF;
    t.i[j] = 0x7fffffff;
  }
}
__device__ __forceinline__ void top5_init(Top5& t) { topn_init<kJ>(t); }

__device__ __forceinline__ bool before(float da, int ia, float db, int ib) {
  return da < db || (da == db && ia < ib);
}

template <int N>
__device__ __forceinline__ void topn_insert(TopN<N>& t, float d, int idx) {
  if (!before(d, idx, t.d[N - 1], t.i[N - 1])) return;
  t.d[N - 1] = d;
  t.i[N - 1] = idx;
#pragma unroll
  for (int p = N - 1; p > 0; --p) {
    if (before(t.d[p], t.i[p], t.d[p - 1], t.i[p - 1])) {
      float td = t.d[p];
      t.d[p] = t.d[p - 1];
      t.d[p - 1] = td;
      int ti = t.i[p];
      t.i[p] = t.i[p - 1];
      t.i[p - 1] = ti;
    }
  }
}

__device__ __forceinline__ float knn_dist(float q0, float q1, float q2, float r0, float r1,
                                          float r2, const float* s) {
  float a = __fmul_rn(__fsub_rn(q0, r0), s[0]);
  float d = __fmul_rn(a, a);
  float b = __fmul_rn(__fsub_rn(q1, r1), s[1]);
  d = __fmaf_rn(b, b, d);
  float c = __fmul_rn(__fsub_rn(q2, r2), s[2]);
  d = __fmaf_rn(c, c, d);
  return isnan(d) ? kInfF : d;
}

// Grid geometry of one point set (the queries' bounding box in scaled space).
struct GridGeom {
  float lo[3];
  float h, inv_h;
  int dims[3];
};

__device__ __forceinline__ int cell_coord(float y, float lo, float inv_h, int dim) {
  float u = (y - lo) * inv_h;
  int c = (u > 0.0f) ? (u < (float)dim ? (int)u : dim - 1) : 0;  // NaN -> 0 (not used)
  return c;
}

__device__ __forceinline__ FrameDesc load_desc(const DevPlan& P, int f) { return P.frames[f]; }

}  // namespace


constexpr int kMaxGridDim = 1024;  // cells along an axis
// Grid geometry over the bounding box [lo, hi] (scaled space): cubic cells of side h,
// about one reference per cell, at most budget-1 cells in total.
__device__ void set_geometry(FrameState* S, const float* lo, const float* hi, int n_ref, int cell_budget,
                             int per_cell = kRefsPerCell) {
  float ext[3];
  double vol = 1.0;
  for (int d = 0; d < 3; d++) {
    ext[d] = fmaxf(hi[d] - lo[d], 1.0f);
    vol *= ext[d];
  }
  // about kRefsPerCell references per cell: the neighbours a supervoxel keeps then usually
  // lie within the first ring of cells around the query
  const int budget = max(cell_budget - 1, 1);
  const int target = max(1, min(budget, n_ref / per_cell));
  float h = (float)cbrt(vol / target);
  int dims[3] = {1, 1, 1};
  for (int guard = 0; guard < 400; guard++) {
    long long tot = 1;
    for (int d = 0; d < 3; d++) {
      dims[d] = max(1, min(kMaxGridDim, (int)ceilf(ext[d] / h)));
      tot *= dims[d];
    }
    if (tot <= budget) break;
    h *= 1.1f;
  }
  for (int d = 0; d < 3; d++) {
    S->lo[d] = lo[d];
    S->dims[d] = dims[d];
  }
  S->h = h;
  S->inv_h = 1.0f / h;
  S->n_cells = dims[0] * dims[1] * dims[2];
}

// The stream record (SvRec) of supervoxel s (frame-local sl) for the voxel pass.
__device__ void write_sv_rec(const DevPlan& P, const FrameDesc& D, int f, int s, int sl) {
  const int64_t a = D.lptr[sl], b = D.lptr[sl + 1];
  const bool ok = !(a < 0 || b < a || b > D.n_vox || b - a >= (1 << 30));
  const int nv = ok ? (int)(b - a) : 0;
  const int nt = (nv + kVoxTile - 1) / kVoxTile;
  const int r0 = nt ? nv - (nt - 1) * kVoxTile : 0;
  SvRec r;
  const float* comp[4] = {D.query, D.query + D.n_vox, D.query + 2 * D.n_vox, D.img};
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const uintptr_t a0 = nt ? (uintptr_t)(comp[c] + a) : 0;
    const uintptr_t a1 = a0 + 4u * (unsigned)r0;  // first voxel of tile 1
    r.lo0[c] = a0 & ~(uintptr_t)15;
    r.lo1[c] = a1 & ~(uintptr_t)15;
    r.n0[c] = nt ? (unsigned)(((a1 + 15) & ~(uintptr_t)15) - r.lo0[c]) : 0u;
    r.nf[c] = (4u * kVoxTile + ((a1 & 15) ? 16u : 0u)) | ((unsigned)((a0 & 15) >> 2) << 16) |
              ((unsigned)((a1 & 15) >> 2) << 20);
  }
  r.ntiles = nt;
  r.nv = nv;
  r.frame = f;
  r.frame_nsv = D.n_sv;
  r.c0 = D.cent[sl];
  r.c1 = D.cent[(int64_t)D.n_sv + sl];
  r.c2 = D.cent[2 * (int64_t)D.n_sv + sl];
  r.r0 = r0;
  P.sv_rec[s] = r;
  SvLL l;
  l.v0 = D.vox_base + (nt ? a : 0);
  l.nv = nv;
  l.pad = 0;
  l.frame = f;
  l.frame_nsv = D.n_sv;
  l.c0 = r.c0;
  l.c1 = r.c1;
  l.c2 = r.c2;
  l.h0 = l.h1 = l.h2 = 0.0f;  // the moment pass's
  P.sv_ll[s] = l;
}

// ===========================================================================
// build_maps: per frame -- supervoxel/Gaussian -> frame maps, CSR validation,
// centroid bounding box and grid geometry, EM state reset.
// ===========================================================================
__global__ void __launch_bounds__(kFrameThreads) k_build_maps(DevPlan P) {
  // block (f, y): the frame's map stores split over kMapSlices blocks; block (f, 0) also
  // checks the CSR, takes the centroids' bounding box and starts the frame's state
  const int f = blockIdx.x;
  if (f >= P.info->n_frames) return;
  const FrameDesc D = load_desc(P, f);
  const int first = blockIdx.y * blockDim.x + threadIdx.x, stride = kMapSlices * blockDim.x;
  for (int i = first; i < D.n_sv; i += stride) P.sv_frame[D.sv_base + i] = f;
#pragma unroll 4
  for (int i = first; i < D.n_gauss; i += stride) {
    P.g_frame[D.g_base + i] = f;
    P.bcnt[D.g_base + i] = 0;  // M-step and assignment buckets start empty
    P.acnt[D.g_base + i] = 0;
  }
  for (int i = first; i < D.cell_budget; i += stride) P.cell_cnt[D.cell_base + i] = 0;
  if (blockIdx.y != 0) return;
  // the voxel passes' counters, which each pass leaves at zero
  if (f == 0 && threadIdx.x < 3) P.work[threadIdx.x] = 0;
  FrameState* S = &P.state[f];
  __shared__ float smin[3][32], smax[3][32];
  __shared__ int sbad;
  if (threadIdx.x == 0) sbad = 0;
  __syncthreads();
  if (threadIdx.x < kOrderBuckets) {  // the supervoxel order's bucket counts and cursors
    P.ord_hist[f * kOrderBuckets + threadIdx.x] = 0;
    P.ord_cur[f * kOrderBuckets + threadIdx.x] = 0;
  }
  int bad = 0;
  float lo[3] = {kInfF, kInfF, kInfF}, hi[3] = {-kInfF, -kInfF, -kInfF};
  // unrolled so that several supervoxels' loads are in flight at once
#pragma unroll 4
  for (int i = threadIdx.x; i < D.n_sv; i += blockDim.x) {
    const int64_t a = D.lptr[i], b = D.lptr[i + 1];
    if (a < 0 || b < a || b > D.n_vox) bad = 1;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float y = D.cent[(int64_t)d * D.n_sv + i] * D.scale[d];
      if (!isfinite(y)) {
        bad |= 2;
        continue;
      }
      lo[d] = fminf(lo[d], y);
      hi[d] = fmaxf(hi[d], y);
    }
  }
  if (bad) atomicOr(&sbad, bad);
#pragma unroll
  for (int d = 0; d < 3; d++) {
    for (int o = 16; o > 0; o >>= 1) {
      lo[d] = fminf(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], o));
      hi[d] = fmaxf(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], o));
    }
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    for (int d = 0; d < 3; d++) {
      smin[d][w] = lo[d];
      smax[d][w] = hi[d];
    }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int d = 0; d < 3; d++) {
      lo[d] = smin[d][0];
      hi[d] = smax[d][0];
      for (int i = 1; i < (int)(blockDim.x >> 5); i++) {
        lo[d] = fminf(lo[d], smin[d][i]);
        hi[d] = fmaxf(hi[d], smax[d][i]);
      }
      if (!(lo[d] <= hi[d])) {
        lo[d] = 0.0f;
        hi[d] = 0.0f;
      }
    }
    int flags = 0;
    if (sbad & 1) flags |= F_BAD_CSR;
    if (sbad & 2) flags |= F_NAN_INPUT;
    if (D.n_gauss < kJ) flags |= F_FEW_GAUSS;
    set_geometry(S, lo, hi, D.n_gauss, D.cell_budget);
    S->iter = 1;
    S->disp_cum = 0.0;
    S->disp_max = 0u;
    S->knn_searches = 0;
    S->done = (flags & (F_BAD_CSR | F_FEW_GAUSS)) ? kNeverRan : 0;
    S->converged = 0;
    S->flags = flags;
    S->n_dead = 0;
    S->ll = -1.0;
    S->ll1 = -10.0;
    S->ll2 = -100.0;
    S->ll3 = -1000.0;
    S->ll_true = 0.0;
    S->ll_ref = 0.0;
    S->total_alpha = 0.0;
    S->ln_alpha = 0.0;
    S->psi_total[0] = S->psi_total[1] = 0.0;
    S->ll_int[0] = S->ll_int[1] = 0;
    S->ll_frac[0] = S->ll_frac[1] = 0;
    S->sv_done = 0;
    S->blk_done = 0;
  }
}

// Gaussian -> grid cell (or -1 when its float centre is unusable for pruning).
__device__ __forceinline__ int ref_cell_of(const FrameState& S, const FrameDesc& D, float x, float y,
                                           float z) {
  const float ys[3] = {x * D.scale[0], y * D.scale[1], z * D.scale[2]};
#pragma unroll
  for (int d = 0; d < 3; d++)
    if (!isfinite(ys[d]) || fabsf(ys[d]) >= 1e25f) return -1;
  const int cx = cell_coord(ys[0], S.lo[0], S.inv_h, S.dims[0]);
  const int cy = cell_coord(ys[1], S.lo[1], S.inv_h, S.dims[1]);
  const int cz = cell_coord(ys[2], S.lo[2], S.inv_h, S.dims[2]);
  return (cz * S.dims[1] + cy) * S.dims[0] + cx;
}

// The next iteration's records of Gaussian k from its parameters: psi(alpha) and
// E[ln|Lambda|] (in the parity slot), the E-step record (nu W, m, 3/beta, psi(alpha) +
// E[ln|Lambda|]/2, or -inf for a dead Gaussian), the log-likelihood record (-nu W/2 with
// doubled off-diagonals, the log weight 1/2 ln(det W nu^3) - 3/2 ln(2 pi) + ln(alpha), the
// mean) and the float centre the kNN sees (kpos).  With `track`, returns how far that
// centre moved since the previous record (scaled distance, 0 unless live both times),
// which bounds the kNN neighbour lists.
__device__ __forceinline__ double write_records(const DevPlan& P, const FrameDesc& D, int k, int parity, bool dead,
                                                const double* W, double nu, double alpha, double beta,
                                                const double* m, bool track, float4 o = float4{}) {
  double corr;
  const double psa = alpha > 1e-6 ? log(digamma_shift(alpha, &corr)) - corr : digamma(alpha);
  const double eld = dead ? -1e32 : expected_log_det(W, nu);
  gcomp(P, G_PSIA0 + parity, k) = psa;
  gcomp(P, G_ELD0 + parity, k) = eld;
  double* E = P.ec + (int64_t)k * kEcStride;
#pragma unroll
  for (int e = 0; e < 6; e++) E[e] = nu * W[e];
  E[6] = m[0];
  E[7] = m[1];
  E[8] = m[2];
  E[9] = 3.0 / beta;
  E[10] = dead ? -(double)kInfF : psa + 0.5 * eld;
  double* L = P.llc + (int64_t)k * 10;
  L[0] = -0.5 * nu * W[0];
  L[1] = -nu * W[1];
  L[2] = -nu * W[2];
  L[3] = -0.5 * nu * W[3];
  L[4] = -nu * W[4];
  L[5] = -0.5 * nu * W[5];
  L[6] = log_weight(det3(W) * nu * nu * nu, alpha);
  L[7] = m[0];
  L[8] = m[1];
  L[9] = m[2];
  const float x = __double2float_rn(m[0]);
  const float y = __double2float_rn(m[1]);
  const float z = __double2float_rn(m[2]);
  double move = 0.0;
  if (track && !dead) {  // o: the centre kpos held before (loaded by the caller)
    if (o.w != 0.0f) {
      const double a = ((double)x - (double)o.x) * (double)D.scale[0];
      const double b = ((double)y - (double)o.y) * (double)D.scale[1];
      const double c = ((double)z - (double)o.z) * (double)D.scale[2];
      move = sqrt(a * a + b * b + c * c);
    }
  }
  P.kpos[k] = make_float4(x, y, z, dead ? 0.0f : 1.0f);
  return move;
}

// A live Gaussian's float centre (kpos) into its grid cell (capacity kCellCap; a full cell
// flags the frame, whose kNN then scans every Gaussian).
// `cell`: ref_cell_of the centre, or -1 (outside every cell: not inserted).
__device__ __forceinline__ void grid_insert_at(const DevPlan& P, const FrameDesc& D, int cell, int k, float4 c4) {
  if (cell >= 0) {
    const int g = D.cell_base + cell;
    const int pos = atomicAdd(&P.cell_cnt[g], 1);
    if (pos < kCellCap)
      P.cell_refs[(int64_t)g * kCellCap + pos] = make_float4(c4.x, c4.y, c4.z, __int_as_float(k - D.g_base));
    else
      atomicOr(&P.state[D.frame_id].flags, F_CELL_OVERFLOW);
  }
}
__device__ __forceinline__ void grid_insert(const DevPlan& P, const FrameDesc& D, const FrameState& S, int k,
                                            float4 c4) {
  grid_insert_at(P, D, ref_cell_of(S, D, c4.x, c4.y, c4.z), k, c4);
}


// Run by the last Gaussian chunk of a frame to finish (import or kill step): the alpha
// total as a fixed-order sum of the chunk partials, psi and ln of it for the next
// iteration, and the dead count.
__device__ void frame_tail(const DevPlan& P, int f, int next_parity) {
  const FrameDesc D = load_desc(P, f);
  FrameState* S = &P.state[f];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (w == 0) {
    const double a = warp_sum_range(P.alpha_part_f, D.gchunk_base, D.n_gchunks);
    int nd = 0;
    for (int i = lane; i < D.n_gchunks; i += 32) nd += P.dead_part[D.gchunk_base + i];
    nd = warp_sum_i(nd);
    if (lane == 0) {
      S->total_alpha = a;
      S->ln_alpha = log(a);
      S->psi_total[next_parity] = digamma(a);
      S->n_dead = nd;
      S->blk_done = 0;
      S->disp_cum += (double)__uint_as_float(S->disp_max);
      S->disp_max = 0u;
    }
  }
}

// The last-arriving chunk of frame f runs frame_tail.  Every chunk calls this after its
// own writes; no thread waits on another.
__device__ __forceinline__ void chunk_done(const DevPlan& P, int f, int n_chunks, int next_parity) {
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = (atomicAdd(&P.state[f].blk_done, 1) == n_chunks - 1) ? 1 : 0;
  __syncthreads();
  if (s_last) {
    __threadfence();
    frame_tail(P, f, next_parity);
  }
}

// ===========================================================================
// import: AoS (288-byte records) -> SoA, validation, preparation of iteration 1.
// ===========================================================================
__global__ void __launch_bounds__(kGChunk) k_import(DevPlan P) {
  const int c = blockIdx.x;
  if (c >= P.info->n_gchunks) return;
  const GChunk ch = P.gchunks[c];
  const FrameDesc D = load_desc(P, ch.frame);
  const FrameState& S = P.state[ch.frame];
  __shared__ double shd[kGChunk / 32];
  __shared__ int shi[kGChunk / 32];
  const int k = ch.g_begin + threadIdx.x;
  double alpha = 0.0;
  int dead = 0;
  if (k < ch.g_end) {
    const TgmmGaussian& g = D.gm[k - D.g_base];
    bool bad = false;
    gcomp(P, G_BETA, k) = g.beta_k;
    gcomp(P, G_NU, k) = g.nu_k;
    gcomp(P, G_ALPHA, k) = g.alpha_k;
    for (int d = 0; d < 3; d++) gcomp(P, G_M0 + d, k) = g.m_k[d];
    for (int e = 0; e < 6; e++) gcomp(P, G_W0 + e, k) = g.W_k[e];
    gcomp(P, G_BETAO, k) = g.beta_o;
    gcomp(P, G_NUO, k) = g.nu_o;
    gcomp(P, G_ALPHAO, k) = g.alpha_o;
    for (int d = 0; d < 3; d++) gcomp(P, G_MO0 + d, k) = g.m_o[d];
    for (int e = 0; e < 6; e++) gcomp(P, G_WO0 + e, k) = g.W_o[e];
    P.fixed[k] = g.fixed ? 1 : 0;
    bad = isnan(g.beta_k) || isnan(g.nu_k) || isnan(g.alpha_k);
    for (int d = 0; d < 3; d++) bad = bad || isnan(g.m_k[d]);
    for (int e = 0; e < 6; e++) bad = bad || isnan(g.W_k[e]);
    if (bad) atomicOr(&P.state[ch.frame].flags, F_NAN_INPUT);
    // the first iteration's records and grid entry from the values just read
    const bool is_dead = is_dead_prior(g.m_o[0]);
    write_records(P, D, k, 1, is_dead, g.W_k, g.nu_k, g.alpha_k, g.beta_k, g.m_k, false);
    if (!is_dead) grid_insert(P, D, S, k, P.kpos[k]);
    alpha = g.alpha_k;
    dead = is_dead ? 1 : 0;
  }
  chunk_partials(alpha, dead, shd, shi, P.alpha_part_f, P.dead_part, c);
  chunk_done(P, ch.frame, D.n_gchunks, 1);
}

// ===========================================================================
// order: once per call.  The supervoxels' stream records, and the supervoxels of each
// frame by descending tile count (counting sort, ties in any order), frames in batch order.
// The voxel passes take supervoxels in this order, so a frame's last supervoxels are its
// smallest and no warp is left with a large one after the others ran out of work.  Their
// sums do not depend on the order.
// ===========================================================================

__device__ __forceinline__ int order_bucket(const FrameDesc& D, int sl) {
  const int64_t a = D.lptr[sl], b = D.lptr[sl + 1];
  const int64_t nv = (a < 0 || b < a || b > D.n_vox) ? 0 : b - a;
  const int64_t nt = (nv + kVoxTile - 1) / kVoxTile;
  return nt < kOrderBuckets - 1 ? (int)nt : kOrderBuckets - 1;
}

// k_sv_records: thread per supervoxel -- its stream record, and its bucket counted in its
// frame's histogram (lanes of a warp with the same frame and bucket add once).
__global__ void __launch_bounds__(256) k_sv_records(DevPlan P) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = s < P.info->total_sv;
  int key = -1;
  if (in) {
    const int f = P.sv_frame[s];
    const FrameDesc D = load_desc(P, f);
    const int sl = s - D.sv_base;
    write_sv_rec(P, D, f, s, sl);
    key = f * kOrderBuckets + order_bucket(D, sl);
  }
  const unsigned m = __match_any_sync(0xffffffffu, key);
  if (in && (m & ((1u << (threadIdx.x & 31)) - 1u)) == 0) atomicAdd(&P.ord_hist[key], __popc(m));
}

// k_order_base: one warp per frame -- the buckets' first places, largest tile counts first.
__global__ void __launch_bounds__(32) k_order_base(DevPlan P) {
  const int f = blockIdx.x;
  if (f >= P.info->n_frames || threadIdx.x != 0) return;
  int run = 0;
  for (int b = kOrderBuckets - 1; b >= 0; b--) {
    const int c = P.ord_hist[f * kOrderBuckets + b];
    P.ord_hist[f * kOrderBuckets + b] = run;  // from here on: the bucket's base
    run += c;
  }
}

// k_order_scatter: thread per supervoxel -- its place, its bucket's base plus a cursor
// (one atomic per warp and bucket).  Places within a bucket depend on the run; the voxel
// pass's sums do not.
__global__ void __launch_bounds__(256) k_order_scatter(DevPlan P) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  const bool in = s < P.info->total_sv;
  int key = -1, base = 0;
  if (in) {
    const int f = P.sv_frame[s];
    const FrameDesc D = load_desc(P, f);
    key = f * kOrderBuckets + order_bucket(D, s - D.sv_base);
    base = D.sv_base + P.ord_hist[key];
  }
  const unsigned m = __match_any_sync(0xffffffffu, key);
  const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
  int start = 0;
  if (in && lane == lead) start = atomicAdd(&P.ord_cur[key], __popc(m));
  start = __shfl_sync(m, start, lead);
  if (in) P.sv_order[base + start + __popc(m & ((1u << lane) - 1u))] = s;
}


// ===========================================================================
// knn_estep: a group of G lanes per supervoxel (32 / G supervoxels per warp; G = 4, 8, 16
// or 32, chosen per plan, by tgmm_plan_autotune or tgmm_plan_set_knn_group; every G gives
// the same bits).
// Exact 5-NN of the centroid among the frame's Gaussian centres: from the supervoxel's list of
// kNbr near Gaussians while that settles them, else by a search of the grid that also renews the
// list.  The kernel of its own collects and ranks the references within a limit
// (knn_group_collect); where that does not settle it, and inside the voxel pass, the group's lanes
// split each ring of grid cells, keep private lists pruned by the group's current last distance,
// and merge them after each ring by rounds of a group-wide (distance, index) arg-min
// (knn_group_search).  Then the E-step from the supervoxel's moments, candidate j
// on lane j mod G of the group (lane 0 also takes candidate 4 when G = 4):
//   L_j = sum_v [-1/2 (3/beta + nu d'Wd) + E ln pi + 1/2 E ln|Lambda|]
//       = -1/2 (3 n/beta + nu tr(W D)) + n (psi(alpha) - psi(sum alpha) + 1/2 E ln|Lambda|),
//   D = sum_v (x_v - m)(x_v - m)' = G2 - G1 u' - u G1' + n u u',  u = m - c_s,
// in FP64; then the reference's float-storage semantics (empty supervoxel -> 0, dead
// candidate or |L| beyond float range -> -inf) and rnk_j = 1 / sum_i exp(L_i - L_j).
// Pairs with rnk > 1e-3 go to the Gaussian's M-step bucket.
// ===========================================================================
constexpr int kKnnWarps = 4;  // warps per block; the lanes per supervoxel (G) come from the plan
#ifndef TGMM_KNN_BLOCKS
#define TGMM_KNN_BLOCKS 8  // 64 registers: the list path of 20,000 supervoxels in one wave at 4 or 8 lanes
#endif
constexpr int kKnnBlocks = TGMM_KNN_BLOCKS;  // resident blocks per SM the kNN/E-step is compiled for

// group-wide lexicographic arg-min of (d, i); every lane of the group gets the winner
template <int G>
__device__ __forceinline__ void group_min_pair(float& d, int& i, unsigned gmask) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const float od = __shfl_xor_sync(gmask, d, o);
    const int oi = __shfl_xor_sync(gmask, i, o);
    if (before(od, oi, d, i)) {
      d = od;
      i = oi;
    }
  }
}

// merge the group's sorted lists into its top-N (identical in every lane of the group)
template <int G, int N>
__device__ __forceinline__ void group_merge_topn(TopN<N>& mine, TopN<N>& out, unsigned gmask) {
#pragma unroll
  for (int r = 0; r < N; r++) {
    float d = mine.d[0];
    int i = mine.i[0];
    group_min_pair<G>(d, i, gmask);
    out.d[r] = d;
    out.i[r] = i;
    if (mine.i[0] == i && mine.d[0] == d && i != 0x7fffffff) {  // pop the front of the winner
#pragma unroll
      for (int q = 0; q < N - 1; q++) {
        mine.d[q] = mine.d[q + 1];
        mine.i[q] = mine.i[q + 1];
      }
      mine.d[N - 1] = kInfF;
      mine.i[N - 1] = 0x7fffffff;
    }
  }
}

// group-wide lexicographic arg-max of (d, i)
template <int G>
__device__ __forceinline__ void group_max_pair(float& d, int& i, unsigned gmask) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    const float od = __shfl_xor_sync(gmask, d, o);
    const int oi = __shfl_xor_sync(gmask, i, o);
    if (before(d, i, od, oi)) {
      d = od;
      i = oi;
    }
  }
}

// Where a query sits in the grid: its cell, the gaps to that cell's faces, and the float
// rounding of the scaled coordinates and faces (eps0; distances of d add 1e-6 d).
struct GridPlace {
  int c[3];
  float f0[3], f1[3];  // gaps to the cell's lower and upper faces
  float delta, eps0;   // the smallest gap; the rounding
  __device__ __forceinline__ GridPlace(float q0, float q1, float q2, const float* s, const GridGeom& g) {
    const float y[3] = {q0 * s[0], q1 * s[1], q2 * s[2]};
    float ymax = 0.0f;
    delta = kInfF;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      c[a] = cell_coord(y[a], g.lo[a], g.inv_h, g.dims[a]);
      f0[a] = y[a] - (g.lo[a] + c[a] * g.h);
      f1[a] = (g.lo[a] + (c[a] + 1) * g.h) - y[a];
      delta = fminf(delta, fminf(f0[a], f1[a]));
      ymax = fmaxf(ymax, fabsf(y[a]));
    }
    delta = fmaxf(delta, 0.0f);
    eps0 = 4e-3f + 1e-6f * ymax;
  }
  // A squared distance below which every reference lies in the cells at Chebyshev distance
  // <= r (0: none is known).  References outside the box sit in the boundary cells, farther
  // from a query inside it than those cells.
  __device__ __forceinline__ float bound2(int r, float h) const {
    const float lb = r * h + delta, m = lb - (eps0 + 1e-6f * lb);
    return m > 0.0f ? m * m : 0.0f;
  }
  // squared lower bound of the distance along axis a to the cells at offset o
  __device__ __forceinline__ float gap2(int a, int o, float h) const {
    const float gap = o < 0 ? f0[a] + (float)(-o - 1) * h : f1[a] + (float)(o - 1) * h;
    const float m = fmaxf(gap - eps0 - 1e-6f * gap, 0.0f);
    return o == 0 ? 0.0f : m * m;
  }
};

// Up to N nearest, at least kJ, by collecting instead of keeping sorted lists: the group's lanes
// put every reference within a limit into `keep` (shared memory, unsorted), then each ranks its
// share against all.  The limit is a distance that should hold 2 N at the grid's mean density
// and for which the 27 cells around the query are complete, on fewer than kJ a wider one; or
// (td0, ti0), a (distance, index) no smaller than the N-th neighbour's, where that is nearer.
// Every reference not returned is at the squared
// distance `rest` or farther.  False when the cells within two of the query's do not settle it:
// the caller runs the ring search.  20,000 supervoxels that all search: 72 us a launch with
// sorted lists of eight per lane and their merges, 49 us this way (8 lanes).
constexpr int kKnnKeep = 64;  // references kept; N more places hold the result
template <int G, int N>
__device__ __forceinline__ bool knn_group_collect(float q0, float q1, float q2, const float* s, const GridGeom& g,
                                                  const int32_t* __restrict__ ccnt, const float4* __restrict__ refs,
                                                  float2* keep, int* count, TopN<N>& best, float& rest,
                                                  unsigned gmask, int gl, float td0, int ti0) {
  const GridPlace p(q0, q1, q2, s, g);
  const float near2 = p.bound2(1, g.h), far2 = p.bound2(2, g.h);
  float lim = fminf(1.17f * g.h * g.h, near2);  // (16 3 / (4 pi 3))^(2/3) h^2
  const bool known = td0 < lim;
  if (known) lim = td0;
  auto scan = [&](int cell, int e) {
    const float4* cr = refs + (int64_t)cell * kCellCap;
    for (int k = 0; k < e; k++) {
      const float4 rr = cr[k];
      const float d = knn_dist(q0, q1, q2, rr.x, rr.y, rr.z, s);
      if (known ? !before(td0, ti0, d, __float_as_int(rr.w)) : d < lim) {
        const int at = atomicAdd(count, 1);
        if (at < kKnnKeep) keep[at] = make_float2(d, rr.w);
      }
    }
  };
  // the cell at an offset, or -1 outside the grid or past the limit
  auto cell_at = [&](int dx, int dy, int dz) {
    const int x = p.c[0] + dx, yy = p.c[1] + dy, z = p.c[2] + dz;
    const bool in = x >= 0 && yy >= 0 && z >= 0 && x < g.dims[0] && yy < g.dims[1] && z < g.dims[2] &&
                    !(p.gap2(0, dx, g.h) + p.gap2(1, dy, g.h) + p.gap2(2, dz, g.h) > lim);
    return in ? (z * g.dims[1] + yy) * g.dims[0] + x : -1;
  };
  for (int tries = 0; tries < 3; tries++) {
    const bool one = lim <= near2;
    if (gl == 0) *count = 0;
    __syncwarp(gmask);
    if (one) {
      constexpr int kPer = (27 + G - 1) / G;
      int cq[kPer], eq[kPer];
#pragma unroll
      for (int q = 0; q < kPer; q++) {
        const int idx = gl + G * q;
        cq[q] = idx < 27 ? cell_at(idx % 3 - 1, (idx / 3) % 3 - 1, idx / 9 - 1) : -1;
        eq[q] = cq[q] >= 0 ? min(ccnt[cq[q]], kCellCap) : 0;
      }
#pragma unroll
      for (int q = 0; q < kPer; q++) scan(cq[q], eq[q]);
    } else {
      for (int idx = gl; idx < 125; idx += G) {
        const int c = cell_at(idx % 5 - 2, (idx / 5) % 5 - 2, idx / 25 - 2);
        if (c >= 0) scan(c, min(ccnt[c], kCellCap));
      }
    }
    __syncwarp(gmask);
    const int n = *count;
    if (n > kKnnKeep) return false;
    if (n >= kJ) {
      for (int a = gl; a < n; a += G) {
        const float2 e = keep[a];
        int rank = 0;
        for (int o = 0; o < n; o++) {
          const float2 f = keep[o];
          rank += before(f.x, __float_as_int(f.y), e.x, __float_as_int(e.y)) ? 1 : 0;
        }
        if (rank < N) keep[kKnnKeep + rank] = e;
      }
      __syncwarp(gmask);
#pragma unroll
      for (int j = 0; j < N; j++) {
        const float2 e = j < n ? keep[kKnnKeep + j] : make_float2(kInfF, __int_as_float(0x7fffffff));
        best.d[j] = e.x;
        best.i[j] = __float_as_int(e.y);
      }
      rest = n < N ? lim : best.d[N - 1];
      return true;
    }
    __syncwarp(gmask);  // every lane has read the count
    if (known || !(lim < far2)) return false;
    lim = fminf(lim * (n == 0 ? 4.0f : 2.0f), far2);
  }
  return false;
}

// Exact N nearest over the grid rings.  (td0, ti0): a (distance, index) no smaller than
// the true N-th neighbour's (the N-th of N known Gaussians), or +inf; refs after it in
// (distance, index) order cannot be among the N and are rejected without an insertion.
template <int G, int N>
__device__ void knn_group_search(float q0, float q1, float q2, const float* s, const GridGeom& g,
                                 const int32_t* __restrict__ ccnt, const float4* __restrict__ refs, TopN<N>& best,
                                 unsigned gmask, int gl, float td0, int ti0) {
  const float y[3] = {q0 * s[0], q1 * s[1], q2 * s[2]};
  int c[3];
  float delta = kInfF;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    c[a] = cell_coord(y[a], g.lo[a], g.inv_h, g.dims[a]);
    const float f0 = y[a] - (g.lo[a] + c[a] * g.h);
    const float f1 = (g.lo[a] + (c[a] + 1) * g.h) - y[a];
    delta = fminf(delta, fminf(f0, f1));
  }
  delta = fmaxf(delta, 0.0f);
  topn_init<N>(best);
  const int maxr = max(1, max(g.dims[0], max(g.dims[1], g.dims[2])));
  // the first pass covers rings 0 and 1 (27 cells), later passes one ring
  for (int r = 1; r <= maxr; ++r) {
    TopN<N> t;
    topn_init<N>(t);
    // prune with the group's current N-th (or the starting bound): a ref must not come
    // after it to matter
    const bool use_best = before(best.d[N - 1], best.i[N - 1], td0, ti0);
    const float td = use_best ? best.d[N - 1] : td0;
    const int ti = use_best ? best.i[N - 1] : ti0;
    auto scan_refs = [&](int cell, int e) {
      const float4* cr = refs + (int64_t)cell * kCellCap;
      for (int k = 0; k < e; ++k) {
        const float4 rr = cr[k];
        const float d = knn_dist(q0, q1, q2, rr.x, rr.y, rr.z, s);
        const int id = __float_as_int(rr.w);
        if (!before(td, ti, d, id)) topn_insert<N>(t, d, id);
      }
    };
    auto scan_cell = [&](int dx, int dy, int dz) {
      const int x = c[0] + dx, yy = c[1] + dy, z = c[2] + dz;
      if (x < 0 || yy < 0 || z < 0 || x >= g.dims[0] || yy >= g.dims[1] || z >= g.dims[2]) return;
      const int cell = (z * g.dims[1] + yy) * g.dims[0] + x;
      scan_refs(cell, min(ccnt[cell], kCellCap));
    };
    // the cells of ring r (the whole cube for r = 1), with constant divisors for the
    // rings a search usually needs
    if (r == 1) {
      // the lane's cells of the 3x3x3 cube: their counts first, as independent loads
      constexpr int kPer = (27 + G - 1) / G;
      int cq[kPer], eq[kPer];
#pragma unroll
      for (int q = 0; q < kPer; q++) {
        const int idx = gl + G * q;
        const int x = c[0] + idx % 3 - 1, yy = c[1] + (idx / 3) % 3 - 1, z = c[2] + idx / 9 - 1;
        const bool in = idx < 27 && x >= 0 && yy >= 0 && z >= 0 && x < g.dims[0] && yy < g.dims[1] && z < g.dims[2];
        cq[q] = in ? (z * g.dims[1] + yy) * g.dims[0] + x : 0;
        eq[q] = in ? min(ccnt[cq[q]], kCellCap) : 0;
      }
#pragma unroll
      for (int q = 0; q < kPer; q++) scan_refs(cq[q], eq[q]);
    } else if (r == 2) {
      for (int idx = gl; idx < 125; idx += G) {
        const int dx = idx % 5 - 2, dy = (idx / 5) % 5 - 2, dz = idx / 25 - 2;
        if (max(abs(dx), max(abs(dy), abs(dz))) == 2) scan_cell(dx, dy, dz);
      }
    } else if (r == 3) {
      for (int idx = gl; idx < 343; idx += G) {
        const int dx = idx % 7 - 3, dy = (idx / 7) % 7 - 3, dz = idx / 49 - 3;
        if (max(abs(dx), max(abs(dy), abs(dz))) == 3) scan_cell(dx, dy, dz);
      }
    } else {
      const int side = 2 * r + 1;
      const int cube = side * side * side;
      for (int idx = gl; idx < cube; idx += G) {
        const int dx = idx % side - r, dy = (idx / side) % side - r, dz = idx / (side * side) - r;
        if (max(abs(dx), max(abs(dy), abs(dz))) == r) scan_cell(dx, dy, dz);
      }
    }
    // lane 0 of the group also carries the previous best (disjoint from this ring's refs)
    if (gl == 0) {
#pragma unroll
      for (int q = 0; q < N; q++) topn_insert<N>(t, best.d[q], best.i[q]);
    }
    TopN<N> merged;
    group_merge_topn<G, N>(t, merged, gmask);
    best = merged;
    const float lb = r * g.h + delta;
    const float eps = 4e-3f + 1e-6f * lb;
    if (lb > eps) {
      const float bound = (lb - eps) * (lb - eps);
      if (best.d[N - 1] < bound) break;
    }
  }
}

// The kNN/E-step of supervoxel s for iteration `it` by the G lanes of one group (lane gl
// of the group whose first lane is gbase).  Its candidates and responsibilities go to the
// buffers of the iteration's parity.  It reads the frame state the kill step of iteration
// it - 1 left (grid, neighbour-list bound, psi of the alpha total) and the done flag:
// when it runs inside the voxel pass of iteration it - 1 (k_ll_stream), that pass may end
// the frame meanwhile, and the results of an iteration that does not run are never read.
// keep, count: the shared scratch of the group for a search (nullptr: the ring search).
template <int G>
__device__ __forceinline__ void knn_estep_sv(const DevPlan& P, int s, int it, int gl, int gbase, unsigned gmask,
                                             float2* keep, int* count) {
  static_assert(G >= 4 && G <= 32 && (G & (G - 1)) == 0, "groups of 4 to 32 lanes");
  // per lane: list members gl + G q (q < kM) and candidates gl + G q (q < kC); one of each
  // for groups of 8 or more lanes
  constexpr int kM = (kNbr + G - 1) / G, kC = (kJ + G - 1) / G;
  // whole groups leave together; every shuffle below names only the group's lanes
  if (s >= P.info->total_sv) return;
  // what needs only s goes out first, ahead of the frame's state and descriptor: the
  // supervoxel's stream record (frame, centroid, voxel count), the list member of this lane
  // (a global Gaussian index, so that its centre loads beside the frame's state) and the
  // list's bound, and (into L1) the moments the E-step reads
  const SvLL R = P.sv_ll[s];
  int lk[kM];
  double nbr_bound = 0.0;
#pragma unroll
  for (int q = 0; q < kM; q++) lk[q] = 0x7fffffff;
  if (it > 1) {
#pragma unroll
    for (int q = 0; q < kM; q++)
      if (gl + G * q < kNbr) lk[q] = P.nbr[(int64_t)s * kNbr + gl + G * q];
    nbr_bound = P.nbr_b[s];
  }
#pragma unroll
  for (int q = 0; q < (9 + G - 1) / G; q++)  // the nine moment rows M_E0 .. M_EE22 over the group
    if (gl + G * q < 9)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(P.mom + (int64_t)(M_E0 + gl + G * q) * P.max_sv + s));
  const int f = R.frame;
  float4 lpos[kM];
#pragma unroll
  for (int q = 0; q < kM; q++) {
    lpos[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (it > 1 && gl + G * q < kNbr && lk[q] != 0x7fffffff) lpos[q] = P.kpos[lk[q]];
  }
  const FrameState& S = P.state[f];
  if (*(volatile const int32_t*)&S.done) return;
  const FrameDesc D = load_desc(P, f);
  const double psi_tot = S.psi_total[it & 1];  // loaded beside the frame's other scalars
  const int sl = s - D.sv_base;
  const int Sf = D.n_sv;
  const float q0 = R.c0, q1 = R.c1, q2 = R.c2;  // the frame's centroid of s, as the E-step reads it
  GridGeom g;
  for (int d = 0; d < 3; d++) {
    g.lo[d] = S.lo[d];
    g.dims[d] = S.dims[d];
  }
  g.h = S.h;
  g.inv_h = S.inv_h;
  const bool grid_ok = !(S.flags & F_CELL_OVERFLOW);
  const double disp = S.disp_cum;
  Top5 t;
  // After the first iteration: the supervoxel's neighbour list, the kNbr nearest Gaussians
  // when it was last searched (at displacement bound disp_b), member i on lane i mod G.  A
  // Gaussian outside the list was then at scaled distance >= rho from the centroid and has
  // since moved at most disp - disp_b, so the five nearest members (current centres, the
  // same FP32 distances and (distance, index) order) are the exact five nearest whenever
  //   sqrt(d5) (1 + 1e-6) + disp < nbr_b = rho (1 - 1e-6) - 4e-3 + disp_b;
  // the margins cover the FP32 rounding of the distances.  Otherwise the supervoxel runs
  // the exact search for the kNbr nearest and keeps them as its new list.
  float ld[kM];
  bool have = false;
#pragma unroll
  for (int q = 0; q < kM; q++) ld[q] = kInfF;
  if (it > 1) {
    Top5 mine;
    top5_init(mine);
#pragma unroll
    for (int q = 0; q < kM; q++) {
      if (gl + G * q < kNbr && lk[q] != 0x7fffffff)
        ld[q] = knn_dist(q0, q1, q2, lpos[q].x, lpos[q].y, lpos[q].z, D.scale);
      if (kM == 1) {
        mine.d[0] = ld[q];
        mine.i[0] = lk[q];
      } else {
        topn_insert<kJ>(mine, ld[q], lk[q]);
      }
    }
    group_merge_topn<G, kJ>(mine, t, gmask);
    have = t.d[kJ - 1] < kInfF && sqrt((double)t.d[kJ - 1]) * (1.0 + 1e-6) + disp < nbr_bound;
  }
  if (!have) {
    // starting bound: the kNbr-th of the list members at their current centres
    float td0 = kInfF;
    int ti0 = 0x7fffffff;
    if (it > 1) {
      float dj = -1.0f;  // lanes without a member never win the arg-max
      int ij = -1;
#pragma unroll
      for (int q = 0; q < kM; q++)
        if (gl + G * q < kNbr && before(dj, ij, ld[q], lk[q])) {
          dj = ld[q];
          ij = lk[q];
        }
      group_max_pair<G>(dj, ij, gmask);
      td0 = dj;
      ti0 = ij >= 0 && ij != 0x7fffffff ? ij - D.g_base : ij;  // the search's frame-local order
      if (gl == 0) atomicAdd(&P.state[f].knn_searches, 1);
    }
    TopN<kNbr> nb;
    topn_init<kNbr>(nb);
    float rest = -1.0f;  // squared distance of what the list leaves out, where it is not its last's
    if (grid_ok && !(keep && knn_group_collect<G, kNbr>(q0, q1, q2, D.scale, g, P.cell_cnt + D.cell_base,
                                                        P.cell_refs + (int64_t)D.cell_base * kCellCap, keep, count, nb,
                                                        rest, gmask, gl, td0, ti0)))
      knn_group_search<G, kNbr>(q0, q1, q2, D.scale, g, P.cell_cnt + D.cell_base,
                                P.cell_refs + (int64_t)D.cell_base * kCellCap, nb, gmask, gl, td0, ti0);
    if (!grid_ok || !(nb.d[kJ - 1] < kInfF)) {
      // fewer than five finite distances: exact scan of every Gaussian of the frame
      TopN<kNbr> m;
      topn_init<kNbr>(m);
      for (int kl = gl; kl < D.n_gauss; kl += G) {
        const int k = D.g_base + kl;
        const float x = __double2float_rn(gcomp(P, G_M0, k));
        const float y = __double2float_rn(gcomp(P, G_M1, k));
        const float z = __double2float_rn(gcomp(P, G_M2, k));
        topn_insert<kNbr>(m, knn_dist(q0, q1, q2, x, y, z, D.scale), kl);
      }
      group_merge_topn<G, kNbr>(m, nb, gmask);
    }
    // (frame-local indices from the search; global ones from here on)
#pragma unroll
    for (int j = 0; j < kJ; j++) {
      t.d[j] = nb.d[j];
      t.i[j] = nb.i[j] == 0x7fffffff ? nb.i[j] : D.g_base + nb.i[j];
    }
#pragma unroll
    for (int m = 0; m < kM; m++) {
      int mi = 0x7fffffff;
#pragma unroll
      for (int q = 0; q < kNbr; q++)
        if (gl + G * m == q) mi = nb.i[q];
      if (gl + G * m < kNbr) P.nbr[(int64_t)s * kNbr + gl + G * m] = mi == 0x7fffffff ? mi : D.g_base + mi;
    }
    if (rest < 0.0f) rest = nb.d[kNbr - 1];
    if (gl == 0) P.nbr_b[s] = rest < kInfF ? sqrt((double)rest) * (1.0 - 1e-6) - 4e-3 + disp : (double)kInfF;
  }
  // E-step: candidate j = gl + G q on its lane (its voxel count: 0 for an invalid range, which
  // flags the frame)
  const double n = (double)R.nv;
  int kc[kC];
  double Lc[kC];
#pragma unroll
  for (int q = 0; q < kC; q++) {
    const int jj = gl + G * q;
    int k = 0;
#pragma unroll
    for (int j = 0; j < kJ; j++)
      if (jj == j) k = t.i[j];
    kc[q] = k;
    double Lj = 0.0;
    if (jj < kJ && n != 0.0) {
      const double* E = P.ec + (int64_t)k * kEcStride;
      const double2 e01 = *(const double2*)(E), e23 = *(const double2*)(E + 2), e45 = *(const double2*)(E + 4);
      const double2 e67 = *(const double2*)(E + 6), e89 = *(const double2*)(E + 8), e10 = *(const double2*)(E + 10);
      const double cst = e10.x;  // psi(alpha) + E[ln|Lambda|]/2, -inf when dead
      if (cst == -(double)kInfF) {
        Lj = -(double)kInfF;
      } else {
        double G1[3], G2[6];
#pragma unroll
        for (int i = 0; i < 3; i++) G1[i] = P.mom[(int64_t)(M_E0 + i) * P.max_sv + s];
#pragma unroll
        for (int i = 0; i < 6; i++) G2[i] = P.mom[(int64_t)(M_EE00 + i) * P.max_sv + s];
        const double u0 = e67.x - (double)q0, u1 = e67.y - (double)q1, u2 = e89.x - (double)q2;
        const double D00 = G2[0] - 2.0 * G1[0] * u0 + n * u0 * u0;
        const double D01 = G2[1] - (G1[0] * u1 + u0 * G1[1]) + n * u0 * u1;
        const double D02 = G2[2] - (G1[0] * u2 + u0 * G1[2]) + n * u0 * u2;
        const double D11 = G2[3] - 2.0 * G1[1] * u1 + n * u1 * u1;
        const double D12 = G2[4] - (G1[1] * u2 + u1 * G1[2]) + n * u1 * u2;
        const double D22 = G2[5] - 2.0 * G1[2] * u2 + n * u2 * u2;
        // nu * tr(W D) with nu*W from the record: W00 D00 + W11 D11 + W22 D22 + 2 (W01 D01 + W02 D02 + W12 D12)
        const double tr = e01.x * D00 + e23.y * D11 + e45.y * D22 + 2.0 * (e01.y * D01 + e23.x * D02 + e45.x * D12);
        Lj = -0.5 * (n * e89.y + tr) + n * (cst - psi_tot);
        if (Lj < -(double)FLT_MAX) Lj = -(double)kInfF;
        if (Lj > (double)FLT_MAX) Lj = (double)kInfF;
      }
    }
    Lc[q] = Lj;
  }
  // rnk_j = 1 / sum_i exp(L_i - L_j), the sum over i in increasing order
  double Li[kJ];
#pragma unroll
  for (int i = 0; i < kJ; i++) Li[i] = __shfl_sync(gmask, Lc[i / G], gbase + i % G);
#pragma unroll
  for (int q = 0; q < kC; q++) {
    const int j = gl + G * q;
    if (j < kJ) {
      const double Lj = Lc[q];
      const int k = kc[q];
      double acc = 0.0;
#pragma unroll
      for (int i = 0; i < kJ; i++) acc += exp(Li[i] - Lj);
      const float r = __double2float_rn(1.0 / acc);
      const int64_t pos = (int64_t)j * Sf + sl;
      cand_buf(P, it)[(int64_t)s * kJ + j] = k;
      rnk_buf(P, it)[(int64_t)s * kJ + j] = r;
      if ((double)r > 1e-3) {
        const int b = atomicAdd(&P.bcnt[k], 1);
        if (b < kBucketCap) P.bucket[(int64_t)k * kBucketCap + b] = (int)pos;
      }
    }
  }
}

template <int G>
__global__ void __launch_bounds__(kKnnWarps * 32, kKnnBlocks) k_knn_estep(DevPlan P) {
  const int lane = threadIdx.x & 31;
  const int gl = lane & (G - 1), gbase = lane - gl;
  const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << G) - 1u) << gbase;
  const int s = blockIdx.x * (kKnnWarps * 32 / G) + (threadIdx.x >> 5) * (32 / G) + gbase / G;
  // the group's shared scratch of a search (see knn_group_collect)
  __shared__ float2 s_keep[kKnnWarps * 32 / G][kKnnKeep + kNbr];
  __shared__ int s_count[kKnnWarps * 32 / G];
  const int grp = threadIdx.x / G;
  knn_estep_sv<G>(P, s, P.iter, gl, gbase, gmask, s_keep[grp], &s_count[grp]);
}

// M-step contribution of one (supervoxel, slot) pair to Gaussian k, moments re-centred
// from the supervoxel centroid to m_ref, the Gaussian's prior mean m_o.  m_o stays fixed
// during a call, so responsibilities that repeat bit for bit give parameters that repeat
// bit for bit -- the exact fixed point the reference's tol = 0 stopping rule looks for:
//   A0 += r H0;  A1 += r (H1 + H0 d);  A2 += r (H2 + H1 d' + d H1' + H0 d d'),  d = c_s - m_ref.
// The inputs of one (supervoxel, slot) pair, loaded apart from their use so that the loads
// of several pairs can be in flight together.
struct MEntry {
  float r, c[3];
  double h0, h1[3], h2[6];
};

__device__ __forceinline__ MEntry mentry_load(const DevPlan& P, const FrameDesc& D, int p) {
  const int Sf = D.n_sv;
  const int j = p / Sf, sl = p - j * Sf;
  const int s = D.sv_base + sl;
  MEntry e;
  e.r = rnk_buf(P, P.iter)[(int64_t)s * kJ + j];
  e.c[0] = D.cent[sl];
  e.c[1] = D.cent[(int64_t)Sf + sl];
  e.c[2] = D.cent[2 * (int64_t)Sf + sl];
  e.h0 = P.mom[(int64_t)M_I * P.max_sv + s];
#pragma unroll
  for (int i = 0; i < 3; i++) e.h1[i] = P.mom[(int64_t)(M_IE0 + i) * P.max_sv + s];
#pragma unroll
  for (int i = 0; i < 6; i++) e.h2[i] = P.mom[(int64_t)(M_IEE00 + i) * P.max_sv + s];
  return e;
}

__device__ __forceinline__ void mentry_add(const MEntry& e, const double* mref, double* A) {
  const double r = (double)e.r;
  const double d0 = (double)e.c[0] - mref[0];
  const double d1 = (double)e.c[1] - mref[1];
  const double d2 = (double)e.c[2] - mref[2];
  const double h0 = e.h0;
  const double* h1 = e.h1;
  const double* h2 = e.h2;
  const double d[3] = {d0, d1, d2};
  A[0] += r * h0;
  A[1] += r * (h1[0] + h0 * d0);
  A[2] += r * (h1[1] + h0 * d1);
  A[3] += r * (h1[2] + h0 * d2);
  const int ia[6] = {0, 0, 0, 1, 1, 2}, ib[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int e = 0; e < 6; e++)
    A[4 + e] += r * (h2[e] + h1[ia[e]] * d[ib[e]] + d[ia[e]] * h1[ib[e]] + h0 * d[ia[e]] * d[ib[e]]);
}

__device__ __forceinline__ void mstep_add(const DevPlan& P, const FrameDesc& D, int p, const double* mref,
                                          double* A) {
  mentry_add(mentry_load(P, D, p), mref, A);
}

// Block-cooperative ordered scan for Gaussians whose bucket overflowed: visit every
// position p = j*S + s of the frame in increasing order, keep those whose candidate is k
// and whose rnk exceeds `thr`; `visit(p)` is called by thread 0 in increasing p order.
template <typename F>
__device__ void ordered_scan(const DevPlan& P, const FrameDesc& D, int it, int k, double thr, int* sh_list,
                             int* sh_cnt, F visit) {
  const int32_t* cand = cand_buf(P, it);
  const float* rnk = rnk_buf(P, it);
  const int64_t total = (int64_t)kJ * D.n_sv;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int64_t base = 0; base < total; base += blockDim.x) {
    const int64_t p = base + threadIdx.x;
    bool pred = false;
    if (p < total) {
      const int j = (int)(p / D.n_sv), sl = (int)(p - (int64_t)j * D.n_sv);
      const int64_t idx = (int64_t)(D.sv_base + sl) * kJ + j;
      pred = (cand[idx] == k) && ((double)rnk[idx] > thr);
    }
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (lane == 0) sh_cnt[w] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
      int run = 0;
      for (int i = 0; i < (int)(blockDim.x >> 5); i++) {
        const int c = sh_cnt[i];
        sh_cnt[i] = run;
        run += c;
      }
      sh_cnt[blockDim.x >> 5] = run;
    }
    __syncthreads();
    if (pred) sh_list[sh_cnt[w] + __popc(m & ((1u << lane) - 1u))] = (int)p;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int i = 0; i < sh_cnt[blockDim.x >> 5]; i++) visit(sh_list[i]);
    __syncthreads();
  }
}

// ===========================================================================
// mstep_update: thread per Gaussian.  Sorted bucket -> FP64 sufficient statistics ->
// Dirichlet / Normal-Wishart update (GMEMupdateCUDA.cu:1601-1677) -> regularisation
// (:1693-1809).  Writes the chunk's alpha sum for the kill step.
// ===========================================================================
__global__ void __launch_bounds__(kMChunk) k_mstep_update(DevPlan P) {
  // two blocks per Gaussian chunk (twice the SMs busy): block b covers half b%2 of chunk b/2
  const int c = blockIdx.x >> 1, half = blockIdx.x & 1;
  if (c >= P.info->n_gchunks) return;
  const GChunk ch = P.gchunks[c];
  __shared__ int s_ovf[kMChunk];
  __shared__ int s_novf;
  __shared__ double s_ovf_acc[kMChunk][10];
  __shared__ int s_list[kMChunk];
  __shared__ int s_cnt[kMChunk / 32 + 1];
  __shared__ double shd[kMChunk / 32];
  __shared__ int s_bk[kBucketCap][kMChunk];  // each thread's bucket, one column per thread
  if (threadIdx.x == 0) s_novf = 0;
  const int k = ch.g_begin + half * kMChunk + threadIdx.x;
  const bool valid = k < ch.g_end;
  double A[10];
#pragma unroll
  for (int i = 0; i < 10; i++) A[i] = 0.0;
  double mref[3] = {0, 0, 0};
  bool ovf = false;
  // the Gaussian's own inputs of the update, loaded ahead of the frame's state and of the bucket
  // work so that they arrive beside them: the prior (m_o also re-centres the pairs), its fixed
  // flag, this iteration's E[ln|Lambda|] (the kill step's NaN test), the centre the kNN saw, and
  // the bucket's count and first eight entries (entries past the count are stale and unused; the
  // bucket rows are 128-byte aligned)
  const int cur = P.iter & 1, nxt = cur ^ 1;
  double bo = 0.0, nuo = 0.0, alo = 0.0, Wo[6] = {0, 0, 0, 0, 0, 0}, eld_cur = 0.0, alpha_old = 0.0;
  bool fixed_k = false;
  float4 kp_old = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  int4 b0 = make_int4(0, 0, 0, 0), b1 = b0;
  int n = 0;
  const int* bk = P.bucket + (int64_t)(valid ? k : 0) * kBucketCap;
  if (valid) {
    n = P.bcnt[k];
    b0 = *reinterpret_cast<const int4*>(bk), b1 = *reinterpret_cast<const int4*>(bk + 4);
    for (int d = 0; d < 3; d++) mref[d] = gcomp(P, G_MO0 + d, k);
    bo = gcomp(P, G_BETAO, k);
    nuo = gcomp(P, G_NUO, k);
    alo = gcomp(P, G_ALPHAO, k);
    for (int e = 0; e < 6; e++) Wo[e] = gcomp(P, G_WO0 + e, k);
    eld_cur = gcomp(P, G_ELD0 + cur, k);
    alpha_old = gcomp(P, G_ALPHA, k);
    fixed_k = P.fixed[k] != 0;
    kp_old = P.kpos[k];
  }
  const FrameDesc D = load_desc(P, ch.frame);
  const int ncell = P.state[ch.frame].n_cells;
  if (P.state[ch.frame].done) return;
  __syncthreads();
  {
    // the grid of this frame was read by this iteration's kNN and is refilled by the kill
    // step: its 2*n_gchunks M-step blocks clear it
    const int nb = 2 * D.n_gchunks, rank = 2 * (c - D.gchunk_base) + half;
    for (int i = rank * kMChunk + threadIdx.x; i < ncell; i += nb * kMChunk) P.cell_cnt[D.cell_base + i] = 0;
  }
  if (valid) {
    P.bcnt[k] = 0;
    const int t = threadIdx.x;
    if (n > kBucketCap) {
      ovf = true;
      const int o = atomicAdd(&s_novf, 1);
      s_ovf[o] = threadIdx.x;
      atomicOr(&P.state[ch.frame].flags, F_BUCKET_OVERFLOW);
    } else if (n <= 8) {
      // up to eight positions (distinct, non-negative): sorted in registers by a 19-comparator
      // network, the unused slots padded with INT_MAX, then into shared memory
      int v[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < 8; i++)
        if (i >= n) v[i] = INT_MAX;
      constexpr int kNet[19][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {0, 2}, {1, 3}, {4, 6}, {5, 7}, {1, 2}, {5, 6},
                                   {0, 4}, {3, 7}, {1, 5}, {2, 6}, {1, 4}, {3, 6}, {2, 4}, {3, 5}, {3, 4}};
#pragma unroll
      for (int c2 = 0; c2 < 19; c2++) {
        const int lo = min(v[kNet[c2][0]], v[kNet[c2][1]]), hi = max(v[kNet[c2][0]], v[kNet[c2][1]]);
        v[kNet[c2][0]] = lo;
        v[kNet[c2][1]] = hi;
      }
#pragma unroll
      for (int i = 0; i < 8; i++)
        if (i < n) s_bk[i][t] = v[i];
    } else {
      // this Gaussian's bucket into shared memory, sorted there by position
#pragma unroll 4
      for (int i = 0; i < n; i++) s_bk[i][t] = bk[i];
      for (int i = 1; i < n; i++) {
        const int v = s_bk[i][t];
        int q = i;
        while (q > 0 && s_bk[q - 1][t] > v) {
          s_bk[q][t] = s_bk[q - 1][t];
          q--;
        }
        s_bk[q][t] = v;
      }
    }
    if (!ovf) {
      // in that order, two pairs' inputs in flight at a time
      int i = 0;
      for (; i + 1 < n; i += 2) {
        const MEntry e0 = mentry_load(P, D, s_bk[i][t]);
        const MEntry e1 = mentry_load(P, D, s_bk[i + 1][t]);
        mentry_add(e0, mref, A);
        mentry_add(e1, mref, A);
      }
      if (i < n) mstep_add(P, D, s_bk[i][t], mref, A);
    }
  }
  __syncthreads();
  const int novf = s_novf;
  for (int o = 0; o < novf; o++) {
    const int tk = s_ovf[o];
    const int kk = ch.g_begin + half * kMChunk + tk;
    double mr[3] = {gcomp(P, G_MO0, kk), gcomp(P, G_MO1, kk), gcomp(P, G_MO2, kk)};
    double acc[10];
    for (int i = 0; i < 10; i++) acc[i] = 0.0;
    ordered_scan(P, D, P.iter, kk, 1e-3, s_list, s_cnt, [&](int p) { mstep_add(P, D, p, mr, acc); });
    if (threadIdx.x == 0)
      for (int i = 0; i < 10; i++) s_ovf_acc[tk][i] = acc[i];
    __syncthreads();
  }
  if (ovf)
    for (int i = 0; i < 10; i++) A[i] = s_ovf_acc[threadIdx.x][i];
  double alpha = 0.0, move = 0.0;
  // what the kill step tests: this Gaussian's alpha if it is live and not fixed, and whether
  // its W or this iteration's E[ln|Lambda|] holds a NaN
  double amin = kInf;
  bool nanw = false;
  if (valid) {
    const bool alive = !is_dead_prior(mref[0]) && !fixed_k;
    nanw = isnan(eld_cur);
    if (!alive)
      for (int e = 0; e < 6; e++) nanw = nanw || isnan(gcomp(P, G_W0 + e, k));
    if (alive) {
      const double N = A[0];
      double xb[3] = {0, 0, 0}, Sk[6] = {0, 0, 0, 0, 0, 0};
      if (N > 0.0) {
        const double iN = 1.0 / N;
        for (int d = 0; d < 3; d++) xb[d] = mref[d] + A[1 + d] * iN;
        const int ia[6] = {0, 0, 0, 1, 1, 2}, ib[6] = {0, 1, 2, 1, 2, 2};
        for (int e = 0; e < 6; e++) Sk[e] = A[4 + e] - A[1 + ia[e]] * A[1 + ib[e]] * iN;
      }
      const double beta = bo + N;
      const double ib_ = 1.0 / beta;
      const double nu = nuo + N;
      const double alpha_n = fmax(alo + N, 0.0);
      gcomp(P, G_BETA, k) = beta;
      gcomp(P, G_NU, k) = nu;
      gcomp(P, G_ALPHA, k) = alpha_n;
      const double* mo = mref;
      double mn[3];
      for (int d = 0; d < 3; d++) {
        mn[d] = (bo * mo[d] + N * xb[d]) * ib_;
        gcomp(P, G_M0 + d, k) = mn[d];
      }
      if (Wo[5] < 1e-8) {
        Wo[5] = 0.5 * (Wo[0] + Wo[3]);
        gcomp(P, G_WO5, k) = Wo[5];
      }
      double Winv[6];
      inv3(Wo, Winv);
      const double dx[3] = {xb[0] - mo[0], xb[1] - mo[1], xb[2] - mo[2]};
      const double fct = N * (bo * ib_);
      const int ia[6] = {0, 0, 0, 1, 1, 2}, ib[6] = {0, 1, 2, 1, 2, 2};
      for (int e = 0; e < 6; e++) Winv[e] += Sk[e] + fct * dx[ia[e]] * dx[ib[e]];
      double W[6];
      inv3(Winv, W);
      RegConst rc;
      for (int d = 0; d < 3; d++) rc.scale[d] = D.reg_scale[d];
      rc.w4dof = D.w4dof;
      rc.lambda_min = D.lambda_min;
      rc.lambda_max = D.lambda_max;
      rc.max_exc = D.max_exc;
      rc.inv_s2 = D.reg_inv_s2;
      regularize_W(W, nu, rc);
      for (int e = 0; e < 6; e++) gcomp(P, G_W0 + e, k) = W[e];
      for (int e = 0; e < 6; e++) nanw = nanw || isnan(W[e]);
      amin = alpha_n;
      alpha = alpha_n;
      // the next iteration's records, as if the Gaussian survives the kill step (which
      // rewrites them for the Gaussians it kills)
      move = write_records(P, D, k, nxt, false, W, nu, alpha_n, beta, mn, true, kp_old);
    } else {
      // fixed or dead: unchanged parameters, unchanged records; psi and E[ln|Lambda|] go
      // on to the next iteration's slot
      gcomp(P, G_PSIA0 + nxt, k) = gcomp(P, G_PSIA0 + cur, k);
      gcomp(P, G_ELD0 + nxt, k) = eld_cur;
      alpha = alpha_old;
    }
  }
  const double a = block_sum_n<kMChunk>(alpha, shd);
  if (threadIdx.x == 0) P.alpha_part_e[blockIdx.x] = a;
  {
    __shared__ double s_amin[kMChunk / 32];
    __shared__ int s_nan[kMChunk / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amin = fmin(amin, __shfl_xor_sync(0xffffffffu, amin, o));
    const int wn = __any_sync(0xffffffffu, nanw) ? 1 : 0;
    if ((threadIdx.x & 31) == 0) {
      s_amin[threadIdx.x >> 5] = amin;
      s_nan[threadIdx.x >> 5] = wn;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double m = kInf;
      int nn = 0;
      for (int i = 0; i < kMChunk / 32; i++) {
        m = fmin(m, s_amin[i]);
        nn |= s_nan[i];
      }
      P.alpha_min_e[blockIdx.x] = m;
      P.nan_e[blockIdx.x] = nn;
    }
  }
  // the block's largest move of a kNN centre, rounded up to a float (non-negative floats
  // order as their bits)
  float mv = __double2float_ru(move);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mv = fmaxf(mv, __shfl_xor_sync(0xffffffffu, mv, o));
  if ((threadIdx.x & 31) == 0 && mv > 0.0f) atomicMax(&P.state[ch.frame].disp_max, __float_as_uint(mv));
}

// The log-likelihood pass's record of a Gaussian (see GaussLL): Cholesky's factor of
// nu W log2(e) / 2 from reciprocal square roots in FP64, rounded once.  Zero where the weight is
// not finite (the candidate then counts for nothing, or rules its supervoxels out); r[0] NaN
// where there is no factor.
__device__ __forceinline__ GaussLL stream_record(const double* W, double nu, double ln_w, double m0, double m1,
                                                 double m2) {
  const double h = 0.5 * 1.4426950408889634 * nu;
  const double i0 = rsqrt(h * W[0]);
  const double r00 = h * W[0] * i0, r01 = h * W[1] * i0, r02 = h * W[2] * i0;
  const double p11 = h * W[3] - r01 * r01, i1 = rsqrt(p11);
  const double r11 = p11 * i1, r12 = (h * W[4] - r01 * r02) * i1;
  const double p22 = h * W[5] - r02 * r02 - r12 * r12;
  const double r22 = p22 * rsqrt(p22);
  GaussLL g;
  g.b = ln_w * 1.4426950408889634;
  g.m[0] = m0, g.m[1] = m1, g.m[2] = m2;
  const double r[6] = {r00, r01, r02, r11, r12, r22};
  bool ok = true;
  for (int e = 0; e < 6; e++) ok = ok && isfinite(r[e]);
  for (int e = 0; e < 6; e++) g.r[e] = !isfinite(ln_w) ? 0.0f : ok ? __double2float_rn(r[e]) : __uint_as_float(0x7fffffffu);
  g.pad[0] = g.pad[1] = 0.0f;
  return g;
}

// ===========================================================================
// kill_prep: dead-Gaussian rule (GMEMcheckDeadCellsKernel, GMEMupdateCUDA.cu:1813-1843)
// with the post-update alpha total, then the preparation of the next iteration.
// ===========================================================================
__global__ void __launch_bounds__(kGChunk) k_kill_prep(DevPlan P) {
  const int c = blockIdx.x;
  if (c >= P.info->n_gchunks) return;
  const GChunk ch = P.gchunks[c];
  const FrameState& S = P.state[ch.frame];
  if (S.done) return;
  const FrameDesc D = load_desc(P, ch.frame);
  __shared__ double s_total;
  __shared__ double shd[kGChunk / 32];
  __shared__ int shi[kGChunk / 32];
  const int cur = P.iter & 1, nxt = cur ^ 1;
  const int k = ch.g_begin + threadIdx.x;
  const bool valid = k < ch.g_end;
  // this Gaussian's inputs are on their way while warp 0 sums the frame's alpha partials
  bool nanw = false, was_dead = true, fixed = true;
  double a = 0.0;
  float4 centre = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  GaussLL rec;
  if (valid) {
    centre = P.kpos[k];
    nanw = isnan(gcomp(P, G_ELD0 + cur, k));
    double Wk[6];
    for (int e = 0; e < 6; e++) Wk[e] = gcomp(P, G_W0 + e, k);
    a = gcomp(P, G_ALPHA, k);
    was_dead = is_dead_prior(gcomp(P, G_MO0, k));
    fixed = P.fixed[k] != 0;
    for (int e = 0; e < 6; e++) nanw = nanw || isnan(Wk[e]);
    rec = stream_record(Wk, gcomp(P, G_NU, k), P.llc[(int64_t)k * 10 + 6], gcomp(P, G_M0, k), gcomp(P, G_M1, k),
                        gcomp(P, G_M2, k));
  }
  __shared__ int s_fast;
  int cell = -1;
  {
    // the frame's M-step block partials, spread over the whole block so that their loads are
    // in flight together: the alpha total (a fixed order: each thread's partials in order, a
    // butterfly per warp, the warps in order -- the same bits in every block of the frame),
    // the smallest live alpha and the NaN flags.  No Gaussian of the frame can die this
    // iteration when none has a NaN and the smallest live alpha passes the rule.
    __shared__ double s_wt[kGChunk / 32], s_wm[kGChunk / 32];
    __shared__ int s_wn[kGChunk / 32];
    const int nb = 2 * D.n_gchunks, base = 2 * D.gchunk_base;
    double tp = 0.0, mp = kInf;
    int np = 0;
    for (int i = threadIdx.x; i < nb; i += kGChunk) {
      tp += P.alpha_part_e[base + i];
      mp = fmin(mp, P.alpha_min_e[base + i]);
      np |= P.nan_e[base + i];
    }
    tp = warp_sum(tp);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mp = fmin(mp, __shfl_xor_sync(0xffffffffu, mp, o));
    np = __any_sync(0xffffffffu, np != 0);
    // the grid cell of a live centre, from the frame's grid geometry, ahead of the barrier
    if (valid && !was_dead) cell = ref_cell_of(S, D, centre.x, centre.y, centre.z);
    if ((threadIdx.x & 31) == 0) {
      s_wt[threadIdx.x >> 5] = tp;
      s_wm[threadIdx.x >> 5] = mp;
      s_wn[threadIdx.x >> 5] = np;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double tot = 0.0, amin = kInf;
      int nn = 0;
#pragma unroll
      for (int w = 0; w < kGChunk / 32; w++) {
        tot += s_wt[w];
        amin = fmin(amin, s_wm[w]);
        nn |= s_wn[w];
      }
      s_total = tot;
      s_fast = !nn && !(amin / tot < TGMM_MIN_PI_FOR_DEAD);
    }
  }
  __syncthreads();
  const double total = s_total;
  if (s_fast) {
    // nothing dies: the live Gaussians go into the grid, and the frame's first chunk writes
    // its totals (the post-kill total is the M-step's; the dead count stays)
    if (valid) P.gll[k] = rec;
    if (valid && !was_dead) grid_insert_at(P, D, cell, k, centre);
    if (c == D.gchunk_base && threadIdx.x == 0) {
      FrameState* Sw = &P.state[ch.frame];
      Sw->total_alpha = total;
      Sw->ln_alpha = log(total);
      Sw->psi_total[nxt] = digamma(total);
      Sw->blk_done = 0;
      Sw->disp_cum += (double)__uint_as_float(Sw->disp_max);
      Sw->disp_max = 0u;
    }
    return;
  }
  double alpha = 0.0;
  int dead = 0;
  if (valid) {
    if (nanw || (a / total < TGMM_MIN_PI_FOR_DEAD && !was_dead && !fixed)) {
      gcomp(P, G_ALPHA, k) = 0.0;
      const double mdead[3] = {-1e32, -1e32, -1e32};
      for (int d = 0; d < 3; d++) {
        gcomp(P, G_MO0 + d, k) = -1e32;
        gcomp(P, G_M0 + d, k) = -1e32;
      }
      const double I6[6] = {1, 0, 0, 1, 0, 1};
      for (int e = 0; e < 6; e++) gcomp(P, G_W0 + e, k) = I6[e];
      write_records(P, D, k, nxt, true, I6, gcomp(P, G_NU, k), 0.0, gcomp(P, G_BETA, k), mdead, false);
      rec = stream_record(I6, gcomp(P, G_NU, k), -kInf, mdead[0], mdead[1], mdead[2]);
      dead = 1;
    } else {
      alpha = a;
      dead = was_dead ? 1 : 0;
      if (!was_dead) grid_insert_at(P, D, cell, k, centre);
    }
    P.gll[k] = rec;
  }
  chunk_partials(alpha, dead, shd, shi, P.alpha_part_f, P.dead_part, c);
  chunk_done(P, ch.frame, D.n_gchunks, nxt);
}

// ===========================================================================
// ll_pass: the per-iteration voxel stream.  Warp per supervoxel:
//   ll_v = ln sum_j (alpha_j/A) sqrt(det(W_j) nu_j^3) (2 pi)^-3/2 exp(-nu_j d'W_j d / 2)
// over the supervoxel's five candidates (GMEMcomputeLikelihoodKernelWithSupervoxels,
// GMEMupdateCUDA.cu:1913-1978), I_v * ll_v summed when the density is positive.  Two
// sums: every voxel (true) and the reference's per-thread overwrite for supervoxels
// above 1024 voxels (as reference).
// k_ll_pass holds the FP64 mode (every component in FP64 with the reference's formula) and, on
// the same tile ring, the once-per-call moment pass; the FP32 mode is k_ll_stream below.
// Voxel tiles reach shared memory through TMA bulk copies (cp.async.bulk, one per
// component and tile, issued by one lane) that complete on a per-slot mbarrier:
// kLLStages tiles of kLLTile voxels are in flight per warp while it computes.  A copy
// covers the 16-byte aligned span around its tile and the lanes index it from the
// component's offset.
// Per-supervoxel results are added into per-frame 64-bit integer accumulators (integer
// part and 2^-40 fraction), so the frame total does not depend on the order in which
// warps finish; the warp that finishes a frame's last supervoxel runs the reference's
// convergence test for that frame.
// ===========================================================================
constexpr float kL2E = 1.4426950408889634f;  // log2(e)

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// FP64 verification mode: the reference's formula, every component in FP64.
struct LLShared64 {
  double u[kJ][3];
  double A[kJ][6];  // nu * W
  double w[kJ];     // c_j * alpha_j / A
};

__device__ __forceinline__ double voxel_ll_fp64(const LLShared64& C, float x0, float x1, float x2, float c0, float c1,
                                                float c2, bool& ok) {
  const double e0 = (double)x0 - (double)c0, e1 = (double)x1 - (double)c1, e2 = (double)x2 - (double)c2;
  double dens = 0.0;
#pragma unroll 1
  for (int j = 0; j < kJ; j++) {
    const double d0 = e0 - C.u[j][0], d1 = e1 - C.u[j][1], d2 = e2 - C.u[j][2];
    const double* A = C.A[j];
    const double q = A[0] * d0 * d0 + A[3] * d1 * d1 + A[5] * d2 * d2 + 2.0 * A[1] * d0 * d1 +
                     2.0 * A[2] * d0 * d2 + 2.0 * A[4] * d1 * d2;
    dens += C.w[j] * exp(-0.5 * q);
  }
  ok = dens > 0.0;
  return ok ? log(dens) : 0.0;
}

// --- TMA bulk staging --------------------------------------------------------
#ifndef TGMM_LL_STAGES
#define TGMM_LL_STAGES 3
#endif
#ifndef TGMM_LL_BLOCKS
#define TGMM_LL_BLOCKS 2
#endif
#ifndef TGMM_LL_WARPS
#define TGMM_LL_WARPS 8
#endif
constexpr int kFp64Parts = 4;                 // parts of a supervoxel in the FP64 log-likelihood
constexpr int kLLWarps = TGMM_LL_WARPS;       // warps per block of the voxel pass
constexpr int kLLTile = kVoxTile;             // voxels per tile (kVoxTile / 32 per lane)
constexpr int kLLStages = TGMM_LL_STAGES;     // tile slots per warp
constexpr int kLLBlocks = TGMM_LL_BLOCKS;     // resident blocks per SM the pass is compiled for
constexpr int kLLSpan = kLLTile + 4;          // floats per component in a slot (16-byte slack)
constexpr int kLLSlotFloats = 4 * kLLSpan;    // x, y, z, I
constexpr unsigned long long kLLWaitNs = 1000000000ull;  // default wait limit of a slot, and the drain's bound

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool mbar_test_wait(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0;
}
// Waits for the phase with the given parity; false after limit_ns without it.  try_wait
// suspends the thread for a while until the phase completes, so at the default limit the
// clock is read only between its returns; a limit below 1 ms polls with the non-blocking
// test_wait, so that the limit is kept to the clock's resolution.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, unsigned long long limit_ns) {
  if (limit_ns < 1000000ull) {
    if (mbar_test_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    while (!mbar_test_wait(bar, parity))
      if (global_ns() - t0 > limit_ns) return false;
    return true;
  }
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (!mbar_try_wait(bar, parity))
    if (global_ns() - t0 > limit_ns) return false;
  return true;
}
// Global -> shared bulk copy (non-multicast) completing on the mbarrier at `bar`.
__device__ __forceinline__ void bulk_g2s(unsigned dst, unsigned long long src, unsigned bytes, unsigned bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}
// Small global -> shared copies (cp.async) for the look-ahead records.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Tile t of a supervoxel (SvRec): one bulk copy per component of the 16-byte chunks
// holding its voxels.  Every chunk copied holds a voxel of the tile, so no byte outside
// its array's pages is read.
__device__ __forceinline__ void ll_issue(const SvRec& R, int t, float* slot, unsigned bar) {
  unsigned n[4], total = 0;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    n[c] = t == 0 ? R.n0[c] : (R.nf[c] & 0xffffu);
    total += n[c];
  }
  mbar_expect_tx(bar, total);
#pragma unroll
  for (int c = 0; c < 4; c++)
    bulk_g2s(smem_addr(slot + c * kLLSpan),
             t == 0 ? R.lo0[c] : R.lo1[c] + (unsigned long long)(4 * kLLTile) * (unsigned)(t - 1), n[c], bar);
}

// Look-ahead records, fetched with cp.async ahead of use: a supervoxel's stream record and
// candidate ids (stage A, two supervoxels ahead) and its candidates' constants (10
// doubles each) with its frame's ln(sum alpha) and done flag (stage B, one ahead).
struct LLRec {
  SvRec rec;  // the SoA spans of the input arrays
  SvLL ll;    // the moment pass: the place in the centred voxel stream
  int32_t cand[8];
};
struct LLConst {
  double llc[kJ][10];
  double ln_alpha;
  int32_t done, pad;
};
static_assert(sizeof(LLRec) % 16 == 0 && sizeof(LLConst) % 16 == 0, "look-ahead records stay 16-byte aligned");

// Per-warp shared region: slots, one mbarrier per slot, three stage-A and two stage-B records.
constexpr int kLLBarOff = kLLStages * kLLSlotFloats * 4;
constexpr int kLLRecOff = (kLLBarOff + kLLStages * 8 + 15) / 16 * 16;
constexpr int kLLConstOff = kLLRecOff + 3 * (int)sizeof(LLRec);
constexpr int kLLWarpBytes = (kLLConstOff + 2 * (int)sizeof(LLConst) + 15) / 16 * 16;
constexpr size_t kLLSmemBytes = (size_t)kLLWarpBytes * kLLWarps;
static_assert((kLLSlotFloats * 4) % 16 == 0 && kLLRecOff % 16 == 0 && kLLConstOff % 16 == 0,
              "slots and records stay 16-byte aligned");
// the moment pass keeps kLLBlocks blocks on an SM (228 KB of shared memory, 1 KB reserved per
// block, its one static LLShared64); the FP64 form sizes its own grid
static_assert(kLLBlocks * (kLLSmemBytes + 1024 + sizeof(LLShared64)) <= 233472, "the voxel pass's blocks fit an SM");

// Stage A: the records (SoA spans: kRec; centred-stream place: kLL) and candidate ids
// (kCand) of supervoxel s, one lane per 16-byte chunk or id.
template <bool kRec, bool kLL, bool kCand>
__device__ __forceinline__ void ll_fetch_a(const DevPlan& P, LLRec& X, int s) {
  const int lane = threadIdx.x & 31;
  constexpr int kRecChunks = kRec ? (int)sizeof(SvRec) / 16 : 0;
  constexpr int kLLChunks = kLL ? (int)sizeof(SvLL) / 16 : 0;
  static_assert(kRecChunks + kLLChunks + kJ <= 32, "one lane per chunk");
  if (lane < kRecChunks) {
    cp_async16(reinterpret_cast<char*>(&X.rec) + 16 * lane, reinterpret_cast<const char*>(P.sv_rec + s) + 16 * lane);
  } else if (lane < kRecChunks + kLLChunks) {
    const int c = lane - kRecChunks;
    cp_async16(reinterpret_cast<char*>(&X.ll) + 16 * c, reinterpret_cast<const char*>(P.sv_ll + s) + 16 * c);
  } else if (kCand && lane < kRecChunks + kLLChunks + kJ) {
    const int j = lane - kRecChunks - kLLChunks;
    cp_async4(&X.cand[j], cand_buf(P, P.iter) + (int64_t)s * kJ + j);
  }
}
// Stage B (after A landed): the candidates' constants and the frame scalars.
__device__ __forceinline__ void ll_fetch_b(const DevPlan& P, const LLRec& A, int frame, LLConst& X) {
  const int lane = threadIdx.x & 31;
  if (lane < 5 * kJ) {
    const int j = lane / 5, c = lane % 5;
    cp_async16(&X.llc[j][2 * c], P.llc + (int64_t)A.cand[j] * 10 + 2 * c);
  } else if (lane == 5 * kJ) {
    cp_async8(&X.ln_alpha, &P.state[frame].ln_alpha);
  } else if (lane == 5 * kJ + 1) {
    cp_async4(&X.done, &P.state[frame].done);
  }
}

// Evaluation of one voxel in FP64.
struct VoxelEval64 {
  const LLShared64& C;
  __device__ __forceinline__ double operator()(float x, float y, float z, float c0, float c1, float c2) const {
    bool ok;
    const double l = voxel_ll_fp64(C, x, y, z, c0, c1, c2, ok);
    return ok ? l : -kInf;
  }
  __device__ __forceinline__ static bool ok(double l) { return l > -kInf; }
};

// One staged tile: lane voxels o = u*32 + lane < rem, sht[c] the offset of component c in the
// slot.  allok turns false when a present voxel has a zero density.
// Rolled (as are the candidates in voxel_ll_fp64): unrolled by eight and five the kernel missed
// the instruction cache six times as often as it issued.
__device__ __forceinline__ void ll_tile(const VoxelEval64& eval, const float* __restrict__ slot, const int* sht, int rem,
                                        float c0, float c1, float c2, double& tsum, bool& allok) {
  const int lane = threadIdx.x & 31;
  const float* bx = slot + sht[0];
  const float* by = slot + kLLSpan + sht[1];
  const float* bz = slot + 2 * kLLSpan + sht[2];
  const float* bi = slot + 3 * kLLSpan + sht[3];
#pragma unroll 2
  for (int o = lane; o < rem; o += 32) {
    const double l = eval(bx[o], by[o], bz[o], c0, c1, c2);
    const bool ok = VoxelEval64::ok(l);
    allok = allok && ok;
    tsum += ok ? (double)bi[o] * l : 0.0;
  }
}

// A kept voxel (one of the last 1024 of a supervoxel above 1024 voxels) with a zero
// density: the reference thread of its stride still holds the last voxel of the stride
// with a positive density (GMEMupdateCUDA.cu:1961-1962).  Rare; reads global memory.
__device__ __noinline__ double ll_walk_back(const VoxelEval64& eval, const SvRec& R, int i, float c0, float c1, float c2) {
  const float* v[4];
#pragma unroll
  for (int c = 0; c < 4; c++) v[c] = reinterpret_cast<const float*>(R.lo0[c]) + ((R.nf[c] >> 16) & 3);
  for (int i2 = i - 1024; i2 >= 0; i2 -= 1024) {
    const double l2 = eval(v[0][i2], v[1][i2], v[2][i2], c0, c1, c2);
    if (VoxelEval64::ok(l2)) return (double)v[3][i2] * (double)l2;
  }
  return 0.0;
}

// The kept tiles (bit t - (nt - kKeptTiles) of `mask`) that hold voxels of zero density, after the
// supervoxel's tiles: their voxels are read again from global memory and each one of zero
// density adds the walk-back value.  Rare.
__device__ __noinline__ double ll_fixup(const VoxelEval64& eval, const SvRec& R, unsigned mask, float c0, float c1,
                                           float c2) {
  const int lane = threadIdx.x & 31;
  const float* v[4];
#pragma unroll
  for (int c = 0; c < 4; c++) v[c] = reinterpret_cast<const float*>(R.lo0[c]) + ((R.nf[c] >> 16) & 3);
  double add = 0.0;
  for (int k = 0; k < kKeptTiles; k++) {
    if (!(mask & (1u << k))) continue;
    const int t = R.ntiles - kKeptTiles + k;
    const int start = t == 0 ? 0 : R.r0 + (t - 1) * kLLTile;
    const int rem = t == 0 ? R.r0 : kLLTile;
    for (int o = lane; o < rem; o += 32) {
      const int i = start + o;
      const double l = eval(v[0][i], v[1][i], v[2][i], c0, c1, c2);
      if (!VoxelEval64::ok(l)) add += ll_walk_back(eval, R, i, c0, c1, c2);
    }
  }
  return add;
}

// The moment pass's tile t (landed in `slot`): the 19 sums e, ee', I, Ie, Iee' (e = x - c in
// FP32, FP64 accumulation) of the lane's voxels o = u*32 + lane, each voxel also written to
// the centred voxel stream (out: the tile's first voxel there) as (e0, e1, e2, I); nan_seen
// turns true on a NaN coordinate or intensity.
template <bool kFull>
__device__ __forceinline__ void mom_tile(const float* __restrict__ slot, const int* sht, int rem, float c0, float c1,
                                         float c2, double* m, float* h, bool& nan_seen, float4* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const float* bx = slot + sht[0] + lane;
  const float* by = slot + kLLSpan + sht[1] + lane;
  const float* bz = slot + 2 * kLLSpan + sht[2] + lane;
  const float* bi = slot + 3 * kLLSpan + sht[3] + lane;
#pragma unroll
  for (int u = 0; u < kLLTile / 32; u++) {
    if (!kFull && u * 32 >= rem) break;
    if (!kFull && u * 32 + lane >= rem) continue;
    const float x = bx[32 * u], y = by[32 * u], z = bz[32 * u], I = bi[32 * u];
    nan_seen |= isnan(x) || isnan(y) || isnan(z) || isnan(I);
    const float e0f = x - c0, e1f = y - c1, e2f = z - c2;
    out[32 * u + lane] = make_float4(e0f, e1f, e2f, I);
    h[0] = fmaxf(h[0], fabsf(e0f));
    h[1] = fmaxf(h[1], fabsf(e1f));
    h[2] = fmaxf(h[2], fabsf(e2f));
    const double e0 = (double)e0f, e1 = (double)e1f, e2 = (double)e2f;
    const double wI = (double)I;
    m[M_E0] += e0;
    m[M_E1] += e1;
    m[M_E2] += e2;
    m[M_EE00] = fma(e0, e0, m[M_EE00]);
    m[M_EE01] = fma(e0, e1, m[M_EE01]);
    m[M_EE02] = fma(e0, e2, m[M_EE02]);
    m[M_EE11] = fma(e1, e1, m[M_EE11]);
    m[M_EE12] = fma(e1, e2, m[M_EE12]);
    m[M_EE22] = fma(e2, e2, m[M_EE22]);
    m[M_I] += wI;
    const double i0 = wI * e0, i1 = wI * e1, i2 = wI * e2;
    m[M_IE0] += i0;
    m[M_IE1] += i1;
    m[M_IE2] += i2;
    m[M_IEE00] = fma(i0, e0, m[M_IEE00]);
    m[M_IEE01] = fma(i0, e1, m[M_IEE01]);
    m[M_IEE02] = fma(i0, e2, m[M_IEE02]);
    m[M_IEE11] = fma(i1, e1, m[M_IEE11]);
    m[M_IEE12] = fma(i1, e2, m[M_IEE12]);
    m[M_IEE22] = fma(i2, e2, m[M_IEE22]);
  }
}

__device__ __forceinline__ void mom_consume(const float* slot, const int* pk, int t, int r0, float c0, float c1,
                                            float c2, double* m, float* h, bool& nan_seen, float4* sv_out) {
  const int sft = t == 0 ? 0 : 4;
  const int sht[4] = {(pk[0] >> sft) & 3, (pk[1] >> sft) & 3, (pk[2] >> sft) & 3, (pk[3] >> sft) & 3};
  const int rem = t == 0 ? r0 : kLLTile;
  float4* out = sv_out + (t == 0 ? 0 : r0 + kLLTile * (t - 1));
  if (rem == kLLTile)
    mom_tile<true>(slot, sht, rem, c0, c1, c2, m, h, nan_seen, out);
  else
    mom_tile<false>(slot, sht, rem, c0, c1, c2, m, h, nan_seen, out);
}

// Tile t (landed in `slot`) of the current supervoxel: its sum goes to lt, and to lr when
// the tile is one of the last kKeptTiles (the reference's kept window of 1024 voxels).  A kept
// tile of a supervoxel above 1024 voxels with a voxel of zero density is marked in fix.
__device__ __forceinline__ void ll_consume(const VoxelEval64& eval, const float* slot, const int* pk, int t, int nt, int nv,
                                           int r0, float c0, float c1, float c2, double& lt, double& lr,
                                           unsigned& fix) {
  const int sft = t == 0 ? 0 : 4;
  const int sht[4] = {(pk[0] >> sft) & 3, (pk[1] >> sft) & 3, (pk[2] >> sft) & 3, (pk[3] >> sft) & 3};
  const int rem = t == 0 ? r0 : kLLTile;
  double tsum = 0.0;
  bool allok = true;
  ll_tile(eval, slot, sht, rem, c0, c1, c2, tsum, allok);
  lt += tsum;
  if (t >= nt - kKeptTiles) {
    lr += tsum;
    if (nv > 1024 && __any_sync(0xffffffffu, !allok)) fix |= 1u << (t - (nt - kKeptTiles));
  }
}

// A frame's order-free sum (see fixed_acc); its fractions come carried from each warp.
__device__ __forceinline__ double fixed_read(const long long* ip, const unsigned long long* fp) {
  long long i = *(volatile const long long*)ip;
  unsigned long long f = *(volatile const unsigned long long*)fp;
  fixed_carry(i, f);
  return (double)i + (double)f / kFracScale;
}

// The reference's convergence test after iteration t (GMEMupdateCUDA.cu:4145-4148), run
// by the warp that finished the frame's last supervoxel.
__device__ void frame_converge(const DevPlan& P, int f) {
  FrameState* S = &P.state[f];
  const FrameDesc D = load_desc(P, f);
  const double lt = fixed_read(&S->ll_int[0], &S->ll_frac[0]);
  const double lr = fixed_read(&S->ll_int[1], &S->ll_frac[1]);
  S->ll_int[0] = S->ll_int[1] = 0;
  S->ll_frac[0] = S->ll_frac[1] = 0;
  S->sv_done = 0;
  S->ll3 = S->ll2;
  S->ll2 = S->ll1;
  S->ll1 = S->ll;
  S->ll_true = lt;
  S->ll_ref = lr;
  S->ll = (D.ll_mode == TGMM_LL_TRUE) ? lt : lr;
  const int next = S->iter + 1;
  S->iter = next;
  const double ll = S->ll;
  const bool go = fabs(ll - S->ll1) / fabs(S->ll1) > D.tol && fabs(ll - S->ll2) / fabs(S->ll2) > D.tol &&
                  fabs(ll - S->ll3) / fabs(S->ll3) > D.tol;
  if (!go) S->converged = 1;
  S->done = (!go || next > D.max_iter) ? P.iter : 0;  // (see FrameState::done)
}

// Each warp streams the supervoxels it takes from the work counter through a ring of
// kLLStages tile slots; the ring runs on from one supervoxel into the next.  Tickets are
// taken two supervoxels ahead: while the warp computes its i-th supervoxel, the stream
// record and candidate ids of the (i+2)-th (stage A) and the candidates' constants of the
// (i+1)-th (stage B) are on their way, so every wait is for copies issued a supervoxel
// earlier.  A warp adds its supervoxels' sums into fixed-point registers and publishes
// them (with the count of supervoxels) when its frame changes and when it leaves; the
// warp that completes a frame's count runs the convergence test.
// kMom: the moment pass (which also writes the centred voxel stream); else the FP64
// log-likelihood, which reads the input arrays too (its terms start from the exact x - c).
template <bool kMom>
__global__ void __launch_bounds__(kLLWarps * 32, kLLBlocks) k_ll_pass(DevPlan P) {
  constexpr bool kRec = true, kLLr = kMom, kCand = !kMom, kFp64 = !kMom;
  // the FP64 log-likelihood takes a supervoxel in kParts parts (part p: tiles p, p + kParts, ...):
  // at one warp a supervoxel its time was that of the largest one (2000 supervoxels, 1.4 M voxels:
  // 106 us in one part, 81 in two, 72 in four, 73 in eight; 174 before it was rolled, see ll_tile)
  constexpr int kParts = kMom ? 1 : kFp64Parts;
  const int total = P.info->total_sv * kParts;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __shared__ LLShared64 sh64[kFp64 ? kLLWarps : 1];
  extern __shared__ __align__(128) unsigned char ll_smem[];
  unsigned char* wbase = ll_smem + (size_t)warp * kLLWarpBytes;
  float* wbuf = reinterpret_cast<float*>(wbase);
  const unsigned bar0 = smem_addr(wbase + kLLBarOff);
  LLRec* RA = reinterpret_cast<LLRec*>(wbase + kLLRecOff);
  LLConst* RB = reinterpret_cast<LLConst*>(wbase + kLLConstOff);
  if (lane == 0)
    for (int q = 0; q < kLLStages; q++) mbar_init(bar0 + 8 * q, 1);
  mbar_fence_init();
  __syncwarp();
  // lane 0: the fixed-point sums (true, as reference) of the warp's current frame run
  int acc_f = -1, acc_nsv = 0, acc_n = 0;
  long long acc_i0 = 0, acc_i1 = 0;
  unsigned long long acc_r0 = 0, acc_r1 = 0;
  auto publish = [&]() {
    if (lane == 0 && acc_n > 0) {
      FrameState* Sp = &P.state[acc_f];
      fixed_carry(acc_i0, acc_r0);
      fixed_carry(acc_i1, acc_r1);
      atomicAdd((unsigned long long*)&Sp->ll_int[0], (unsigned long long)acc_i0);
      atomicAdd((unsigned long long*)&Sp->ll_int[1], (unsigned long long)acc_i1);
      atomicAdd(&Sp->ll_frac[0], acc_r0);
      atomicAdd(&Sp->ll_frac[1], acc_r1);
      __threadfence();
      if (atomicAdd(&Sp->sv_done, acc_n) == acc_nsv - acc_n) {
        __threadfence();
        frame_converge(P, acc_f);
      }
    }
    acc_n = 0;
    acc_i0 = acc_i1 = 0;
    acc_r0 = acc_r1 = 0;
  };
  // tiles issued / consumed by this warp in this launch (slot = count mod kLLStages,
  // mbarrier phase = count / kLLStages), and tiles of the current and the next supervoxel
  // already issued; every lane keeps the same counts
  unsigned gi = 0, gc = 0;
  int ic = 0;
  FrameState* S = nullptr;
  bool failed = false;
  // tickets: the current, the next, and (lane 0) the one after
  // a ticket t is part t % kParts of the supervoxel sv_order[t / kParts] (each frame's largest
  // first), as supervoxel * kParts + part, total at the end
  auto take = [&]() {
    const int t = atomicAdd(&P.work[0], 1);
    return t < total ? P.sv_order[t / kParts] * kParts + t % kParts : total;
  };
  int tk = 0;
  if (lane == 0) tk = take();
  int sc = __shfl_sync(0xffffffffu, tk, 0);
  if (lane == 0 && sc < total) tk = take();
  int sn = sc < total ? __shfl_sync(0xffffffffu, tk, 0) : total;
  if (lane == 0 && sn < total) tk = take();
  auto frame_of = [](const LLRec& A) { return A.rec.frame; };
  if (sc < total) {
    ll_fetch_a<kRec, kLLr, kCand>(P, RA[0], sc / kParts);
    if (sn < total) ll_fetch_a<kRec, kLLr, kCand>(P, RA[1], sn / kParts);
    cp_commit();
    cp_wait_all();
    __syncwarp();
    if (!kMom) ll_fetch_b(P, RA[0], frame_of(RA[0]), RB[0]);
    cp_commit();
  }
  for (unsigned i = 0; sc < total; i++) {
    // everything fetched so far was issued at least a supervoxel ago
    cp_wait_all();
    __syncwarp();
    const LLRec& CA = RA[i % 3];
    const LLConst& CB = RB[i & 1];
    const LLRec& NA = RA[(i + 1) % 3];
    const int s2 = __shfl_sync(0xffffffffu, tk, 0);
    if (lane == 0 && s2 < total) tk = take();
    if (!kMom && sn < total) ll_fetch_b(P, NA, frame_of(NA), RB[(i + 1) & 1]);
    if (s2 < total) ll_fetch_a<kRec, kLLr, kCand>(P, RA[(i + 2) % 3], s2 / kParts);
    cp_commit();
    int in = 0;
    // this part's tiles, and the next one's, which may start early
    const int part = sc % kParts, part_n = sn % kParts;
    const int n_nt = sn < total ? (NA.rec.ntiles - part_n + kParts - 1) / kParts : 0;
    const int nv = CA.rec.nv, nt = CA.rec.ntiles;
    const int f = frame_of(CA), nsv = CA.rec.frame_nsv * kParts;
    const float c0 = CA.rec.c0, c1 = CA.rec.c1, c2 = CA.rec.c2;
    S = &P.state[f];
    int pk[4] = {0, 0, 0, 0};  // SoA slot offsets of the components: tile 0 in bits 0-1, later tiles in bits 4-5
    if constexpr (kRec) {
#pragma unroll
      for (int c = 0; c < 4; c++) pk[c] = (int)(CA.rec.nf[c] >> 16);
    }
    const int r0 = CA.rec.r0;
    // the next staged tile of the supervoxel (of ntr): the ring is refilled first, with the
    // current supervoxel's tiles and then the next one's; nullptr if the tile never arrived
    auto ring_next = [&](int ntr) -> const float* {
      __syncwarp();  // every lane is done with the slots refilled below
      while (gi < gc + kLLStages) {
        const bool mine = ic < ntr;
        if (!mine && in >= n_nt) break;
        const int tt = mine ? part + kParts * ic++ : part_n + kParts * in++;
        if (lane == 0) {
          const unsigned q = gi % kLLStages;
          ll_issue(mine ? CA.rec : NA.rec, tt, wbuf + q * kLLSlotFloats, bar0 + 8 * q);
        }
        gi++;
      }
      const unsigned q = gc % kLLStages;
      if (!__all_sync(0xffffffffu, mbar_wait(bar0 + 8 * q, (gc / kLLStages) & 1, P.stage_wait_ns))) return nullptr;
      return wbuf + q * kLLSlotFloats;
    };
    if constexpr (kMom) {
      // the moment pass: 19 sums per lane over its voxels of every tile, then per supervoxel
      double m[kNumMoments];
#pragma unroll
      for (int j = 0; j < kNumMoments; j++) m[j] = 0.0;
      float h[3] = {0.0f, 0.0f, 0.0f};  // the largest |e| along each axis
      bool nan_seen = false;
      for (int t = 0; t < nt; t++) {
        const float* slot = ring_next(nt);
        if (!slot) {
          failed = true;
          break;
        }
        mom_consume(slot, pk, t, r0, c0, c1, c2, m, h, nan_seen, P.vox4 + CA.ll.v0);
        gc++;
      }
      if (failed) break;
      if (__any_sync(0xffffffffu, nan_seen) && lane == 0) atomicOr(&S->flags, F_NAN_INPUT);
#pragma unroll
      for (int d = 0; d < 3; d++) {
        h[d] = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(h[d])));
        if (lane == d) (&P.sv_ll[sc].h0)[d] = h[d];
      }
#pragma unroll
      for (int j = 0; j < kNumMoments; j++) m[j] = warp_sum(m[j]);
#pragma unroll
      for (int j = 0; j < kNumMoments; j++)  // lane j writes moment j
        if (lane == j) P.mom[(int64_t)j * P.max_sv + sc] = m[j];
    } else {
    const bool run = CB.done == 0;
    // candidate j on lane j: u = m - c, weight b = ln(w) - ln(A), -nu W/2
    double u[3] = {0, 0, 0}, h[6] = {0, 0, 0, 0, 0, 0}, b = 0.0;
    if (lane < kJ) {
      const double* L = CB.llc[lane];
      for (int e = 0; e < 6; e++) h[e] = L[e];
      b = L[6] - CB.ln_alpha;
      u[0] = L[7] - (double)c0;
      u[1] = L[8] - (double)c1;
      u[2] = L[9] - (double)c2;
    }
    const unsigned fin = __ballot_sync(0xffffffffu, lane < kJ && isfinite(b));
    const unsigned nan_w = __ballot_sync(0xffffffffu, lane < kJ && (isnan(b) || b == (double)kInfF));
    // a NaN weight makes the reference's density NaN for every voxel (skipped); no finite
    // weight means a zero density everywhere: the tiles are consumed unread
    const bool compute = run && fin && !nan_w;
    LLShared64& Q = sh64[warp];
    if (lane < kJ) {
      for (int d = 0; d < 3; d++) Q.u[lane][d] = u[d];
      for (int e = 0; e < 6; e++) Q.A[lane][e] = (e == 0 || e == 3 || e == 5) ? -2.0 * h[e] : -h[e];
      Q.w[lane] = exp(b);
    }
    __syncwarp();
    double lt = 0.0, lr = 0.0;
    unsigned fix = 0;  // kept tiles with voxels of zero density
    // a finished frame issues no more tiles; those issued early are consumed unread
    const int ntr = run ? (nt - part + kParts - 1) / kParts : ic;
    // the supervoxel's tiles and, rarely, the kept window's zero-density voxels
    const VoxelEval64 eval{Q};
    for (int t = 0; t < ntr; t++) {
      const float* slot = ring_next(ntr);
      if (!slot) {
        failed = true;
        break;
      }
      if (compute) ll_consume(eval, slot, pk, part + kParts * t, nt, nv, r0, c0, c1, c2, lt, lr, fix);
      gc++;
    }
    if (!failed && fix) lr += ll_fixup(eval, CA.rec, fix, c0, c1, c2);
    if (failed) break;
    if (run) {
      lt = warp_sum(lt);
      lr = warp_sum(lr);
      if (lane == 0) {
        if (f != acc_f) {
          publish();
          acc_f = f;
          acc_nsv = nsv;
        }
        fixed_acc(acc_i0, acc_r0, lt);
        fixed_acc(acc_i1, acc_r1, lr);
        acc_n++;
      }
    }
    }  // the log-likelihood pass
    __syncwarp();  // the records of this supervoxel are refilled from the next iteration on
    sc = sn;
    sn = s2;
    ic = in;
  }
  if (failed) {
    // a tile was not delivered within the plan's wait limit: before the warp leaves, every
    // copy it issued -- the late one included -- must have landed in its shared memory, so
    // it waits for them with the fixed bound kLLWaitNs, then reports and leaves
    for (unsigned g = gc; g < gi; g++) mbar_wait(bar0 + 8 * (g % kLLStages), (g / kLLStages) & 1, kLLWaitNs);
    if (lane == 0) atomicOr(&S->flags, F_STAGE_TIMEOUT);
  }
  cp_wait_all();
  publish();
  if (lane == 0 && atomicAdd(&P.work[1], 1) == (int)(gridDim.x * kLLWarps) - 1) {
    P.work[0] = 0;
    P.work[1] = 0;
  }
}

// ===========================================================================
// ll_stream: the log-likelihood pass over the centred voxel stream, FP32 terms (k_ll_pass keeps
// the moment sums and the FP64 terms).  Per voxel and candidate, with the Gaussian's record of
// the kill step (R the upper triangle of Cholesky's factor, R'R = nu W log2(e) / 2):
//   n_j = |R_j (e - u_j)|^2 - log2(weight_j),  ll_v = ln 2 (log2 sum_j 2^(n_min - n_j) - n_min)
// R (e - u) = R e - k with k = R u formed in FP64 from the factor's FP32 values, so that a
// candidate takes seven multiply-adds (4-DOF shape) and no subtraction from every voxel.
//  - A warp's first three supervoxels come by a fixed rule, snake order over the largest-first
//    list (warp w takes places w, 2W-1-w, 2W+w), the others by ticket, three supervoxels ahead:
//    no ticket is waited for, and none is taken on a frame with few supervoxels.
//  - Units of 128 voxels, each lane copying (cp.async) the very voxels it will read, so that a
//    lane waits for its own copies only: no barrier, no elected lane.  Units are end-aligned as
//    the tiles are; the first one's missing voxels are copied as zeros (intensity 0: they add
//    nothing), so that one form of the loop serves every unit.
//  - Each lane's sum over a block of four units goes into its own fixed-point pair, so that no
//    warp reduction is left per supervoxel; lanes are added when the warp's frame changes.
//  - Candidates that cannot come within 2^-30 of the largest term anywhere in the supervoxel's
//    box are left out of its sums (1-Gvoxel frame: one candidate for 18% of the voxels, two for
//    28, three 25, four 19, five 10; where nuclei crowd at one per 3000 voxels all five stay).
// 14.5 M voxels a launch: 57.3 us, 31.0 M warp instructions (as one float4 tile ring over five
// candidates, tickets and a warp reduction per supervoxel: 69.3 us, 40.9 M); 12.6 M voxels in 16
// crowded volumes 67.1 -> 63.5; twelve nuclei 10.6 -> 7.1.  The stream itself takes 35 us at the
// measured 6.5 TB/s; what is left is issue (51% of the slots; the top stall is dependent
// instructions) at 16 warps an SM.  Measured beside it: 20 warps 59.4 / 64.0 us, 24 with a
// shared ring of two or three 70 and more (spills), 256-voxel units 70.5, rings of 4 to 6 units
// 61 to 70 (the L1 that the ring takes is missed), every supervoxel by rule 58.8 / 65.1, the
// candidates' constants held in registers through the loop 61.1 / 65.5.
// ===========================================================================
#ifndef TGMM_LS_WARPS
#define TGMM_LS_WARPS 4
#endif
#ifndef TGMM_LS_BLOCKS
#define TGMM_LS_BLOCKS 4
#endif
constexpr int kLSWarps = TGMM_LS_WARPS;
constexpr int kLSBlocks = TGMM_LS_BLOCKS;
#ifndef TGMM_LS_RING
#define TGMM_LS_RING 3
#endif
constexpr int kLSRing = TGMM_LS_RING;   // units in flight per warp
constexpr int kLSUnit = 128;            // voxels per unit, four per lane
constexpr int kLSFixed = 3;             // supervoxels a warp takes by rule
constexpr int kLSKept = 1024 / kLSUnit; // units of the reference's kept window
// A supervoxel of more than a million voxels leaves carried sums, so that a warp's 32 lanes hold
// fewer than 2^23 parts together: 2^27 voxels of one frame in smaller ones between publications,
// where the device's memory divided by the warps is some 2^22.
constexpr int kLSCarryUnits = (1 << 20) / kLSUnit;
constexpr float kLSZero = -745.13f * kL2E;  // log2 of the smallest positive density
// Candidates whose terms stay this many bits below the largest one over a whole supervoxel are
// left out of its sums: at most 4 2^-30 of them, 5e-9 in log2, below the last bit of an FP32 term.
constexpr float kLSDrop = 30.0f;

// Per-warp shared region: the ring, the fixed-point sums the kept window leaves out (a pair per
// lane), the candidates' FP32 constants, three supervoxel records with their candidate ids
// (fetched two supervoxels ahead) and two sets of candidate records (one ahead).
struct LSRec {
  SvLL ll;
  int32_t cand[8];
};
struct LSCand {
  GaussLL g[kJ];
  double ln_alpha;
  int32_t done, pad;
};
struct LSWarp {
  float4 ring[kLSRing][kLSUnit];
  long long di[32];
  unsigned long long dr[32];
  float cst[56];
  LSRec rec[3];
  LSCand cand[2];
};
static_assert(sizeof(LSRec) % 16 == 0 && sizeof(LSCand) % 16 == 0 && sizeof(LSWarp) % 16 == 0 &&
                  offsetof(LSWarp, rec) % 16 == 0 && offsetof(LSWarp, cst) % 16 == 0,
              "copies of 16 bytes");
constexpr size_t kLSSmemBytes = (size_t)kLSWarps * sizeof(LSWarp);

// The candidates' constants in LSWarp::cst: two packed pairs (two floats a field) and a single
// one, each r00 r01 -k0 r11 -k1 r22 -k2 -log2(weight), then r02 r12 (zero in the 4-DOF form).
// They are read where they are used, once per unit: holding the five candidates' 40 values in
// registers through the loop left no room for more warps (128 registers and spills at 16 warps
// an SM).
struct CandPair {
  float2 r00, r01, r11, r22, k0, k1, k2, b;
};
__device__ __forceinline__ CandPair ls_load_pair(const float* c) {
  const float4* p = reinterpret_cast<const float4*>(c);
  const float4 x = p[0], y = p[1], z = p[2], w = p[3];
  CandPair C;
  C.r00 = make_float2(x.x, x.y), C.r01 = make_float2(x.z, x.w);
  C.k0 = make_float2(y.x, y.y), C.r11 = make_float2(y.z, y.w);
  C.k1 = make_float2(z.x, z.y), C.r22 = make_float2(z.z, z.w);
  C.k2 = make_float2(w.x, w.y), C.b = make_float2(w.z, w.w);
  return C;
}
// n of a pair of candidates
__device__ __forceinline__ float2 ls_pair(const CandPair& C, const float4& v) {
  const float2 E0 = make_float2(v.x, v.x), E1 = make_float2(v.y, v.y), E2 = make_float2(v.z, v.z);
  const float2 s0 = __ffma2_rn(C.r00, E0, __ffma2_rn(C.r01, E1, C.k0));
  const float2 s1 = __ffma2_rn(C.r11, E1, C.k1);
  const float2 s2 = __ffma2_rn(C.r22, E2, C.k2);
  return __ffma2_rn(s0, s0, __ffma2_rn(s1, s1, __ffma2_rn(s2, s2, C.b)));
}
// n of one candidate whose constants lie `st` floats apart
template <bool kGeneral>
__device__ __forceinline__ float ls_single(const float* c, int st, const float4& v) {
  float s0 = fmaf(c[0], v.x, fmaf(c[st], v.y, c[2 * st])), s1 = fmaf(c[3 * st], v.y, c[4 * st]);
  if (kGeneral) {
    s0 = fmaf(c[8 * st], v.z, s0);
    s1 = fmaf(c[9 * st], v.z, s1);
  }
  const float s2 = fmaf(c[5 * st], v.z, c[6 * st]);
  return fmaf(s0, s0, fmaf(s1, s1, fmaf(s2, s2, c[7 * st])));
}

__device__ __forceinline__ float fmin3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// log2 of the densities of kN voxels of this lane in the 4-DOF form, from the first kForm
// candidates (of three, the third is the single one), or (kForm 0) from all five in the general
// form.
template <int kForm, int kN>
__device__ __forceinline__ void ls_log2(const float* cst, const float4 (&v)[kN], float (&l)[kN]) {
  if constexpr (kForm == 1) {
#pragma unroll
    for (int q = 0; q < kN; q++) l[q] = -ls_single<false>(cst, 2, v[q]);
  } else if constexpr (kForm >= 2) {
    float2 n0[kN], n1[kN];
    float n4[kN];
    {
      const CandPair C = ls_load_pair(cst);
#pragma unroll
      for (int q = 0; q < kN; q++) n0[q] = ls_pair(C, v[q]);
    }
    if constexpr (kForm >= 4) {
      const CandPair C = ls_load_pair(cst + 20);
#pragma unroll
      for (int q = 0; q < kN; q++) n1[q] = ls_pair(C, v[q]);
    }
    if constexpr (kForm == 3 || kForm == 5) {
#pragma unroll
      for (int q = 0; q < kN; q++) n4[q] = ls_single<false>(cst + 40, 1, v[q]);
    }
#pragma unroll
    for (int q = 0; q < kN; q++) {
      float nm = fminf(n0[q].x, n0[q].y);
      if constexpr (kForm == 3) nm = fminf(nm, n4[q]);
      if constexpr (kForm == 4) nm = fmin3(nm, n1[q].x, n1[q].y);
      if constexpr (kForm == 5) nm = fmin3(fmin3(n0[q].x, n0[q].y, n1[q].x), n1[q].y, n4[q]);
      float s = ex2_approx(nm - n0[q].x) + ex2_approx(nm - n0[q].y);
      if constexpr (kForm >= 4) s += ex2_approx(nm - n1[q].x) + ex2_approx(nm - n1[q].y);
      if constexpr (kForm == 3 || kForm == 5) s += ex2_approx(nm - n4[q]);
      l[q] = lg2_approx(s) - nm;
    }
  } else {
#pragma unroll
    for (int q = 0; q < kN; q++) {
      float n[kJ], s = 0.0f;
#pragma unroll
      for (int j = 0; j < kJ; j++) n[j] = ls_single<true>(cst + (j < 4 ? (j >> 1) * 20 + (j & 1) : 40), j < 4 ? 2 : 1, v[q]);
      const float nm = fmin3(fmin3(n[0], n[1], n[2]), n[3], n[4]);
#pragma unroll
      for (int j = 0; j < kJ; j++) s += ex2_approx(nm - n[j]);
      l[q] = lg2_approx(s) - nm;
    }
  }
}
__device__ __forceinline__ float ls_log2_one(const float* cst, float4 x) {
  const float4 v[1] = {x};
  float l[1];
  ls_log2<0, 1>(cst, v, l);
  return l[0];
}

// 16 bytes global -> shared by this lane; `bytes` 0 writes zeros and reads nothing.
__device__ __forceinline__ void cp_async16_fill(unsigned dst, const void* src, unsigned bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async16_to(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// Waits until at most n of this lane's groups of copies are outstanding (n >= kLSRing - 1: that
// many).
template <int N = kLSRing - 1>
__device__ __forceinline__ void ls_wait(int n) {
  if constexpr (N > 0) {
    if (n < N) {
      ls_wait<N - 1>(n);
      return;
    }
  }
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// A unit with the per-voxel zero-density test (the reference skips such a voxel), from its
// place `first` on.  Rare.
__device__ __noinline__ float ls_unit_tested(const float* cst, const float4* slot, int first, bool* allok) {
  const int lane = threadIdx.x & 31;
  float s = 0.0f;
  for (int u = 0; u < kLSUnit / 32; u++) {
    const float4 v = slot[32 * u + lane];
    const float l = ls_log2_one(cst, v);
    const bool ok = l > kLSZero, in = 32 * u + lane >= first;
    *allok = *allok && (ok || !in);
    s += (in && ok) ? v.w * l : 0.0f;
  }
  return s;
}

// The kept units (bit k of `mask`: unit nu - kLSKept + k) that hold voxels of zero density: the
// reference's value for each such voxel, the last one of its stride of 1024 with a positive
// density (in log2).  Rare; reads global memory.
__device__ __noinline__ double ls_fixup(const float* cst, const float4* v, int nu, int r0, unsigned mask) {
  const int lane = threadIdx.x & 31;
  double add = 0.0;
  for (int k = 0; k < kLSKept; k++) {
    if (!(mask & (1u << k))) continue;
    const int t = nu - kLSKept + k;
    const int start = t == 0 ? 0 : r0 + (t - 1) * kLSUnit, rem = t == 0 ? r0 : kLSUnit;
    for (int o = lane; o < rem; o += 32) {
      const float4 x = v[start + o];
      if (ls_log2_one(cst, x) > kLSZero) continue;
      for (int i = start + o - 1024; i >= 0; i -= 1024) {
        const float4 y = v[i];
        const float l = ls_log2_one(cst, y);
        if (l > kLSZero) {
          add += (double)y.w * (double)l;
          break;
        }
      }
    }
  }
  return add;
}

// This lane's part of a unit (its slot, from the lane's own voxel on) in one of the forms: sum
// of I log2(density), smallest log2(density).
template <int kForm>
__device__ __forceinline__ void ls_unit(const float* cst, const float4* slot, float& s, float& lmin) {
  float4 v[4];
  float l[4];
#pragma unroll
  for (int q = 0; q < 4; q++) v[q] = slot[32 * q];
  ls_log2<kForm, 4>(cst, v, l);
#pragma unroll
  for (int q = 0; q < 4; q++) {
    lmin = fminf(lmin, l[q]);
    s = fmaf(v[q].w, l[q], s);
  }
}

// A supervoxel with a candidate whose precision has no Cholesky factor (records handed in with
// an indefinite matrix, which the regularisation never produces): every voxel from the
// quadratic form itself in FP64.  Adds this lane's share to the two fixed-point pairs.
__device__ __noinline__ void ls_general(const DevPlan& P, const SvLL& R, const int32_t* cand, double ln_alpha,
                                        long long* ai, unsigned long long* ar, long long* di,
                                        unsigned long long* dr) {
  const int lane = threadIdx.x & 31;
  const float4* v = P.vox4 + R.v0;
  auto ll_of = [&](float4 x) {
    double dens = 0.0;
    for (int j = 0; j < kJ; j++) {
      const double* L = P.llc + (int64_t)cand[j] * 10;
      const double d0 = (double)x.x + ((double)R.c0 - L[7]), d1 = (double)x.y + ((double)R.c1 - L[8]),
                   d2 = (double)x.z + ((double)R.c2 - L[9]);
      dens += exp(L[6] - ln_alpha + L[0] * d0 * d0 + L[1] * d0 * d1 + L[2] * d0 * d2 + L[3] * d1 * d1 +
                  L[4] * d1 * d2 + L[5] * d2 * d2);
    }
    return dens > 0.0 ? log(dens) : -kInf;
  };
  double all = 0.0, kept = 0.0;
  for (int i = lane; i < R.nv; i += 32) {
    const float4 x = v[i];
    double l = ll_of(x);
    if (l > -kInf) all += (double)x.w * l;
    if (i < R.nv - 1024) continue;
    double w = x.w;
    for (int b = i - 1024; !(l > -kInf) && R.nv > 1024 && b >= 0; b -= 1024) {
      l = ll_of(v[b]);
      w = v[b].w;
    }
    if (l > -kInf) kept += w * l;
  }
  fixed_acc(*ai, *ar, all);
  long long ki = 0;
  unsigned long long kr = 0;
  fixed_acc(ki, kr, kept);
  long long bi = 0;
  unsigned long long br = 0;
  fixed_acc(bi, br, all);
  *di += ki - bi;
  *dr += kr - br;
}

// With G > 0 the warps also run the kNN/E-step of the next iteration (G lanes per
// supervoxel, 32/G supervoxels an item, from a second work counter): one item after each
// supervoxel's look-ahead copies are issued, and the rest once the voxel work has run out.
// It needs only what the kill step left, and its results go to the next iteration's
// buffers, so it runs ahead of the convergence test; a frame that converges here never
// reads them.
template <int G>
__global__ void __launch_bounds__(kLSWarps * 32, kLSBlocks) k_ll_stream(DevPlan P) {
  const int total = P.info->total_sv;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // A lone frame that an earlier launch ended leaves nothing to do.  One that this launch ends
  // while a block is still waiting for a place on an SM does not count: its warps arrive at the
  // work counters like the others, whose last one resets them.
  if (P.info->n_frames == 1) {
    const int done = *(volatile const int32_t*)&P.state[0].done;
    if (done != 0 && done != P.iter) return;
  }
  extern __shared__ __align__(128) unsigned char ll_smem[];
  LSWarp& Sh = reinterpret_cast<LSWarp*>(ll_smem)[warp];
  const unsigned ring_a = smem_addr(&Sh.ring[0][lane]);
  const int W = gridDim.x * kLSWarps, w = warp * gridDim.x + blockIdx.x;
  // the supervoxel this warp takes i-th, or -1: the first kLSFixed by rule, then by ticket
  auto take = [&](int i) {
    int64_t p = (int64_t)i * W + ((i & 1) ? W - 1 - w : w);
    if (i >= kLSFixed) {
      p = total;
      if (total > kLSFixed * W && lane == 0) p = (int64_t)kLSFixed * W + atomicAdd(&P.work[0], 1);
      // (lane 0's place; the others get the supervoxel where it is first used)
    }
    return p < total ? P.sv_order[p] : -1;
  };
  auto fetch_rec = [&](int s, LSRec& X) {
    if (s < 0) return;
    if (lane < 3)
      cp_async16(reinterpret_cast<char*>(&X.ll) + 16 * lane, reinterpret_cast<const char*>(P.sv_ll + s) + 16 * lane);
    else if (lane < 3 + kJ)
      cp_async4(&X.cand[lane - 3], cand_buf(P, P.iter) + (int64_t)s * kJ + lane - 3);
  };
  static_assert(sizeof(GaussLL) == 64, "four lanes a candidate");
  auto fetch_cand = [&](int s, const LSRec& A, LSCand& X) {
    if (s < 0) return;
    if (lane < 4 * kJ) {
      const int j = lane >> 2;
      cp_async16(reinterpret_cast<char*>(&X.g[j]) + 16 * (lane & 3),
                 reinterpret_cast<const char*>(P.gll + A.cand[j]) + 16 * (lane & 3));
    } else if (lane == 4 * kJ) {
      cp_async8(&X.ln_alpha, &P.state[A.ll.frame].ln_alpha);
    } else if (lane == 4 * kJ + 1) {
      cp_async4(&X.done, &P.state[A.ll.frame].done);
    }
  };
  // this lane's fixed-point sums over the warp's run of supervoxels of one frame: every voxel
  // here, what the reference's kept window leaves out in Sh.di, Sh.dr
  int acc_f = -1, acc_nsv = 0, acc_n = 0;
  long long ai = 0;
  unsigned long long ar = 0;
  Sh.di[lane] = 0;
  Sh.dr[lane] = 0;
  auto publish = [&]() {
    if (acc_n > 0) {
      long long ri = ai + Sh.di[lane];
      unsigned long long rr = ar + Sh.dr[lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        ai += __shfl_xor_sync(0xffffffffu, ai, o);
        ar += __shfl_xor_sync(0xffffffffu, ar, o);
        ri += __shfl_xor_sync(0xffffffffu, ri, o);
        rr += __shfl_xor_sync(0xffffffffu, rr, o);
      }
      if (lane == 0) {
        FrameState* S = &P.state[acc_f];
        fixed_carry(ai, ar);
        fixed_carry(ri, rr);
        atomicAdd((unsigned long long*)&S->ll_int[0], (unsigned long long)ai);
        atomicAdd((unsigned long long*)&S->ll_int[1], (unsigned long long)ri);
        atomicAdd(&S->ll_frac[0], ar);
        atomicAdd(&S->ll_frac[1], rr);
        __threadfence();
        if (atomicAdd(&S->sv_done, acc_n) == acc_nsv - acc_n) {
          __threadfence();
          frame_converge(P, acc_f);
        }
      }
      __syncwarp();
    }
    acc_n = 0;
    ai = 0;
    ar = 0;
    Sh.di[lane] = 0;
    Sh.dr[lane] = 0;
  };
  constexpr int kPerItem = G > 0 ? 32 / G : 1;
  const int knn_items = G > 0 ? (total + kPerItem - 1) / kPerItem : 0;
  bool knn_more = G > 0;
  auto knn_step = [&]() {
    if constexpr (G > 0) {
      int item = 0;
      if (lane == 0) item = atomicAdd(&P.work[2], 1);
      item = __shfl_sync(0xffffffffu, item, 0);
      if (item < knn_items) {
        const int gl = lane & (G - 1), gbase = lane - gl;
        const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << G) - 1u) << gbase;
        knn_estep_sv<G>(P, item * kPerItem + gbase / G, P.iter + 1, gl, gbase, gmask, nullptr, nullptr);
        __syncwarp();
      } else {
        knn_more = false;
      }
    }
  };
  int s0 = take(0), s1 = take(1), s2 = take(2);
  fetch_rec(s0, Sh.rec[0]);
  fetch_rec(s1, Sh.rec[1]);
  cp_commit();
  cp_wait_all();
  __syncwarp();
  fetch_cand(s0, Sh.rec[0], Sh.cand[0]);
  cp_commit();
  // units copied and read by this warp; the unit to copy next and how many of its supervoxel
  // (the current one, or with on_next the one after) are left to copy; the units copied when
  // the last records were asked for
  unsigned gi = 0, gc = 0, g_rec = 0;
  const float4* src = nullptr;
  int left = 0, part = 0;
  bool on_next = false, asked = false;
  for (int i = 0; s0 >= 0; i++) {
    // the records asked for a supervoxel ago, which went with the unit copied next
    if (asked) cp_commit();
    ls_wait(asked ? 0 : (int)(gi - g_rec));
    __syncwarp();
    const LSRec& A = Sh.rec[i % 3];
    const LSRec& B = Sh.rec[(i + 1) % 3];
    const LSCand& K = Sh.cand[i & 1];
    const int nv = A.ll.nv, f = A.ll.frame;
    const int nu = (nv + kLSUnit - 1) / kLSUnit, gap = nu * kLSUnit - nv;
    if (!on_next) {  // its copies start here
      src = P.vox4 + A.ll.v0 + lane - gap;
      left = nu;
      part = gap;
    }
    on_next = false;
    const bool run = K.done == 0;
    if (run && f != acc_f) {  // the sums so far are the previous frame's
      publish();
      acc_f = f;
      acc_nsv = A.ll.frame_nsv;
    }
    // the candidates' FP32 constants, a candidate on each of five lanes, and bounds of its n over
    // the supervoxel's box (each row of R (e - u) lies in an interval there)
    float b = 0.0f, r00 = 0.0f, least = kInfF, most = kInfF;
    bool wide = false;
    float r01 = 0.0f, r02 = 0.0f, r11 = 0.0f, r12 = 0.0f, r22 = 0.0f, k0 = 0.0f, k1 = 0.0f, k2 = 0.0f;
    if (lane < kJ) {
      const GaussLL& g = K.g[lane];
      const double u0 = g.m[0] - (double)A.ll.c0, u1 = g.m[1] - (double)A.ll.c1, u2 = g.m[2] - (double)A.ll.c2;
      r00 = g.r[0], r01 = g.r[1], r02 = g.r[2], r11 = g.r[3], r12 = g.r[4], r22 = g.r[5];
      k0 = __double2float_rn((double)r00 * u0 + (double)r01 * u1 + (double)r02 * u2);
      k1 = __double2float_rn((double)r11 * u1 + (double)r12 * u2);
      k2 = __double2float_rn((double)r22 * u2);
      b = __double2float_rn(K.ln_alpha * 1.4426950408889634 - g.b);
      wide = r02 != 0.0f || r12 != 0.0f;
      const float h0 = A.ll.h0, h1 = A.ll.h1, h2 = A.ll.h2;
      const float w0 = fabsf(r00) * h0 + fabsf(r01) * h1 + fabsf(r02) * h2, w1 = fabsf(r11) * h1 + fabsf(r12) * h2,
                  w2 = fabsf(r22) * h2;
      const float x0 = fmaxf(fabsf(k0) - w0, 0.0f), x1 = fmaxf(fabsf(k1) - w1, 0.0f), x2 = fmaxf(fabsf(k2) - w2, 0.0f);
      const float z0 = fabsf(k0) + w0, z1 = fabsf(k1) + w1, z2 = fabsf(k2) + w2;
      least = x0 * x0 + x1 * x1 + x2 * x2 + b;
      most = z0 * z0 + z1 * z1 + z2 * z2 + b;
    }
    const unsigned fin = __ballot_sync(0xffffffffu, lane < kJ && isfinite(b));
    const unsigned bad = __ballot_sync(0xffffffffu, lane < kJ && (isnan(b) || b == -kInfF));
    const unsigned odd = __ballot_sync(0xffffffffu, lane < kJ && isnan(r00) && isfinite(b));
    const bool w4 = !__any_sync(0xffffffffu, wide);
    float top = most;  // some candidate's n is at most this everywhere
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) top = fminf(top, __shfl_xor_sync(0xffffffffu, top, o));
    top = __shfl_sync(0xffffffffu, top, 0);
    // kept: the candidates that can come within kLSDrop bits of the largest term somewhere
    const unsigned keep = __ballot_sync(0xffffffffu, lane < kJ && !(least > top + kLSDrop)) & 31u;
    const int nk = __popc(keep);
    if (lane < kJ) {  // the kept ones first
      const unsigned below = (1u << lane) - 1u;
      int at = (keep >> lane) & 1u ? __popc(keep & below) : nk + __popc(~keep & below);
      if (nk == 3 && (at == 2 || at == 4)) at = 6 - at;  // the third is the single one
      float* c = Sh.cst + (at < 4 ? (at >> 1) * 20 + (at & 1) : 40);
      const int st = at < 4 ? 2 : 1;
      c[0] = r00;
      c[st] = r01;
      c[2 * st] = -k0;
      c[3 * st] = r11;
      c[4 * st] = -k1;
      c[5 * st] = r22;
      c[6 * st] = -k2;
      c[7 * st] = b;
      c[8 * st] = r02;
      c[9 * st] = r12;
    }
    const int form = w4 ? nk : 0;
    __syncwarp();
    // what the next supervoxels need
    fetch_cand(s1, B, Sh.cand[(i + 1) & 1]);
    if (i > 0) s2 = __shfl_sync(0xffffffffu, s2, 0);  // taken a supervoxel ago
    fetch_rec(s2, Sh.rec[(i + 2) % 3]);
    asked = true;
    const int s3 = s2 >= 0 ? take(i + 3) : -1;
    if (knn_more) knn_step();
    // a NaN weight makes the reference's density NaN for every voxel (skipped); no finite weight
    // means a zero density everywhere
    const bool compute = run && fin && !bad;
    const int nnv = s1 >= 0 ? B.ll.nv : 0;
    unsigned fix = 0;
    if (compute && !odd) {
      double lt = 0.0;  // log2 units
      for (int u = 0; u < nu; u++) {
        // refill the ring: this supervoxel's units, then the next one's
        while (gi - gc < kLSRing) {
          if (left == 0) {
            if (on_next || nnv == 0) break;
            on_next = true;
            left = (nnv + kLSUnit - 1) / kLSUnit;
            part = left * kLSUnit - nnv;
            src = P.vox4 + B.ll.v0 + lane - part;
          }
          const unsigned dst = ring_a + (gi % kLSRing) * (kLSUnit * 16);
          if (part == 0) {
#pragma unroll
            for (int q = 0; q < kLSUnit / 32; q++) cp_async16_to(dst + 512 * q, src + 32 * q);
          } else {
#pragma unroll
            for (int q = 0; q < kLSUnit / 32; q++) {
              const bool in = 32 * q + lane >= part;
              cp_async16_fill(dst + 512 * q, in ? src + 32 * q : P.vox4, in ? 16u : 0u);
            }
          }
          cp_commit();
          src += kLSUnit;
          part = 0;
          left--;
          gi++;
          if (asked) {
            asked = false;
            g_rec = gi;
          }
        }
        ls_wait((int)(gi - gc) - 1);  // at most the units after this one
        const float4* slot = &Sh.ring[gc % kLSRing][lane];
        float s = 0.0f, lmin = kInfF;
        switch (form) {
          case 1:
            ls_unit<1>(Sh.cst, slot, s, lmin);
            break;
          case 2:
            ls_unit<2>(Sh.cst, slot, s, lmin);
            break;
          case 3:
            ls_unit<3>(Sh.cst, slot, s, lmin);
            break;
          case 4:
            ls_unit<4>(Sh.cst, slot, s, lmin);
            break;
          case 5:
            ls_unit<5>(Sh.cst, slot, s, lmin);
            break;
          default:
            ls_unit<0>(Sh.cst, slot, s, lmin);
            break;
        }
        if (__any_sync(0xffffffffu, !(lmin > kLSZero) || isnan(s))) {
          bool allok = true;
          s = ls_unit_tested(Sh.cst, slot - lane, u == 0 ? gap : 0, &allok);
          const bool some = __any_sync(0xffffffffu, !allok);
          if (some && nu > kLSKept && u >= nu - kLSKept) fix |= 1u << (u - (nu - kLSKept));
        }
        gc++;
        lt += (double)s;
        if (((nu - 1 - u) & (512 / kLSUnit - 1)) == 0) {  // a block of 512 voxels, from the end
          lt *= kLn2;
          const double fl = floor(lt);
          const long long bi = (long long)fl;
          const unsigned long long br = (unsigned long long)((lt - fl) * kFracScale);
          ai += bi;
          ar += br;
          if (nu - u > kLSKept) {  // before the kept window
            Sh.di[lane] -= bi;
            Sh.dr[lane] -= br;
          }
          lt = 0.0;
        }
      }
      if (fix) {
        long long bi = 0;
        unsigned long long br = 0;
        fixed_acc(bi, br, kLn2 * ls_fixup(Sh.cst, P.vox4 + A.ll.v0, nu, kLSUnit - gap, fix));
        Sh.di[lane] += bi;
        Sh.dr[lane] += br;
      }
      if (nu > kLSCarryUnits) {
        fixed_carry(ai, ar);
        fixed_carry(Sh.di[lane], Sh.dr[lane]);
      }
    } else {
      // its units on their way (all that is) are let land and passed over
      ls_wait(0);
      gc = gi;
      if (compute) ls_general(P, A.ll, A.cand, K.ln_alpha, &ai, &ar, &Sh.di[lane], &Sh.dr[lane]);
    }
    if (run) acc_n++;
    s0 = s1, s1 = s2, s2 = s3;
  }
  cp_wait_all();
  publish();
  while (knn_more) knn_step();
  if ((G > 0 || total > kLSFixed * W) && lane == 0 && atomicAdd(&P.work[1], 1) == W - 1) {
    P.work[0] = 0;
    P.work[1] = 0;
    P.work[2] = 0;
  }
}

// ===========================================================================
// assign + export: post-loop supervoxel assignment (rnk > 0.5, at most 16 per Gaussian,
// GMEMupdateCUDA.cu:4310-4350) and SoA -> AoS.
// ===========================================================================
__global__ void __launch_bounds__(kSvPerBlockT) k_assign(DevPlan P) {
  const int s = blockIdx.x * kSvPerBlockT + threadIdx.x;
  if (s >= P.info->total_sv) return;
  const int f = P.sv_frame[s];
  const FrameDesc D = load_desc(P, f);
  const FrameState& S = P.state[f];
  if (S.flags & (F_BAD_CSR | F_FEW_GAUSS)) return;
  const int sl = s - D.sv_base;
  // the last E-step that ran (a kNN/E-step run ahead of a converged frame is ignored); its
  // responsibilities and candidates are the call's outputs
  const int last = S.iter - 1;
  const float* rnk = rnk_buf(P, last);
  const int32_t* cand = cand_buf(P, last);
#pragma unroll
  for (int j = 0; j < kJ; j++) {
    const float r = rnk[(int64_t)s * kJ + j];
    const int k = cand[(int64_t)s * kJ + j];
    if (last >= 1) {
      D.rnk_out[(int64_t)j * D.n_sv + sl] = r;
      D.ind_out[(int64_t)j * D.n_sv + sl] = k - D.g_base;
    }
    if ((double)r > 0.5) {
      const int b = atomicAdd(&P.acnt[k], 1);
      if (b < kBucketCap) P.abucket[(int64_t)k * kBucketCap + b] = j * D.n_sv + sl;
    }
  }
}

__global__ void __launch_bounds__(kGChunk) k_export(DevPlan P) {
  const int c = blockIdx.x;
  if (c >= P.info->n_gchunks) return;
  const GChunk ch = P.gchunks[c];
  const FrameDesc D = load_desc(P, ch.frame);
  const FrameState S = P.state[ch.frame];
  __shared__ int s_ovf[kGChunk];
  __shared__ int s_novf;
  __shared__ int s_first[kGChunk][TGMM_MAX_SV_PER_GAUSSIAN + 1];
  __shared__ int s_list[kGChunk];
  __shared__ int s_cnt[kGChunk / 32 + 1];
  if (threadIdx.x == 0) s_novf = 0;
  __syncthreads();
  const int k = ch.g_begin + threadIdx.x;
  const bool valid = k < ch.g_end;
  const bool ran = !(S.flags & (F_BAD_CSR | F_FEW_GAUSS));
  int n = 0;
  if (valid && ran) {
    n = P.acnt[k];
    P.acnt[k] = 0;
    if (n > kBucketCap) {
      const int o = atomicAdd(&s_novf, 1);
      s_ovf[o] = threadIdx.x;
      atomicOr(&P.state[ch.frame].flags, F_ASSIGN_OVERFLOW);
    } else {
      int* bk = P.abucket + (int64_t)k * kBucketCap;  // this Gaussian's own bucket
      for (int i = 1; i < n; i++) {                   // insertion sort by position
        const int v = bk[i];
        int q = i;
        while (q > 0 && bk[q - 1] > v) {
          bk[q] = bk[q - 1];
          q--;
        }
        bk[q] = v;
      }
    }
  }
  __syncthreads();
  const int novf = s_novf;
  for (int o = 0; o < novf; o++) {
    const int tk = s_ovf[o];
    int taken = 0;
    int* dst = s_first[tk];
    ordered_scan(P, D, S.iter - 1, ch.g_begin + tk, 0.5, s_list, s_cnt, [&](int p) {
      if (taken < TGMM_MAX_SV_PER_GAUSSIAN) dst[taken++] = p;
    });
    if (threadIdx.x == 0) dst[TGMM_MAX_SV_PER_GAUSSIAN] = taken;
    __syncthreads();
  }
  if (!valid) return;
  TgmmGaussian& g = D.gm[k - D.g_base];
  if (ran) {
    g.beta_k = gcomp(P, G_BETA, k);
    g.nu_k = gcomp(P, G_NU, k);
    g.alpha_k = gcomp(P, G_ALPHA, k);
    for (int d = 0; d < 3; d++) g.m_k[d] = gcomp(P, G_M0 + d, k);
    for (int e = 0; e < 6; e++) g.W_k[e] = gcomp(P, G_W0 + e, k);
    const int last = (S.iter - 1) & 1;  // parity of the last iteration that ran
    const double eld = gcomp(P, G_ELD0 + last, k);
    g.expectedLogDetCovarianceCUDA = eld;
    g.expectedLogResponsivityCUDA = (eld == -1e32) ? -1e32 : gcomp(P, G_PSIA0 + last, k) - S.psi_total[last];
    for (int d = 0; d < 3; d++) g.m_o[d] = gcomp(P, G_MO0 + d, k);
    g.W_o[5] = gcomp(P, G_WO5, k);
    if (n > kBucketCap) {
      const int taken = s_first[threadIdx.x][TGMM_MAX_SV_PER_GAUSSIAN];
      for (int i = 0; i < taken; i++) g.supervoxelIdx[i] = s_first[threadIdx.x][i] % D.n_sv;
      g.supervoxelNum = taken;
    } else {
      const int taken = min(n, TGMM_MAX_SV_PER_GAUSSIAN);
      const int* bk = P.abucket + (int64_t)k * kBucketCap;
      for (int i = 0; i < taken; i++) g.supervoxelIdx[i] = bk[i] % D.n_sv;
      g.supervoxelNum = taken;
    }
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static inline int div_up(int a, int b) { return (a + b - 1) / b; }

void launch_build_maps(const DevPlan& P, cudaStream_t st) {
  k_build_maps<<<dim3(P.max_frames, kMapSlices), kFrameThreads, 0, st>>>(P);
}
// The caller's page-locked records into the plan's device records, 16 bytes a thread, read
// by the SMs over the bus (not a copy engine, so they do not queue behind the caller's own
// uploads), for every frame whose descriptor names a source.
__global__ void __launch_bounds__(256) k_fetch_records(DevPlan P) {
  const int nf = P.info->n_frames;
  for (int f = 0; f < nf; f++) {
    const FrameDesc& D = P.frames[f];
    const uint4* src = reinterpret_cast<const uint4*>(D.gm_src);
    if (!src) continue;
    uint4* dst = reinterpret_cast<uint4*>(D.gm);
    const int64_t n16 = (int64_t)D.n_gauss * (int64_t)sizeof(TgmmGaussian) / 16;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n16; i += (int64_t)gridDim.x * blockDim.x)
      dst[i] = src[i];
  }
}
void launch_fetch_records(const DevPlan& P, cudaStream_t st) {
  k_fetch_records<<<min(P.max_gchunks * (kGChunk * (int)sizeof(TgmmGaussian) / 16 / 256), 148 * 4), 256, 0, st>>>(P);
}
void launch_import(const DevPlan& P, cudaStream_t st) { k_import<<<P.max_gchunks, kGChunk, 0, st>>>(P); }
void launch_order(const DevPlan& P, cudaStream_t st) {
  k_sv_records<<<div_up(P.max_sv, 256), 256, 0, st>>>(P);
  k_order_base<<<P.max_frames, 32, 0, st>>>(P);
  k_order_scatter<<<div_up(P.max_sv, 256), 256, 0, st>>>(P);
}
void launch_moments(const DevPlan& P, cudaStream_t st) {
  k_ll_pass<true><<<P.ll_blocks, kLLWarps * 32, kLLSmemBytes, st>>>(P);
}
void launch_knn_estep(const DevPlan& P, cudaStream_t st) {
  const int G = P.knn_group;
  const int grid = div_up(P.max_sv, kKnnWarps * 32 / G);
  if (G == 32)
    k_knn_estep<32><<<grid, kKnnWarps * 32, 0, st>>>(P);
  else if (G == 16)
    k_knn_estep<16><<<grid, kKnnWarps * 32, 0, st>>>(P);
  else if (G == 8)
    k_knn_estep<8><<<grid, kKnnWarps * 32, 0, st>>>(P);
  else
    k_knn_estep<4><<<grid, kKnnWarps * 32, 0, st>>>(P);
}
void launch_mstep_update(const DevPlan& P, cudaStream_t st) {
  k_mstep_update<<<2 * P.max_gchunks, kMChunk, 0, st>>>(P);
}
void launch_kill_prep(const DevPlan& P, cudaStream_t st) {
  k_kill_prep<<<P.max_gchunks, kGChunk, 0, st>>>(P);
}
void launch_ll_pass(const DevPlan& P, int fp64, int knn_group, cudaStream_t st) {
  const int bs = kLLWarps * 32;
  if (fp64)
    k_ll_pass<false><<<P.ll_blocks64, bs, kLLSmemBytes, st>>>(P);
  else if (knn_group == 8)
    k_ll_stream<8><<<P.ls_blocks, kLSWarps * 32, kLSSmemBytes, st>>>(P);
  else if (knn_group == 16)
    k_ll_stream<16><<<P.ls_blocks, kLSWarps * 32, kLSSmemBytes, st>>>(P);
  else if (knn_group == 32)
    k_ll_stream<32><<<P.ls_blocks, kLSWarps * 32, kLSSmemBytes, st>>>(P);
  else
    k_ll_stream<0><<<P.ls_blocks, kLSWarps * 32, kLSSmemBytes, st>>>(P);
}

// Host tables reach the device as launch parameters of k_stage (24 KB a launch), so staging
// a batch takes no copy engine: a batch is not queued behind large uploads of other frames.
constexpr int kStageChunk16 = 1536;
struct StageArgs {
  uint4* dst;
  int n16;
  int pad;
  uint4 data[kStageChunk16];
};

__global__ void __launch_bounds__(256) k_stage(const __grid_constant__ StageArgs a) {
  for (int i = threadIdx.x; i < a.n16; i += blockDim.x) a.dst[i] = a.data[i];
}

cudaError_t launch_stage_bytes(void* dst, const void* src, size_t bytes, cudaStream_t st) {
  StageArgs a;
  const unsigned char* s = static_cast<const unsigned char*>(src);
  for (size_t off = 0; off < bytes; off += 16 * (size_t)kStageChunk16) {
    const size_t n = std::min(bytes - off, 16 * (size_t)kStageChunk16);
    memset(a.data, 0, 16 * ((n + 15) / 16));
    memcpy(a.data, s + off, n);
    a.dst = reinterpret_cast<uint4*>(static_cast<unsigned char*>(dst) + off);
    a.n16 = (int)((n + 15) / 16);
    a.pad = 0;
    k_stage<<<1, 256, 0, st>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t configure_kernels(DevPlan& P, int device) {
  // the persistent grids: the moment pass, the FP64 log-likelihood (whose per-warp constants take
  // more shared memory), and the fewest blocks an SM of the FP32 log-likelihood's forms
  const void* forms[2] = {(const void*)k_ll_pass<true>, (const void*)k_ll_pass<false>};
  int sms = 0, per = 1 << 30, per64 = 1 << 30;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  for (int i = 0; i < 2; i++) {
    int p = 0;
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(forms[i], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLLSmemBytes);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, forms[i], kLLWarps * 32, kLLSmemBytes);
    int& m = i < 1 ? per : per64;
    m = p < m ? p : m;
  }
  const void* stream_forms[4] = {(const void*)k_ll_stream<0>, (const void*)k_ll_stream<8>,
                                 (const void*)k_ll_stream<16>, (const void*)k_ll_stream<32>};
  int pers = 1 << 30;
  for (const void* fn : stream_forms) {
    int p = 0;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLSSmemBytes);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&p, fn, kLSWarps * 32, kLSSmemBytes);
    pers = std::min(pers, p);
  }
  // no more blocks than supervoxels: a small plan's warps spread over the SMs
  P.ls_blocks = std::max(1, std::min(P.max_sv, sms * (pers > 0 && pers < (1 << 30) ? pers : 1)));
  P.ll_blocks = sms * (per > 0 && per < (1 << 30) ? per : 1);
  P.ll_blocks64 = sms * (per64 > 0 && per64 < (1 << 30) ? per64 : 1);
  return e;
}
// The condition of the next iteration's conditional graph node: whether any frame of the
// batch is still running (its done flag is set by the voxel pass's convergence test, or at
// the start for a frame that cannot run).  A batch whose frames have all stopped skips the
// remaining iterations' launches, which would find nothing to do.
__global__ void __launch_bounds__(1024) k_iter_cond(DevPlan P, cudaGraphConditionalHandle h) {
  const int nf = P.info->n_frames;
  int running = 0;
  for (int f = threadIdx.x; f < nf; f += blockDim.x) running |= P.state[f].done == 0;
  running = __syncthreads_or(running);
  if (threadIdx.x == 0) cudaGraphSetConditional(h, running ? 1u : 0u);
}
void launch_iter_cond(const DevPlan& P, cudaGraphConditionalHandle h, cudaStream_t st) {
  k_iter_cond<<<1, 1024, 0, st>>>(P, h);
}

void launch_assign(const DevPlan& P, cudaStream_t st) {
  k_assign<<<div_up(P.max_sv, kSvPerBlockT), kSvPerBlockT, 0, st>>>(P);
}
void launch_export(const DevPlan& P, cudaStream_t st) { k_export<<<P.max_gchunks, kGChunk, 0, st>>>(P); }


// ---------------------------------------------------------------------------
// Standalone exact kNN (tgmm_knn, tgmm_knn_k, tgmm_knn_noalloc): a uniform grid over one
// point set, then the queries.
//   k_sa_bounds  the queries' bounding box and the grid over it (many blocks, the last one
//                to finish sets the geometry);
//   k_sa_count   each reference point's cell and its place within the cell, and the extent of the
//                cells that hold any;
//   k_sa_start   each cell's place in the sorted references: the cells of an x-row one after the
//                other (the searches read a stretch of a row as one range), the rows in any order
//                (the searches order by (distance, index));
//   k_sa_fill    the references into their places;
//   k_sa_query_group, k_sa_query_warp   16 lanes per query, or a warp per 32 (see sa_query).
// ---------------------------------------------------------------------------

// Scratch of one search over nref points, carved from one buffer (the first kSaClear +
// 4 * budget bytes start at zero).
struct SaScratch {
  FrameState* S;   // the grid geometry (lo, h, inv_h, dims, n_cells)
  unsigned* box;   // keys of the box (see box_key), arrived blocks, next free place, and from
                   // kSaExtent on the extent of the cells that hold references (see k_sa_count)
  int* cnt;        // [budget] references per cell
  int* start;      // [budget] the cell's first place
  int2* place;     // [nref] cell (-1: in none) and place within it
  float4* refs;    // [nref] coordinates and index, cell by cell
};
constexpr int kSaExtent = 8;
static_assert((kSaExtent + 6) * 4 <= (int)(kSaClear - kSaBox), "the header holds the box and the extent");
static_assert(sizeof(FrameState) <= kSaBox, "the grid geometry record fits its part of the scratch header");

static SaScratch sa_carve(char* buf, int32_t nref) {
  SaScratch w;
  w.S = (FrameState*)buf;
  w.box = (unsigned*)(buf + kSaBox);
  w.cnt = (int*)(buf + kSaClear);
  w.start = (int*)(buf + knn_scratch_start(nref));
  w.place = (int2*)(buf + knn_scratch_place(nref));
  w.refs = (float4*)(buf + knn_scratch_refs(nref));
  return w;
}

// Floats as unsigned keys in the same order; the key of the smallest is above 0, so that a
// cleared word is the identity of a maximum (minima are kept as the maxima of ~key).
__device__ __forceinline__ unsigned box_key(float f) {
  const unsigned b = __float_as_uint(f);
  return b & 0x80000000u ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float box_value(unsigned k) {
  return __uint_as_float(k & 0x80000000u ? k & 0x7fffffffu : ~k);
}

// Bounded by the read of the queries (12 bytes each); one block took 187 us for 1.43 M
// queries, the whole device 5-6 us.  Non-finite coordinates are left out of the box.
__global__ void __launch_bounds__(256) k_sa_bounds(const float* __restrict__ q, int64_t nq, float s0, float s1,
                                                   float s2, int nref, int budget, int per_cell, SaScratch w) {
  __shared__ unsigned sm[6][8];
  const float sc[3] = {s0, s1, s2};
  unsigned lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};  // lo: the largest ~key
#pragma unroll 4
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nq; i += (int64_t)gridDim.x * blockDim.x)
#pragma unroll
    for (int d = 0; d < 3; d++) {
      const float y = q[d * nq + i] * sc[d];
      if (!isfinite(y)) continue;
      const unsigned k = box_key(y);
      lo[d] = max(lo[d], ~k);
      hi[d] = max(hi[d], k);
    }
  const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    lo[d] = __reduce_max_sync(0xffffffffu, lo[d]);
    hi[d] = __reduce_max_sync(0xffffffffu, hi[d]);
    if (lane == 0) {
      sm[d][wp] = lo[d];
      sm[3 + d][wp] = hi[d];
    }
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    unsigned m = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) m = max(m, sm[threadIdx.x][i]);
    if (m) atomicMax(&w.box[threadIdx.x], m);
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (atomicAdd(&w.box[6], 1u) != gridDim.x - 1) return;
  __threadfence();
  float flo[3], fhi[3];
  for (int d = 0; d < 3; d++) {
    const unsigned a = __ldcg(&w.box[d]), b = __ldcg(&w.box[3 + d]);
    flo[d] = fhi[d] = 0.0f;  // no finite coordinate
    if (b != 0) {
      flo[d] = box_value(~a);
      fhi[d] = box_value(b);
    }
  }
  set_geometry(w.S, flo, fhi, nref, budget, per_cell);
}

// Reference point k, coordinate d, sits at ref[k * step + d * comp]: AoS xyz (step 3,
// comp 1) or SoA x-block, y-block, z-block (step 1, comp nref).
__global__ void __launch_bounds__(256) k_sa_count(const float* __restrict__ ref, int nref, int step, int64_t comp,
                                                  float s0, float s1, float s2, SaScratch w) {
  // the block's extent of cells, as maxima over cleared words: kMaxGridDim - the smallest, and one
  // more than the largest
  __shared__ unsigned ext[6];
  if (threadIdx.x < 6) ext[threadIdx.x] = 0;
  __syncthreads();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  int2 p = make_int2(-1, 0);
  unsigned m[6] = {0, 0, 0, 0, 0, 0};
  if (k < nref) {
    const float* rk = ref + (int64_t)k * step;
    const float ys[3] = {rk[0] * s0, rk[comp] * s1, rk[2 * comp] * s2};
    bool in = true;
    for (int d = 0; d < 3; d++)
      if (!isfinite(ys[d]) || fabsf(ys[d]) >= 1e25f) in = false;
    if (in) {
      int c[3];
#pragma unroll
      for (int d = 0; d < 3; d++) {
        c[d] = cell_coord(ys[d], w.S->lo[d], w.S->inv_h, w.S->dims[d]);
        m[d] = (unsigned)(kMaxGridDim - c[d]);
        m[3 + d] = (unsigned)(c[d] + 1);
      }
      p.x = (c[2] * w.S->dims[1] + c[1]) * w.S->dims[0] + c[0];
      p.y = atomicAdd(&w.cnt[p.x], 1);
    }
    w.place[k] = p;
  }
#pragma unroll
  for (int d = 0; d < 6; d++) {
    m[d] = __reduce_max_sync(0xffffffffu, m[d]);
    if ((threadIdx.x & 31) == 0 && m[d]) atomicMax(&ext[d], m[d]);
  }
  __syncthreads();
  if (threadIdx.x < 6 && ext[threadIdx.x]) atomicMax(&w.box[kSaExtent + threadIdx.x], ext[threadIdx.x]);
}

// A warp per x-row of cells: the row's references get one contiguous range, its cells in
// order, the rows in any order (the searches order by (distance, index)).
__global__ void __launch_bounds__(256) k_sa_start(SaScratch w) {
  const int lane = threadIdx.x & 31;
  const int nx = w.S->dims[0], rows = w.S->dims[1] * w.S->dims[2];
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += (gridDim.x * blockDim.x) >> 5) {
    int total = 0;
    for (int x = lane; x < nx; x += 32) total += w.cnt[r * nx + x];
    total = __reduce_add_sync(0xffffffffu, total);
    int base = 0;
    if (lane == 0 && total > 0) base = (int)atomicAdd(&w.box[7], (unsigned)total);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int x0 = 0; x0 < nx; x0 += 32) {
      const int x = x0 + lane;
      const int m = x < nx ? w.cnt[r * nx + x] : 0;
      int inc = m;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (x < nx) w.start[r * nx + x] = base + inc - m;
      base += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
}

__global__ void __launch_bounds__(256) k_sa_fill(const float* __restrict__ ref, int nref, int step, int64_t comp,
                                                 SaScratch w) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nref) return;
  const int2 p = w.place[k];
  if (p.x < 0) return;
  const float* rk = ref + (int64_t)k * step;
  w.refs[w.start[p.x] + p.y] = make_float4(rk[0], rk[comp], rk[2 * comp], __int_as_float(k));
}

template <typename F>
__device__ __forceinline__ void sa_scan_cell(const SaScratch& w, int cell, float q0, float q1, float q2, const float* s,
                                             F take) {
  const int n = w.cnt[cell];
  if (n == 0) return;  // (most cells of a far query's rings)
  const int b = w.start[cell], e = b + n;
  for (int k = b; k < e; ++k) {
    const float4 rr = w.refs[k];
    take(knn_dist(q0, q1, q2, rr.x, rr.y, rr.z, s), __float_as_int(rr.w));
  }
}

// The rings of cells of a ring search: those at Chebyshev distance first .. last from the query's
// cell, clipped to the cells [lo, hi] that hold the references.  A query far from all of them
// starts at their box: no ring before it holds a cell.  first > last without a reference.
struct SaRings {
  int lo[3], hi[3], first, last;
  __device__ __forceinline__ SaRings(const GridPlace& p, const SaScratch& w) {
    first = last = 0;
    const unsigned* e = w.box + kSaExtent;
    if (e[3] == 0) first = 1;  // no reference in the grid
#pragma unroll
    for (int a = 0; a < 3; a++) {
      lo[a] = kMaxGridDim - (int)e[a];
      hi[a] = (int)e[3 + a] - 1;
      first = max(first, max(lo[a] - p.c[a], p.c[a] - hi[a]));
      last = max(last, max(p.c[a] - lo[a], hi[a] - p.c[a]));
    }
    if (e[3] == 0) last = 0;
  }
  // A squared distance below which every reference lies in the rings up to r (infinite when there
  // is no other): the nearest side behind which rings are left.  A query past the grid's edge (or
  // on a face along an axis of few cells) is not held back by the sides that have none.
  __device__ __forceinline__ float bound2(const GridPlace& p, int r, float h) const {
    float lb = kInfF;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (p.c[a] - r > lo[a]) lb = fminf(lb, p.f0[a] + r * h);
      if (p.c[a] + r < hi[a]) lb = fminf(lb, p.f1[a] + r * h);
    }
    if (lb == kInfF) return kInfF;
    const float m = lb - (p.eps0 + 1e-6f * lb);
    return m > 0.0f ? m * m : 0.0f;
  }
};

// The N nearest of one query by one thread: the cells of one ring after the other, passing over
// those farther than the N-th distance so far.  Ends when the N-th distance is strictly below the
// bound of every cell not visited.  A ring's cells are taken face by face -- across z, across y,
// across x -- so that none off the ring is looked at.  The list is a local of the function: by
// reference it would lie in memory, and a query far from a crowd of references compares with it
// thousands of times.
template <int N>
__device__ __noinline__ void sa_search_thread(float q0, float q1, float q2, const float* s, const GridGeom& g,
                                              const SaScratch& w, TopN<N>& out) {
  const GridPlace p(q0, q1, q2, s, g);
  TopN<N> best;
  topn_init<N>(best);
  const SaRings R(p, w);
  // the cells [x0, x1] x [y0, y1] x [z0, z1]
  auto scan = [&](int x0, int x1, int y0, int y1, int z0, int z1) {
    for (int z = z0; z <= z1; z++) {
      const float gz = p.gap2(2, z - p.c[2], g.h);
      if (gz > best.d[N - 1]) continue;
      for (int y = y0; y <= y1; y++) {
        const float gy = gz + p.gap2(1, y - p.c[1], g.h);
        if (gy > best.d[N - 1]) continue;
        const int row = (z * g.dims[1] + y) * g.dims[0];
        // (a row's cells lie one after the other in w.refs: one that holds nothing is passed over)
        if (x0 < x1 && w.start[row + x1] + w.cnt[row + x1] == w.start[row + x0]) continue;
        for (int x = x0; x <= x1; x++) {
          if (gy + p.gap2(0, x - p.c[0], g.h) > best.d[N - 1]) continue;
          sa_scan_cell(w, row + x, q0, q1, q2, s, [&](float d, int id) { topn_insert<N>(best, d, id); });
        }
      }
    }
  };
  for (int r = R.first; r <= R.last; ++r) {
    int lo[3], hi[3], in0[3], in1[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      lo[a] = max(p.c[a] - r, R.lo[a]);
      hi[a] = min(p.c[a] + r, R.hi[a]);
      in0[a] = max(p.c[a] - r + 1, R.lo[a]);
      in1[a] = min(p.c[a] + r - 1, R.hi[a]);
    }
    for (int side = r == 0 ? 1 : 0; side < 2; side++) {  // (r = 0: the query's cell, once)
      const int d = side ? r : -r, x = p.c[0] + d, y = p.c[1] + d, z = p.c[2] + d;
      if (z >= R.lo[2] && z <= R.hi[2]) scan(lo[0], hi[0], lo[1], hi[1], z, z);
      if (y >= R.lo[1] && y <= R.hi[1]) scan(lo[0], hi[0], y, y, in0[2], in1[2]);
      if (x >= R.lo[0] && x <= R.hi[0]) scan(x, x, in0[1], in1[1], in0[2], in1[2]);
    }
    if (best.d[N - 1] < R.bound2(p, r, g.h)) break;
  }
  out = best;
}

// The same by the G lanes of a group.  A ring's cells are stretches of x-rows, each one range of
// w.refs: whole rows on the faces across z and y, single cells on those across x.  A lane takes
// a stretch's range, then the group scans the ranges that hold anything, a reference a lane, and
// merges its lists when something was kept.  Rings 0 and 1 are one.  20,000 queries over a box,
// 20,000 references in one corner of it, K = 10: 3.0 ms (a thread per query over rings clipped to
// the grid alone 52); half of the box 0.34 ms (1.6); eight spots of one slice 1.2 ms (13); one end
// of a line 0.13 ms (3.1).
template <int G, int N>
__device__ __noinline__ void sa_search_group(float q0, float q1, float q2, const float* s, const GridGeom& g,
                                             const SaScratch& w, TopN<N>& best, int gl, unsigned gmask) {
  const GridPlace p(q0, q1, q2, s, g);
  topn_init<N>(best);
  const SaRings R(p, w);
  for (int r = R.first == 0 ? 1 : R.first; r <= max(R.last, R.first == 0 ? 1 : 0); ++r) {
    TopN<N> t;
    topn_init<N>(t);
    bool kept = false;
    const float td = best.d[N - 1];
    const int ti = best.i[N - 1];
    // the ring's extent clipped to the references' cells, and without its faces
    int lo[3], hi[3], in0[3], n_in[3];
    bool face0[3], face1[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const int c0 = p.c[a] - r, c1 = p.c[a] + r;
      face0[a] = c0 >= R.lo[a] && c0 <= R.hi[a];
      face1[a] = c1 >= R.lo[a] && c1 <= R.hi[a];
      lo[a] = max(c0, R.lo[a]);
      hi[a] = min(c1, R.hi[a]);
      in0[a] = max(c0 + 1, R.lo[a]);
      n_in[a] = max(min(c1 - 1, R.hi[a]) - in0[a] + 1, 0);
    }
    const bool whole = r == 1 && R.first == 0;
    const int ny = hi[1] - lo[1] + 1, area = n_in[1] * n_in[2];
    // stretches: the rows across z, the rows across y, the cells across x (whole: every row)
    const int z_rows = whole ? ny * (hi[2] - lo[2] + 1) : (face0[2] + face1[2]) * ny;
    const int y_rows = whole ? 0 : (face0[1] + face1[1]) * n_in[2];
    const int total = z_rows + y_rows + (whole ? 0 : (face0[0] + face1[0]) * area);
    for (int i0 = 0; i0 < total; i0 += G) {
      int i = i0 + gl, b = 0, e = 0;
      if (i < total) {
        int y, z, xa = lo[0], xb = hi[0];
        if (i < z_rows) {
          y = lo[1] + i % ny;
          z = whole ? lo[2] + i / ny : face0[2] && i < ny ? p.c[2] - r : p.c[2] + r;
        } else if ((i -= z_rows) < y_rows) {
          z = in0[2] + i % n_in[2];
          y = face0[1] && i < n_in[2] ? p.c[1] - r : p.c[1] + r;
        } else {
          i -= y_rows;
          xa = xb = face0[0] && i < area ? p.c[0] - r : p.c[0] + r;
          if (i >= area) i -= area;
          y = in0[1] + i % n_in[1];
          z = in0[2] + i / n_in[1];
        }
        const float gap = p.gap2(1, y - p.c[1], g.h) + p.gap2(2, z - p.c[2], g.h) +
                          (xa == xb ? p.gap2(0, xa - p.c[0], g.h) : 0.0f);
        if (!(gap > td)) {
          const int row = (z * g.dims[1] + y) * g.dims[0];
          b = w.start[row + xa];
          e = w.start[row + xb] + w.cnt[row + xb];
        }
      }
      for (unsigned m = __ballot_sync(gmask, e > b) & gmask; m; m &= m - 1) {
        const int from = __ffs(m) - 1, eb = __shfl_sync(gmask, e, from);
        for (int k = __shfl_sync(gmask, b, from) + gl; k < eb; k += G) {
          const float4 rr = w.refs[k];
          const float d = knn_dist(q0, q1, q2, rr.x, rr.y, rr.z, s);
          const int id = __float_as_int(rr.w);
          if (!before(td, ti, d, id)) {
            topn_insert<N>(t, d, id);
            kept = true;
          }
        }
        __syncwarp(gmask);
      }
    }
    if (__any_sync(gmask, kept)) {
      if (gl == 0) {
#pragma unroll
        for (int j = 0; j < N; j++) topn_insert<N>(t, best.d[j], best.i[j]);
      }
      TopN<N> merged;
      group_merge_topn<G, N>(t, merged, gmask);
      best = merged;
    }
    if (best.d[N - 1] < R.bound2(p, r, g.h)) break;
  }
}

__device__ __forceinline__ GridGeom sa_geometry(const SaScratch& w) {
  GridGeom g;
  for (int d = 0; d < 3; d++) {
    g.lo[d] = w.S->lo[d];
    g.dims[d] = w.S->dims[d];
  }
  g.h = w.S->h;
  g.inv_h = w.S->inv_h;
  return g;
}

// Slot j of query i.  kMark (tgmm_knn_k): a slot with no reference closer than 1e32 (squared)
// gets index -1 and distance 1e32; else every slot holds its index.
template <bool kMark>
__device__ __forceinline__ void sa_write(int32_t* ind, float* dist, int64_t nq, int64_t i, int j, float d, int id) {
  const bool real = !kMark || (id != 0x7fffffff && d < 1e32f);
  ind[(int64_t)j * nq + i] = real ? id : -1;
  if (kMark && dist) dist[(int64_t)j * nq + i] = real ? d : 1e32f;
}

// References per grid cell for searches of K: the sphere of the cell's side then holds about
// 2 K references on average.
constexpr int sa_per_cell(int K) { return K <= 4 ? 2 : (K + 1) / 2; }
// The first radius of a search, expected to hold 2 K references at the grid's mean density.
template <int K>
__device__ __forceinline__ float sa_first_radius(float h) {
  return h * cbrtf(2.0f * K * (3.0f / (4.0f * 3.14159265f)) / sa_per_cell(K));
}
// The next radius after n references were found where K to kSaKeep are wanted.
template <int K>
__device__ __forceinline__ float sa_next_radius(float rad, int n) {
  const float f = cbrtf((n < K ? 2.0f * K : 1.5f * K) / ((float)n + 0.5f));
  return rad * (n < K ? fminf(fmaxf(f, 1.25f), 2.0f) : fminf(f, 0.9f));
}

// Blocks an SM of the two query kernels: what the collecting search needs, so that the ring search
// they fall back to, which keeps more in registers, does not cost the others theirs (1.43 M voxels,
// K = 5: 173 us with eight blocks, 178 with the seven of 72 registers).
constexpr int sa_warp_blocks(int K) { return K <= 4 ? 9 : K <= 6 ? 8 : K == 7 ? 7 : K <= 9 ? 6 : 5; }
constexpr int sa_group_blocks(int K) { return K <= 2 ? 10 : K == 3 ? 9 : K <= 5 ? 8 : K == 6 ? 7 : K == 7 ? 6 : K <= 9 ? 5 : 4; }

constexpr int kSaKeep = 64;       // references kept per query of a group
constexpr int kSaKeepWarp = 128;  // references kept per warp of queries
constexpr int kSaTries = 4;       // radii tried before the ring search
constexpr int kSaRounds = 4;      // sets of near queries a warp is split into before it
constexpr int kSaSet = 4;         // fewest queries of a set
constexpr int kSaRows = 256;      // rows of cells scanned at most in one try

// The references within `rad` of the box [lo, hi] (scaled space), collected by the G lanes of a
// group into keep[0 .. cap) in any order: for a point box (kPoint) as (distance, index) of those
// closer than rad by the exact distance, else the references themselves.  Rows of cells are
// contiguous in w.refs; a row is passed over when its gap to the box along y and z is rad or
// more.  Returns how many there are (more than cap: the rest were dropped), or -1 when the rows
// are too many.  References outside the grid's box sit in its boundary cells, farther from a
// box inside it than those cells.  Every lane of the group takes part in every step.
template <int G, bool kPoint, typename T>
__device__ __forceinline__ int sa_collect(const float* qv, const float* lo, const float* hi, float rad, float eps0,
                                          const float* s, const GridGeom& g, const SaScratch& w, T* keep, int cap,
                                          int gl, unsigned gmask) {
  int c0[3], c1[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float m = rad + 2.0f * eps0;
    c0[a] = cell_coord(lo[a] - m, g.lo[a], g.inv_h, g.dims[a]);
    c1[a] = cell_coord(hi[a] + m, g.lo[a], g.inv_h, g.dims[a]);
  }
  if ((int64_t)(c1[1] - c0[1] + 1) * (c1[2] - c0[2] + 1) > kSaRows) return -1;
  const float r2 = rad * rad;
  // squared lower bound of a gap of `v` along one axis
  auto sq = [&](float v) {
    const float m = fmaxf(v - eps0 - 1e-6f * v, 0.0f);
    return m * m;
  };
  int n = 0;
  const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
  for (int z = c0[2]; z <= c1[2]; z++) {
    const float fz = g.lo[2] + z * g.h;
    const float gz = sq(fmaxf(lo[2] - (fz + g.h), fz - hi[2]));
    if (!(gz < r2)) continue;
    for (int y = c0[1]; y <= c1[1]; y++) {
      const float fy = g.lo[1] + y * g.h;
      if (!(gz + sq(fmaxf(lo[1] - (fy + g.h), fy - hi[1])) < r2)) continue;
      const int row = (z * g.dims[1] + y) * g.dims[0];
      const int b = w.start[row + c0[0]], e = w.start[row + c1[0]] + w.cnt[row + c1[0]];
      for (int k0 = b; k0 < e; k0 += G) {
        const int k = k0 + gl;
        bool take = false;
        float4 rr = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float d = 0.0f;
        if (k < e) {
          rr = w.refs[k];
          if (kPoint) {
            d = knn_dist(qv[0], qv[1], qv[2], rr.x, rr.y, rr.z, s);
          } else {
            const float yr[3] = {rr.x * s[0], rr.y * s[1], rr.z * s[2]};
#pragma unroll
            for (int a = 0; a < 3; a++) d += sq(fmaxf(lo[a] - yr[a], yr[a] - hi[a]));
          }
          take = d < r2;
        }
        const unsigned m = __ballot_sync(gmask, take) & gmask;
        const int at = n + __popc(m & below);
        if (take && at < cap) {
          if constexpr (kPoint)
            keep[at] = make_float2(d, rr.w);
          else
            keep[at] = rr;
        }
        n += __popc(m);
      }
    }
  }
  return n;
}

// The K nearest of the n references kept for a warp, in (distance, index) order.  First the
// K + 1 smallest keys -- the distance's upper bits with the place in `keep` below them, two
// instructions a level -- then the K of them in exact order.  Returns false when the K-th and
// the next key share their distance bits, which leaves open which of them belongs.
template <int K>
__device__ __forceinline__ bool sa_select(const float* qv, const float* s, const float4* keep, int n, TopN<K>& t) {
  static_assert(kSaKeepWarp == 128, "seven bits of place in a key");
  unsigned key[K + 1];
#pragma unroll
  for (int j = 0; j <= K; j++) key[j] = 0xffffffffu;
#pragma unroll 4
  for (int k = 0; k < n; k++) {
    const float4 rr = keep[k];
    const float d = knn_dist(qv[0], qv[1], qv[2], rr.x, rr.y, rr.z, s);
    unsigned v = (__float_as_uint(d) & ~127u) | (unsigned)k;
#pragma unroll
    for (int j = 0; j <= K; j++) {
      const unsigned lo = min(key[j], v);
      v = max(key[j], v);
      key[j] = lo;
    }
  }
  topn_init<K>(t);
#pragma unroll
  for (int j = 0; j < K; j++) {
    const float4 rr = keep[key[j] & 127u];
    topn_insert<K>(t, knn_dist(qv[0], qv[1], qv[2], rr.x, rr.y, rr.z, s), __float_as_int(rr.w));
  }
  return (key[K - 1] & ~127u) != (key[K] & ~127u);
}

// A warp's 32 consecutive queries together, for queries whose neighbours in the array are near
// one another (the voxels of a supervoxel): the queries within a cell's side of the first
// collect the references within a radius of their bounding box, then each lane orders them for
// its own query.  A lane's K nearest are exact when its K-th is closer than the radius, since
// every reference not collected is at least the radius away from the box; the largest K-th
// distance is the next radius, which serves all of them.  Queries elsewhere (the warp runs into
// the next supervoxel) are the next set; what is left over (scattered queries, crowded cells,
// distances too close to tell apart by their keys) runs the ring search.  1.43 M voxels against
// 2000 references: 133 us, 71% of the issue slots busy (a thread per query: 239 us).
template <int K, bool kMark>
__global__ void __launch_bounds__(128, sa_warp_blocks(K)) k_sa_query_warp(const float* __restrict__ q, int64_t nq,
                                                       const float* __restrict__ ref, int nref, int step,
                                                       int64_t comp, float s0, float s1, float s2, SaScratch w,
                                                       int32_t* ind, float* dist) {
  __shared__ float4 s_keep[4][kSaKeepWarp];
  const int lane = threadIdx.x & 31;
  float4* keep = s_keep[threadIdx.x >> 5];
  const int64_t i0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) & ~(int64_t)31;
  if (i0 >= nq) return;  // whole warps leave
  const int64_t i = min(i0 + lane, nq - 1);  // the last warp's spare lanes repeat its last query
  const float sc[3] = {s0, s1, s2};
  const float qv[3] = {q[i], q[nq + i], q[2 * nq + i]};
  const float yq[3] = {qv[0] * s0, qv[1] * s1, qv[2] * s2};
  const GridGeom g = sa_geometry(w);
  TopN<K> t;
  topn_init<K>(t);
  const bool fin = isfinite(yq[0]) && isfinite(yq[1]) && isfinite(yq[2]);
  bool waits = fin, done = false;
  for (int round = 0; round < kSaRounds; round++) {
    const unsigned left = __ballot_sync(0xffffffffu, waits);
    if (!left) break;
    const int lead = __ffs(left) - 1;
    bool mine = waits;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float yl = __shfl_sync(0xffffffffu, yq[a], lead);  // every lane takes part
      mine = mine && fabsf(yq[a] - yl) <= g.h;
    }
    if (__popc(__ballot_sync(0xffffffffu, mine)) < kSaSet) break;  // scattered queries
    float lo[3], hi[3], ymax = 0.0f;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const unsigned k = box_key(yq[a]);
      lo[a] = box_value(~__reduce_max_sync(0xffffffffu, mine ? ~k : 0u));
      hi[a] = box_value(__reduce_max_sync(0xffffffffu, mine ? k : 0u));
      ymax = fmaxf(ymax, fmaxf(fabsf(lo[a]), fabsf(hi[a])));
    }
    const float eps0 = 4e-3f + 1e-6f * ymax;
    float rad = sa_first_radius<K>(g.h);
    for (int u = 0; u < kSaTries; u++) {
      const int n = sa_collect<32, false>(qv, lo, hi, rad, eps0, sc, g, w, keep, kSaKeepWarp, lane, 0xffffffffu);
      __syncwarp();
      if (n < 0) break;
      if (n >= K && n <= kSaKeepWarp) {
        bool tell = true, ok = true;
        if (mine) {
          tell = sa_select<K>(qv, sc, keep, n, t);
          ok = t.d[K - 1] < rad * rad * (1.0f - 2e-6f);
          done = tell && ok;
        }
        if (__all_sync(0xffffffffu, ok)) break;
        const float far = __uint_as_float(__reduce_max_sync(0xffffffffu, mine ? __float_as_uint(t.d[K - 1]) : 0u));
        rad = fmaxf(sqrtf(far) * (1.0f + 4e-6f), rad * 1.01f);
      } else {
        rad = sa_next_radius<K>(rad, n);
      }
      __syncwarp();  // every lane is done with the kept references
    }
    __syncwarp();
    waits = waits && !mine;
  }
  if (!done) {
    topn_init<K>(t);
    if (fin) sa_search_thread<K>(qv[0], qv[1], qv[2], sc, g, w, t);
    if (!(t.d[K - 1] < kInfF)) {  // fewer than K finite distances: every reference point
      topn_init<K>(t);
      for (int k = 0; k < nref; k++) {
        const float* rk = ref + (int64_t)k * step;
        topn_insert<K>(t, knn_dist(qv[0], qv[1], qv[2], rk[0], rk[comp], rk[2 * comp], sc), k);
      }
    }
  }
  if (i0 + lane < nq)
#pragma unroll
    for (int j = 0; j < K; j++) sa_write<kMark>(ind, dist, nq, i, j, t.d[j], t.i[j]);
}

// A group of G lanes per query, for queries that are scattered or too few to fill the device
// with a warp per 32: the group collects the references within a radius of the query, and with
// K to kSaKeep of them each lane ranks its share against all and writes those of rank < K, so
// that no sorted list is kept.  Radii are tried in turn, then the ring search.  20,019 queries,
// 20,007 references, K = 10: 48 us, bound by the chain of dependent loads (a thread per query,
// 625 warps on the device: 195 us).
template <int G, int K, bool kMark>
__global__ void __launch_bounds__(128, sa_group_blocks(K)) k_sa_query_group(const float* __restrict__ q, int64_t nq,
                                                        const float* __restrict__ ref, int nref, int step,
                                                        int64_t comp, float s0, float s1, float s2, SaScratch w,
                                                        int32_t* ind, float* dist) {
  __shared__ float2 s_keep[128 / G][kSaKeep];
  const int lane = threadIdx.x & 31, gl = lane & (G - 1);
  float2* keep = s_keep[threadIdx.x / G];
  const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << G) - 1u) << (lane - gl);
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
  if (i >= nq) return;  // whole groups leave together
  const float sc[3] = {s0, s1, s2};
  const float qv[3] = {q[i], q[nq + i], q[2 * nq + i]};
  const float yq[3] = {qv[0] * s0, qv[1] * s1, qv[2] * s2};
  const GridGeom g = sa_geometry(w);
  const bool fin = isfinite(yq[0]) && isfinite(yq[1]) && isfinite(yq[2]);
  if (fin) {
    const float eps0 = 4e-3f + 1e-6f * fmaxf(fmaxf(fabsf(yq[0]), fabsf(yq[1])), fabsf(yq[2]));
    float rad = sa_first_radius<K>(g.h);
    for (int u = 0; u < kSaTries; u++) {
      const int n = sa_collect<G, true>(qv, yq, yq, rad, eps0, sc, g, w, keep, kSaKeep, gl, gmask);
      __syncwarp(gmask);
      if (n < 0) break;
      if (n >= K && n <= kSaKeep) {
        for (int a = gl; a < n; a += G) {
          const float2 e = keep[a];
          int rank = 0;
#pragma unroll 4
          for (int o = 0; o < n; o++) {
            const float2 f = keep[o];
            rank += before(f.x, __float_as_int(f.y), e.x, __float_as_int(e.y)) ? 1 : 0;
          }
          if (rank < K) sa_write<kMark>(ind, dist, nq, i, rank, e.x, __float_as_int(e.y));
        }
        return;
      }
      if (n == 0) break;  // far from the references: the ring search starts at them
      rad = sa_next_radius<K>(rad, n);
    }
  }
  TopN<K> t;
  topn_init<K>(t);
  // (no distance of a query with a NaN or infinite coordinate is finite)
  if (fin) sa_search_group<G, K>(qv[0], qv[1], qv[2], sc, g, w, t, gl, gmask);
  if (!(t.d[K - 1] < kInfF)) {
    TopN<K> mine;
    topn_init<K>(mine);
    for (int k = gl; k < nref; k += G) {
      const float* rk = ref + (int64_t)k * step;
      topn_insert<K>(mine, knn_dist(qv[0], qv[1], qv[2], rk[0], rk[comp], rk[2 * comp], sc), k);
    }
    group_merge_topn<G, K>(mine, t, gmask);
  }
#pragma unroll
  for (int j = 0; j < K; j++)
    if (j % G == gl) sa_write<kMark>(ind, dist, nq, i, j, t.d[j], t.i[j]);
}

// Below this many queries a group of 16 lanes per query, from it on a warp per 32.  Query kernel
// alone, group / warp: 20,019 queries, K = 10: 48 / 147 us; 60,000: 141 / 196; 200,000 voxels,
// K = 5: 150 / 82; 1.43 M: 838 / 133.  Groups of 8 and 32: 52 and 47, 150 and 140, 121 and 239.
// Scattered queries, which the warp form gives to its threads one by one, cost the same on either
// side of the line: 99,999 of them, 20,000 references, K = 5, 144 us by groups, 100,000 by warps 134
// (a thread per query without either form 398).
constexpr int64_t kSaGroupBelow = 100000;

template <int K, bool kMark>
static void sa_query(const float* q, int64_t nq, const float* ref, int32_t nref, int step, int64_t comp,
                     const float scale[3], const SaScratch& w, int32_t* ind, float* dist, cudaStream_t st) {
  if (nq < kSaGroupBelow)
    k_sa_query_group<16, K, kMark><<<(unsigned)((nq * 16 + 127) / 128), 128, 0, st>>>(
        q, nq, ref, nref, step, comp, scale[0], scale[1], scale[2], w, ind, dist);
  else
    k_sa_query_warp<K, kMark><<<(unsigned)((nq + 127) / 128), 128, 0, st>>>(
        q, nq, ref, nref, step, comp, scale[0], scale[1], scale[2], w, ind, dist);
}

// The grid over the references and the queries' box, in `buf` (knn_grid_scratch_bytes(nref)).
static cudaError_t sa_build(const float* q, int64_t nq, const float* ref, int32_t nref, int step, int64_t comp,
                            const float scale[3], int K, char* buf, SaScratch* w, cudaStream_t st) {
  *w = sa_carve(buf, nref);
  const int budget = 2 * nref + 2;
  cudaError_t e = cudaMemsetAsync(buf + kSaBox, 0, kSaClear - kSaBox + 4 * (size_t)budget, st);
  if (e != cudaSuccess) return e;
  const int64_t nb = (nq + 1023) / 1024;
  k_sa_bounds<<<(unsigned)(nb < 592 ? nb : 592), 256, 0, st>>>(q, nq, scale[0], scale[1], scale[2], nref, budget,
                                                             sa_per_cell(K), *w);
  const int gb = (nref + 255) / 256;
  k_sa_count<<<gb, 256, 0, st>>>(ref, nref, step, comp, scale[0], scale[1], scale[2], *w);
  k_sa_start<<<(unsigned)std::min(592, (budget + 255) / 256), 256, 0, st>>>(*w);
  k_sa_fill<<<gb, 256, 0, st>>>(ref, nref, step, comp, *w);
  return cudaGetLastError();
}

cudaError_t knn_grid_standalone(const float* q, int64_t nq, const float* ref, int32_t nref, const float scale[3],
                                int32_t* ind, cudaStream_t st) {
  char* buf = nullptr;
  cudaError_t e = scratch_alloc((void**)&buf, knn_grid_scratch_bytes(nref), st);
  if (e != cudaSuccess) return e;
  e = knn_grid_in_scratch(q, nq, ref, nref, scale, ind, st, buf);
  const cudaError_t ef = cudaFreeAsync(buf, st);
  return e != cudaSuccess ? e : ef;
}

// The K-nearest grid search (1 <= K <= kMaxK) over reference points in AoS or SoA layout
// (see k_sa_count), with distances; scratch from the stream-ordered allocator.
cudaError_t knn_grid_topk(const float* q, int64_t nq, const float* ref, int32_t nref, int soa, int K,
                          const float scale[3], int32_t* ind, float* dist, cudaStream_t st) {
  const int step = soa ? 1 : 3;
  const int64_t comp = soa ? nref : 1;
  char* buf = nullptr;
  cudaError_t e = scratch_alloc((void**)&buf, knn_grid_scratch_bytes(nref), st);
  if (e != cudaSuccess) return e;
  SaScratch w;
  e = sa_build(q, nq, ref, nref, step, comp, scale, K, buf, &w, st);
  if (e == cudaSuccess) {
    switch (K) {
#define TGMM_TOPK_CASE(KK)                                                              \
  case KK:                                                                              \
    sa_query<KK, true>(q, nq, ref, nref, step, comp, scale, w, ind, dist, st);          \
    break;
      TGMM_TOPK_CASE(1) TGMM_TOPK_CASE(2) TGMM_TOPK_CASE(3) TGMM_TOPK_CASE(4) TGMM_TOPK_CASE(5) TGMM_TOPK_CASE(6)
      TGMM_TOPK_CASE(7) TGMM_TOPK_CASE(8) TGMM_TOPK_CASE(9) TGMM_TOPK_CASE(10) TGMM_TOPK_CASE(11)
#undef TGMM_TOPK_CASE
      default:
        break;
    }
    e = cudaGetLastError();
  }
  const cudaError_t ef = cudaFreeAsync(buf, st);
  return e != cudaSuccess ? e : ef;
}

// The grid kNN on caller-provided scratch (at least knn_grid_scratch_bytes(nref), 256-byte
// aligned); allocates nothing.
cudaError_t knn_grid_in_scratch(const float* q, int64_t nq, const float* ref, int32_t nref, const float scale[3],
                                int32_t* ind, cudaStream_t st, void* scratch) {
  SaScratch w;
  cudaError_t e = sa_build(q, nq, ref, nref, 3, 1, scale, kJ, (char*)scratch, &w, st);
  if (e != cudaSuccess) return e;
  sa_query<kJ, false>(q, nq, ref, nref, 3, 1, scale, w, ind, nullptr, st);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Posterior -> prior on the device (GaussianMixtureModel::updatePriors,
// GaussianMixtureModel.cpp:892-910; N_k = nu_k - nu_o as copyFromGMEM_CUDA/updateNk
// derive it; then nu_k *= 2, W_k /= 2 as mainTrackingGaussianMixtureModel.cpp:961-969).
// kPriorsPerBlock records a block.  The optional alpha total (alpha_k is not written here) is
// the same fixed-order sum in every block, so no block waits for another: a 32-byte sector of
// each record read again per block, against a second launch.  Bound by latency; 5000 records: 76
// us in one block, 9.4 us this way.  Those reads grow with the square of the record count: from
// kPriorsOwnTotal records on one block forms the total and writes alpha_o ahead of the others.
// ---------------------------------------------------------------------------
constexpr int kPriorsPerBlock = 256;
// Every block the total / one block ahead: 20,000 records 28 / 41 us, 40,000 63 / 64, 60,000 85 /
// 87, 100,000 181 / 132, 1 M 13,893 / 1204 (all in one block 14,801).
constexpr int kPriorsOwnTotal = 65536;

// The alpha total of a block of 1024 threads: thread-strided sums in index order, a warp's lanes,
// then the warps.
__device__ __forceinline__ double priors_alpha_total(const TgmmGaussian* gm, int n, double* sh) {
  double a = 0.0;
#pragma unroll 8
  for (int k = threadIdx.x; k < n; k += 1024) a += gm[k].alpha_k;
  a = warp_sum(a);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = a;
  __syncthreads();
  double total = 0.0;
#pragma unroll
  for (int i = 0; i < 32; i++) total += sh[i];
  return total;
}

__global__ void __launch_bounds__(1024) k_priors_alpha(TgmmGaussian* gm, int n, double ap) {
  __shared__ double sh[32];
  const double total = priors_alpha_total(gm, n, sh);
  if (total >= 0.0)
    for (int k = threadIdx.x; k < n; k += 1024) gm[k].alpha_o = total * TGMM_MIN_PI_FOR_DEAD * ap;
}

__global__ void __launch_bounds__(1024) k_update_priors(TgmmGaussian* gm, int n, double bp, double np, double ap,
                                                        double atot, int compute) {
  __shared__ double sh[32];
  if (compute && atot < 0.0) atot = priors_alpha_total(gm, n, sh);
  const int k = blockIdx.x * kPriorsPerBlock + threadIdx.x;
  if (threadIdx.x >= kPriorsPerBlock || k >= n) return;
  TgmmGaussian& g = gm[k];
  const double nu = g.nu_k, Nk = nu - g.nu_o, nuo = fmax(np * Nk, 3.0);
  double m[3], W[6];
#pragma unroll
  for (int d = 0; d < 3; d++) m[d] = g.m_k[d];
#pragma unroll
  for (int e = 0; e < 6; e++) W[e] = g.W_k[e];
#pragma unroll
  for (int d = 0; d < 3; d++) g.m_o[d] = m[d];
  g.beta_o = fmax(bp * Nk, 1e-5);
  g.nu_o = nuo;
#pragma unroll
  for (int e = 0; e < 6; e++) g.W_o[e] = W[e] * nu / nuo;
  if (atot >= 0.0) g.alpha_o = atot * TGMM_MIN_PI_FOR_DEAD * ap;
  g.nu_k = nu * 2.0;
#pragma unroll
  for (int e = 0; e < 6; e++) g.W_k[e] = W[e] / 2.0;
}

cudaError_t update_priors_device(TgmmGaussian* gm, int32_t n, double bp, double np, double ap, double atot,
                                 int compute, cudaStream_t st) {
  if (compute && atot < 0.0 && n >= kPriorsOwnTotal) {
    k_priors_alpha<<<1, 1024, 0, st>>>(gm, n, ap);
    compute = 0;
  }
  k_update_priors<<<(n + kPriorsPerBlock - 1) / kPriorsPerBlock, 1024, 0, st>>>(gm, n, bp, np, ap, atot, compute);
  return cudaGetLastError();
}

}  // namespace tgmm
