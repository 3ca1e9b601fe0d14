// local_ll.cu -- the local log-likelihood of supervoxel lists: the likelihood the split
// round compares before and after a proposed cell division (calculateLocalLikelihood,
// UtilsCUDA/GMEMupdateCUDA.h:120, body GMEMupdateCUDA.cu:2952-3055, over
// addLocalLikelihoodWithSupervoxels :2876-2949 and the kernel
// GMEMcomputeLocalLikelihoodKernelWithSupervoxels :1989-2103).
//
// For each list and each supervoxel s in it (a supervoxel listed twice counts twice), with
// s's five candidates ind[j*n_sv+s] and the given Gaussians, each voxel's density is
//   sum_j sqrt(det W_j nu_j^3)/(2 pi)^{3/2} exp(-nu_j d'W_j d/2) alpha_j/A,  d = x - m_j,
// A the sum of alpha over every Gaussian, all in FP64 as the reference evaluates it.  The
// supervoxel's value keeps the reference's per-thread overwrite: of the voxels v = t + 1024 i
// (t < 1024, relative to s's first voxel) only the last one with a positive density adds
// I_v ln(density_v).  The reference then sums in float (a block tree per supervoxel, a
// power-of-two pass over the list, a double sum of the blocks on the host); here every sum
// is FP64 in a fixed order: a block's threads, its warps, then the supervoxels in list order.
//
// Launches: k_local_alpha (one block: A), k_local_items (a block per listed supervoxel),
// k_local_lists (a thread per list).
#include <cuda_runtime.h>

#include <string.h>

#include <algorithm>
#include <vector>

#include "tgmm_internal.cuh"

namespace tgmm {
namespace {

constexpr double kTwoPi15 = 15.749609945722419;  // (2 pi)^(3/2)
constexpr int kLocalThreads = 256;               // threads per listed supervoxel

__device__ __forceinline__ double det_sym3(const double* w) {
  return w[0] * (w[3] * w[5] - w[4] * w[4]) - w[1] * (w[1] * w[5] - w[2] * w[4]) +
         w[2] * (w[1] * w[4] - w[2] * w[3]);
}

// A = sum of alpha_k in FP64: thread-strided partials in index order (eight loads in flight),
// a warp's lanes, then the warps.  Also clears the call's flag.
__global__ void __launch_bounds__(1024) k_local_alpha(const TgmmGaussian* gm, int n, double* out, int* bad) {
  __shared__ double sh[32];
  double s = 0.0;
#pragma unroll 8
  for (int k = threadIdx.x; k < n; k += 1024) s += gm[k].alpha_k;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double a = 0.0;
#pragma unroll
    for (int i = 0; i < 32; i++) a += sh[i];
    *out = a;
    *bad = 0;
  }
}

struct LocalCand {
  double m[3];
  double W[6];
  double nu, c;  // c = sqrt(det W nu^3)/(2 pi)^{3/2} * alpha/A
};

__device__ __forceinline__ double local_density(const LocalCand* C, float x0, float x1, float x2) {
  double acc = 0.0;
#pragma unroll
  for (int j = 0; j < kJ; j++) {
    const double* W = C[j].W;
    const double d0 = (double)x0 - C[j].m[0], d1 = (double)x1 - C[j].m[1], d2 = (double)x2 - C[j].m[2];
    const double maha = C[j].nu * (W[0] * d0 * d0 + W[3] * d1 * d1 + W[5] * d2 * d2 + 2.0 * W[1] * d0 * d1 +
                                   2.0 * W[2] * d0 * d2 + 2.0 * W[4] * d1 * d2);
    acc += C[j].c * exp(-0.5 * maha);
  }
  return acc;
}

// Block per listed supervoxel (item p of the flattened lists): its local log-likelihood into
// item_ll[p].  Thread t handles the reference's threads t, t + 256, ... < min(n, 1024): the last
// voxel of each one's stride, walking back a stride at a time past zero densities.  Bound by
// each voxel's chain of FP64 exponentials: a warp per supervoxel gave every lane some twenty
// voxels one after the other while most of the device stood idle (400 supervoxels of ~720
// voxels: the call's device work 56 -> 30 us with a block each).
__global__ void __launch_bounds__(kLocalThreads) k_local_items(const float* __restrict__ query,
                                                               const float* __restrict__ img,
                                                               const int64_t* __restrict__ lptr, int64_t n_vox,
                                                               int n_sv, const int32_t* __restrict__ ind,
                                                               const TgmmGaussian* __restrict__ gm, int n_gauss,
                                                               const int32_t* __restrict__ list_idx,
                                                               const double* alpha_total, double* item_ll,
                                                               int* bad) {
  __shared__ LocalCand C[kJ];
  __shared__ double s_sum[kLocalThreads / 32];
  const int p = blockIdx.x, lane = threadIdx.x & 31;
  const int s = list_idx[p];
  const int64_t a = lptr[s], b = lptr[s + 1];
  int ok = 1;
  if (threadIdx.x < kJ) {
    const int j = threadIdx.x, k = ind[(int64_t)j * n_sv + s];
    if (k < 0 || k >= n_gauss) {
      ok = 0;
    } else {
      const TgmmGaussian& g = gm[k];
      for (int d = 0; d < 3; d++) C[j].m[d] = g.m_k[d];
      for (int e = 0; e < 6; e++) C[j].W[e] = g.W_k[e];
      C[j].nu = g.nu_k;
      const double c = sqrt(det_sym3(g.W_k) * pow(g.nu_k, 3.0)) / kTwoPi15;
      C[j].c = c * (g.alpha_k / *alpha_total);
    }
  }
  if (!__syncthreads_and(ok)) {
    if (threadIdx.x == 0) {
      atomicOr(bad, 1);
      item_ll[p] = 0.0;
    }
    return;
  }
  const int64_t n = b - a;
  double acc = 0.0;
  for (int64_t t = threadIdx.x; t < (n < 1024 ? n : 1024); t += kLocalThreads) {
    for (int64_t v = a + t + ((n - 1 - t) / 1024) * 1024; v >= a; v -= 1024) {
      const double dens = local_density(C, query[v], query[n_vox + v], query[2 * n_vox + v]);
      if (dens > 0.0) {
        acc += (double)img[v] * log(dens);
        break;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) s_sum[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double sum = 0.0;
    for (int i = 0; i < kLocalThreads / 32; i++) sum += s_sum[i];
    item_ll[p] = sum;
  }
}

__global__ void k_local_lists(const int32_t* list_ptr, int n_lists, const double* item_ll, double* ll) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_lists) return;
  double s = 0.0;
  for (int p = list_ptr[i]; p < list_ptr[i + 1]; p++) s += item_ll[p];
  ll[i] = s;
}

}  // namespace
}  // namespace tgmm

extern "C" int tgmm_local_likelihood(const TgmmFrame* frame, const int32_t* ind_dev, const TgmmGaussian* gm_dev,
                                     int32_t n_gauss, const int32_t* list_ptr, const int32_t* list_idx,
                                     int32_t n_lists, double* ll_out, void* stream) {
  using namespace tgmm;
  if (!frame || !ind_dev || !gm_dev || !list_ptr || !ll_out || n_lists < 0 || n_gauss < TGMM_J)
    return report_error(TGMM_ERR_INVALID_ARG, "tgmm_local_likelihood: null argument or fewer than 5 Gaussians",
                        cudaSuccess);
  if (!frame->query || !frame->img || !frame->label_ptr || frame->n_sv < 1 || frame->n_vox < 0)
    return report_error(TGMM_ERR_INVALID_ARG, "tgmm_local_likelihood: bad frame", cudaSuccess);
  if (n_lists == 0) return TGMM_OK;
  if (list_ptr[0] != 0) return report_error(TGMM_ERR_INVALID_ARG, "tgmm_local_likelihood: list_ptr[0] != 0", cudaSuccess);
  for (int32_t i = 0; i < n_lists; i++)
    if (list_ptr[i + 1] < list_ptr[i])
      return report_error(TGMM_ERR_INVALID_ARG, "tgmm_local_likelihood: list_ptr not monotone", cudaSuccess);
  const int32_t n_items = list_ptr[n_lists];
  if (n_items > 0 && !list_idx) return report_error(TGMM_ERR_INVALID_ARG, "tgmm_local_likelihood: null list_idx", cudaSuccess);
  for (int32_t p = 0; p < n_items; p++)
    if (list_idx[p] < 0 || list_idx[p] >= frame->n_sv)
      return report_error(TGMM_ERR_INVALID_ARG, "tgmm_local_likelihood: supervoxel index out of range", cudaSuccess);
  cudaStream_t st = (cudaStream_t)stream;
  // one stream-ordered scratch: lists (ptr, idx; one upload), per-item values, A, and, read back
  // together, the per-list values and a flag
  const size_t n_up = (size_t)n_lists + 1 + (size_t)n_items;
  const size_t o_item = (4 * n_up + 7) / 8 * 8;
  const size_t o_a = o_item + 8 * (size_t)(n_items > 0 ? n_items : 1);
  const size_t o_ll = o_a + 8, total = o_ll + 8 * ((size_t)n_lists + 1);
  char* buf = nullptr;
  cudaError_t e = scratch_alloc((void**)&buf, total, st);
  if (e != cudaSuccess) return report_error(TGMM_ERR_OOM, "tgmm_local_likelihood: scratch", e);
  int32_t* d_ptr = (int32_t*)buf;
  int32_t* d_idx = d_ptr + n_lists + 1;
  double* d_item = (double*)(buf + o_item);
  double* d_a = (double*)(buf + o_a);
  double* d_ll = (double*)(buf + o_ll);
  int* d_bad = (int*)(d_ll + n_lists);
  std::vector<int32_t> up(n_up);
  std::copy(list_ptr, list_ptr + n_lists + 1, up.begin());
  std::copy(list_idx, list_idx + n_items, up.begin() + n_lists + 1);
  std::vector<double> down((size_t)n_lists + 1);
  e = cudaMemcpyAsync(d_ptr, up.data(), 4 * n_up, cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    k_local_alpha<<<1, 1024, 0, st>>>(gm_dev, n_gauss, d_a, d_bad);
    if (n_items > 0)
      k_local_items<<<n_items, kLocalThreads, 0, st>>>(frame->query, frame->img, frame->label_ptr, frame->n_vox,
                                                       frame->n_sv, ind_dev, gm_dev, n_gauss, d_idx, d_a, d_item,
                                                       d_bad);
    k_local_lists<<<(n_lists + 255) / 256, 256, 0, st>>>(d_ptr, n_lists, d_item, d_ll);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(down.data(), d_ll, 8 * ((size_t)n_lists + 1), cudaMemcpyDeviceToHost, st);
  cudaError_t ef = cudaFreeAsync(buf, st);
  if (e == cudaSuccess) e = ef;
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return report_error(TGMM_ERR_CUDA, "tgmm_local_likelihood", e);
  int bad = 0;
  memcpy(&bad, &down[n_lists], sizeof(bad));
  if (bad) return report_error(TGMM_ERR_INVALID_ARG, "tgmm_local_likelihood: a candidate index is out of range", cudaSuccess);
  std::copy(down.begin(), down.begin() + n_lists, ll_out);
  return TGMM_OK;
}
