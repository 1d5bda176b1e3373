// pairwise_knn.cu -- refine kernels of the exact kNN path for symmetric
// Hausdorff and lock-step Euclidean: one warp per (query, candidate) pair.
//
// Hausdorff (FP32): the two directions by hausdorff.cuh.  A pair whose maximum
// exceeds the query's threshold is abandoned; most pairs of a pruned round
// are, so with a threshold a sample of 32 points of either side, spread over
// it, is tested first.
// Reference kernel replaced: hausdorff_tiled_rtree_kernel
// (CudaRuntime1/hausdorff.cu:84-122), one CTA per query over 256-point tiles.
//
// Euclidean: lane-strided sum of squared point differences, compensated
// FP32 (TwoSum) for candidates of up to 1024 points, FP64 beyond (the error
// of an uncompensated FP32 sum grows with length).  Reference kernel
// replaced: euclidean_rtree_csr_kernel_global (CudaRuntime1/euclidean.cu:17-73).
//
// FP64 kernels compute the oracle's arithmetic (oracle/oracle.c
// orc_hausdorff64, orc_euclid64) for the pairs the FP32 values cannot order.
#include "dfloat.cuh"
#include "hausdorff.cuh"
#include "tsim_internal.cuh"

namespace tsim {
namespace {

constexpr int kPwThreads = 128;
__device__ __forceinline__ float d2f(float ax, float ay, float bx, float by) {
  const float dx = ax - bx, dy = ay - by;
  return fmaf(dy, dy, dx * dx);
}

constexpr int kSampleMin = 64;  // a side is sampled from this many points on

__global__ void __launch_bounds__(kPwThreads) hausdorff_refine_kernel(PwArgs a) {
  __shared__ __align__(16) float targets[kPwThreads / 32][haus::kStageFloats];
  const int lane = threadIdx.x & 31;
  float* sm = targets[threadIdx.x >> 5];
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const int npairs = a.npairs_dev ? min(*a.npairs_dev, a.npairs) : a.npairs;
  for (int w = gw; w < npairs; w += nw) {
    const int pid = a.order ? a.order[w] : w;
    const int2 pr = a.pairs[pid];
    if (pr.y < 0) continue;
    const int64_t qo = a.qoff[pr.x], co = a.coff[pr.y];
    const int n = (int)(a.qoff[pr.x + 1] - qo), m = (int)(a.coff[pr.y + 1] - co);
    const float2* Q = a.qpts + qo;
    const float2* C = a.cpts + co;
    float v = TSIM_INF;
    long long pairs = 0;
    if (n > 0 && m > 0) {
      const float stop = a.thr ? a.thr[pr.x] : TSIM_INF;
      v = 0.0f;
      const bool sample = stop < TSIM_INF;
      if (sample && n >= kSampleMin) v = haus::warp_directed<true>(Q, n, C, m, v, stop, sm, true, &pairs);
      if (sample && m >= kSampleMin && v <= stop)
        v = haus::warp_directed<true>(C, m, Q, n, v, stop, sm, true, &pairs);
      if (v <= stop) v = haus::warp_directed<true>(Q, n, C, m, v, stop, sm, false, &pairs);
      if (v <= stop) v = haus::warp_directed<true>(C, m, Q, n, v, stop, sm, false, &pairs);
      if (v > stop) v = TSIM_INF;  // abandoned: cannot be among the k best
    }
    if (lane == 0) {
      a.out[pid] = v;
      if (a.cells && pairs) atomicAdd(a.cells, (unsigned long long)pairs);
    }
  }
}

__device__ __forceinline__ void two_sum_acc(float& s, float& c, float t) {
  float ns, e;
  two_sum_f(s, t, ns, e);
  s = ns;
  c += e;
}

// lock-step sum over the candidate's m points against the query's first m
// (+inf when the query is shorter)
__global__ void __launch_bounds__(kPwThreads) euclid_refine_kernel(PwArgs a) {
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const int npairs = a.npairs_dev ? min(*a.npairs_dev, a.npairs) : a.npairs;
  for (int w = gw; w < npairs; w += nw) {
    const int pid = a.order ? a.order[w] : w;
    const int2 pr = a.pairs[pid];
    if (pr.y < 0) continue;
    const int64_t qo = a.qoff[pr.x], co = a.coff[pr.y];
    const int n = (int)(a.qoff[pr.x + 1] - qo), m = (int)(a.coff[pr.y + 1] - co);
    const float2* A = a.qpts + qo;
    const float2* B = a.cpts + co;
    float v = TSIM_INF;
    if (n >= m && m > 0) {
      if (m <= 1024) {
        float s = 0.0f, c = 0.0f;
        for (int i = lane; i < m; i += 32) {
          const float2 p = A[i], r = B[i];
          two_sum_acc(s, c, d2f(p.x, p.y, r.x, r.y));
        }
        for (int o = 16; o; o >>= 1) {
          const float s2 = __shfl_xor_sync(0xffffffffu, s, o);
          const float c2 = __shfl_xor_sync(0xffffffffu, c, o);
          float ns, e;
          two_sum_f(s, s2, ns, e);
          s = ns;
          c = c + c2 + e;
        }
        v = s + c;
      } else {
        double s = 0.0;
        for (int i = lane; i < m; i += 32) {
          const float2 p = A[i], r = B[i];
          const double dx = (double)p.x - (double)r.x, dy = (double)p.y - (double)r.y;
          s += dx * dx + dy * dy;
        }
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        v = __double2float_rn(s);
      }
      const float stop = a.thr ? a.thr[pr.x] : TSIM_INF;
      if (v > stop) v = TSIM_INF;
    }
    if (lane == 0) {
      a.out[pid] = v;
      if (a.cells && n >= m && m > 0) atomicAdd(a.cells, (unsigned long long)m);
    }
  }
}

// ---- FP64 (the oracle's arithmetic) -----------------------------------------
__device__ __forceinline__ double d2_64f(float ax, float ay, float bx, float by) {
  const double dx = (double)ax - (double)bx, dy = (double)ay - (double)by;
  return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
}

__device__ double warp_directed64(const float2* S, int ns, const float2* T, int nt) {
  const int lane = threadIdx.x & 31;
  double run = 0.0;
  for (int i0 = 0; i0 < ns; i0 += 32) {
    const int i = i0 + lane;
    double mn = __longlong_as_double(0x7ff0000000000000ll);
    if (i < ns) {
      const float2 p = S[i];
      for (int j = 0; j < nt; ++j) {
        const float2 t = T[j];
        const double d = d2_64f(p.x, p.y, t.x, t.y);
        mn = d < mn ? d : mn;
      }
    } else {
      mn = 0.0;
    }
    for (int o = 16; o; o >>= 1) {
      const double x = __shfl_xor_sync(0xffffffffu, mn, o);
      mn = x > mn ? x : mn;
    }
    run = mn > run ? mn : run;
  }
  return run;
}

__global__ void __launch_bounds__(kPwThreads) pairwise64_kernel(PwArgs a, int euclid) {
  const int lane = threadIdx.x & 31;
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw = (gridDim.x * blockDim.x) >> 5;
  const int npairs = a.npairs_dev ? min(*a.npairs_dev, a.npairs) : a.npairs;
  for (int wk = gw; wk < npairs; wk += nw) {
    const int w = a.order ? a.order[wk] : wk;
    const int2 pr = a.pairs[w];
    if (pr.y < 0) continue;
    const int64_t qo = a.qoff[pr.x], co = a.coff[pr.y];
    const int n = (int)(a.qoff[pr.x + 1] - qo), m = (int)(a.coff[pr.y + 1] - co);
    const float2* A = a.qpts + qo;
    const float2* B = a.cpts + co;
    double v = __longlong_as_double(0x7ff0000000000000ll);
    if (euclid) {
      if (n >= m && m > 0 && lane == 0) {  // left to right, as the oracle sums
        double s = 0.0;
        for (int i = 0; i < m; ++i) s = __dadd_rn(s, d2_64f(A[i].x, A[i].y, B[i].x, B[i].y));
        v = s;
      }
    } else if (n > 0 && m > 0) {
      const double h1 = warp_directed64(A, n, B, m), h2 = warp_directed64(B, m, A, n);
      v = h1 > h2 ? h1 : h2;
    }
    if (lane == 0) a.out64[w] = v;
  }
}

int launch_pw(tsim_ctx* ctx, void (*kern)(PwArgs), const PwArgs& a) {
  if (a.npairs <= 0) return TSIM_OK;
  int per_sm = 0;
  TSIM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kPwThreads, 0));
  const long long warps = kPwThreads / 32;
  long long blocks = std::min<long long>((a.npairs + warps - 1) / warps,
                                         (long long)std::max(per_sm, 1) * ctx->num_sms);
  kern<<<(unsigned)std::max(blocks, 1ll), kPwThreads, 0, ctx->stream>>>(a);
  TSIM_CUDA(cudaGetLastError());
  launched(ctx);
  return TSIM_OK;
}

}  // namespace

int launch_pairwise(tsim_ctx* ctx, int measure, const PwArgs& a) {
  return launch_pw(ctx, measure == TSIM_HAUSDORFF ? hausdorff_refine_kernel : euclid_refine_kernel,
                   a);
}

int launch_pairwise64(tsim_ctx* ctx, int measure, const PwArgs& a) {
  if (a.npairs <= 0) return TSIM_OK;
  int per_sm = 0;
  TSIM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pairwise64_kernel, kPwThreads, 0));
  const long long warps = kPwThreads / 32;
  long long blocks = std::min<long long>((a.npairs + warps - 1) / warps,
                                         (long long)std::max(per_sm, 1) * ctx->num_sms);
  pairwise64_kernel<<<(unsigned)std::max(blocks, 1ll), kPwThreads, 0, ctx->stream>>>(
      a, measure == TSIM_EUCLIDEAN ? 1 : 0);
  TSIM_CUDA(cudaGetLastError());
  launched(ctx);
  return TSIM_OK;
}

}  // namespace tsim
