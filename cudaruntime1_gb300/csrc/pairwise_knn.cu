// pairwise_knn.cu -- refine kernels of the exact kNN path for symmetric
// Hausdorff and lock-step Euclidean: one warp per (query, candidate) pair.
//
// Hausdorff (FP32): a lane holds up to 8 points of one side in registers; the
// other side passes through shared memory, x and y apart, so that a packed
// instruction takes two points, and each lane keeps its points' minimum
// squared distances.  The warp maximum is h(Q,C); the reverse direction swaps
// the roles.  What bounds it is the FP32 pipe: four operations a point pair
// (two differences, a multiply, an FMA; the minima are a half instruction on
// another pipe).  A pair whose maximum exceeds the query's threshold is
// abandoned; most pairs of a pruned round are, so with a threshold a sample of
// 32 points of either side, spread over it, is tested first.
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
#include "f32x2.cuh"
#include "tsim_internal.cuh"

namespace tsim {
namespace {

constexpr int kPwThreads = 128;
__device__ __forceinline__ float d2f(float ax, float ay, float bx, float by) {
  const float dx = ax - bx, dy = ay - by;
  return fmaf(dy, dy, dx * dx);
}

constexpr int kTargets = 512;    // targets staged at a time, per warp
constexpr int kSampleMin = 64;   // a side is sampled from this many points on

// points T[t0 .. t0 + len) to shared memory (x, then y), padded to a multiple
// of four with the last one
__device__ __forceinline__ void stage_targets(const float2* T, int t0, int len, float* sm) {
  const int lane = threadIdx.x & 31;
  __syncwarp();  // the last targets are used
  for (int j = lane; j < ((len + 3) & ~3); j += 32) {
    const float2 p = __ldg(T + t0 + min(j, len - 1));
    sm[j] = p.x;
    sm[kTargets + j] = p.y;
  }
  __syncwarp();
}

// The largest of the minimum squared distances of 32 R points of S to T's;
// lane's point u is S[row(u)] (a row past the end repeats one of the others).
template <int R, class Row>
__device__ __forceinline__ float rows_max_min(const float2* S, const float2* T, int nt, float* sm,
                                              Row row) {
  float2 sx[R], sy[R];
  float mn[R];
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const float2 p = __ldg(S + row(u));
    sx[u] = make_float2(p.x, p.x);
    sy[u] = make_float2(p.y, p.y);
    mn[u] = TSIM_INF;
  }
  for (int t0 = 0; t0 < nt; t0 += kTargets) {
    const int len = min(kTargets, nt - t0);
    if (nt > kTargets) stage_targets(T, t0, len, sm);  // else staged by the caller
#pragma unroll 2
    for (int j = 0; j < len; j += 4) {
      const float4 X = *reinterpret_cast<const float4*>(sm + j);
      const float4 Y = *reinterpret_cast<const float4*>(sm + kTargets + j);
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const float2 dx = sub2(make_float2(X.x, X.y), sx[u]), ex = sub2(make_float2(X.z, X.w), sx[u]);
        const float2 dy = sub2(make_float2(Y.x, Y.y), sy[u]), ey = sub2(make_float2(Y.z, Y.w), sy[u]);
        const float2 d = fma2(dy, dy, mul2(dx, dx)), e = fma2(ey, ey, mul2(ex, ex));
        mn[u] = min3f(min3f(mn[u], d.x, d.y), e.x, e.y);
      }
    }
  }
  float loc = mn[0];
#pragma unroll
  for (int u = 1; u < R; ++u) loc = fmaxf(loc, mn[u]);
  for (int o = 16; o; o >>= 1) loc = fmaxf(loc, __shfl_xor_sync(0xffffffffu, loc, o));
  return loc;
}

// max over S of min over T of |s - t|^2 (FP32), at least `run`; stops above
// `stop`.  *pairs grows by the point pairs compared.  sample: 32 points of S
// only.
__device__ float warp_directed(const float2* S, int ns, const float2* T, int nt, float run,
                               float stop, float* sm, bool sample, long long* pairs) {
  const int lane = threadIdx.x & 31;
  if (nt <= kTargets) stage_targets(T, 0, nt, sm);
  if (sample) {
    *pairs += 32ll * nt;
    return fmaxf(run, rows_max_min<1>(S, T, nt, sm, [&](int) {
                   return (int)((2 * lane + 1) * (long long)ns >> 6);
                 }));
  }
  for (int base = 0; base < ns;) {
    // as many points a lane as the rest fills
    const int r = (ns - base + 31) >> 5;
    const int take = r >= 8 ? 8 : r >= 4 ? 4 : r >= 2 ? 2 : 1;
    auto row = [&](int u) { return min(base + u * 32 + lane, ns - 1); };
    const float loc = take == 8   ? rows_max_min<8>(S, T, nt, sm, row)
                      : take == 4 ? rows_max_min<4>(S, T, nt, sm, row)
                      : take == 2 ? rows_max_min<2>(S, T, nt, sm, row)
                                  : rows_max_min<1>(S, T, nt, sm, row);
    *pairs += (long long)min(32 * take, ns - base) * nt;
    run = fmaxf(run, loc);
    if (run > stop) return run;
    base += 32 * take;
  }
  return run;
}

__global__ void __launch_bounds__(kPwThreads) hausdorff_refine_kernel(PwArgs a) {
  __shared__ __align__(16) float targets[kPwThreads / 32][2 * kTargets];
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
      if (sample && n >= kSampleMin) v = warp_directed(Q, n, C, m, v, stop, sm, true, &pairs);
      if (sample && m >= kSampleMin && v <= stop)
        v = warp_directed(C, m, Q, n, v, stop, sm, true, &pairs);
      if (v <= stop) v = warp_directed(Q, n, C, m, v, stop, sm, false, &pairs);
      if (v <= stop) v = warp_directed(C, m, Q, n, v, stop, sm, false, &pairs);
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
