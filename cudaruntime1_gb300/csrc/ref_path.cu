// ref_path.cu -- reference-semantics batch path for DTW, LCSS and Frechet.
//
// The reference (CudaRuntime1/dtw.cu:99-234, lcss.cu:114-250,
// frechet.cu:120-253) builds the r=5 query envelopes on the host, computes a
// full num_t x num_t bound matrix on the GPU, copies it back, selects the
// K=10 best candidates per query with partial_sort on the host, copies the
// pair list in again, refines on the GPU and reduces on the host.
//
// Here everything after the H2D copy of the trajectories stays on the device:
//   1. ref_filter_kernel: a CTA per one or two queries builds the envelopes
//      in shared memory, evaluates the bound of every candidate (summed in the
//      same order as the reference CPU code, so values are bit-identical), and
//      selects the K best by (bound, index) without materialising the matrix;
//   2. the strip DP kernel (dp_strip.cu; LCSS: dp_kernels.cu) refines the
//      num_t*K pairs;
//   3. ref_reduce_kernel keeps the best refined value per query.
// Outputs equal the reference's CPU functions (dtw.cpp:14-113,
// lcss.cpp:13-115, frechet.cpp:13-124) bit for bit.
#include "f32x2.cuh"
#include "topk.cuh"
#include "tsim_internal.cuh"

namespace tsim {
namespace {

constexpr int kFilterThreads = 256;
constexpr float kRefBig = 1e20f;  // the reference's infinity (dtw.cpp:23)
constexpr size_t kRefSmemCap = 200 * 1024;

__device__ __forceinline__ float smax(float a, float b) { return (a < b) ? b : a; }
__device__ __forceinline__ float smin(float a, float b) { return (b < a) ? b : a; }

// kind: 0 = DTW (sum of envelope distances), 1 = LCSS (eps-box count,
// descending), 2 = Frechet (max of envelope distances).
//
// A CTA takes TQ queries, a thread one candidate at a time for all of them,
// its points in order (the sums are the reference's, bit for bit).  256
// candidates' points pass through shared memory kRefCols at a time: read
// straight from global memory, each lane walks its own row, every load of a
// warp touches 32 lines and the rows of a CTA do not stay in L1, which set the
// kernel's time (1,024 x 1,024 x 128 points, DTW: 488 us; now 168, bound by
// issue: about 17 instructions a point and query, half of them the square
// root).  Two queries a CTA share the staging where that leaves at least two
// CTAs per SM.
//
// The distances to the envelope, max(0, lo - p, p - hi), take one three-way
// maximum, equal to the reference's comparisons for every input: a NaN on
// either side leaves 0 in both.
constexpr int kRefCols = 8;
constexpr int kRefStride = kFilterThreads + 2;  // 4 banks from one column to the next
constexpr size_t kRefTileBytes = sizeof(float2) * kRefCols * kRefStride;

template <int KIND, int TQ>
__global__ void __launch_bounds__(kFilterThreads)
    ref_filter_kernel(const float2* __restrict__ t1, const float2* __restrict__ t2, int num_t,
                      int n, int m, float eps, int K, unsigned long long* __restrict__ gkeys,
                      int2* __restrict__ pairs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ SelScratch red;
  const int q0 = blockIdx.x * TQ;
  // envelope of query point v*n/m for each candidate position v, as (min_x,
  // min_y, max_x, max_y); LCSS: inflated by eps
  float4* envv = reinterpret_cast<float4*>(smem_raw);  // [TQ][m]
  float2* tile = reinterpret_cast<float2*>(envv + (size_t)TQ * m);
  unsigned long long* skeys = reinterpret_cast<unsigned long long*>(tile + kRefCols * kRefStride);
  const int r = 5;
  for (int x = threadIdx.x; x < TQ * m; x += blockDim.x) {
    const int q = min(q0 + x / m, num_t - 1), v = x % m;
    const float2* A = t1 + (size_t)q * n;
    const int i = (int)(((long long)v * n) / m);
    float min_x = kRefBig, max_x = -kRefBig, min_y = kRefBig, max_y = -kRefBig;
    const int s = max(0, i - r), e = min(n - 1, i + r);
    for (int k = s; k <= e; ++k) {
      float2 p = A[k];
      min_x = smin(min_x, p.x);
      max_x = smax(max_x, p.x);
      min_y = smin(min_y, p.y);
      max_y = smax(max_y, p.y);
    }
    if (KIND == 1) {
      min_x = __fsub_rn(min_x, eps);
      min_y = __fsub_rn(min_y, eps);
      max_x = __fadd_rn(max_x, eps);
      max_y = __fadd_rn(max_y, eps);
    }
    envv[x] = make_float4(min_x, min_y, max_x, max_y);
  }
  const int min_len = min(n, m);
  auto point = [&](const float4 e, const float2 p, float& acc) {
    if (KIND == 1) {
      if (p.x > e.x && p.x < e.z && p.y > e.y && p.y < e.w) acc += 1.0f;  // exact: below 2^24
    } else {
      const float2 lo = sub2(make_float2(e.x, e.y), p), hi = sub2(p, make_float2(e.z, e.w));
      const float2 d = make_float2(max3f(lo.x, hi.x, 0.0f), max3f(lo.y, hi.y, 0.0f));
      const float2 dd = mul2(d, d);
      const float dist = __fsqrt_rn(__fadd_rn(dd.x, dd.y));
      acc = KIND == 0 ? __fadd_rn(acc, dist) : fmaxf(acc, dist);
    }
  };
  for (int c0 = 0; c0 < num_t; c0 += kFilterThreads) {
    float2 pre[kRefCols];  // the next columns, in flight while these are used
    auto fetch = [&](int v0) {
#pragma unroll
      for (int i = 0; i < kRefCols; ++i) {
        const int x = i * kFilterThreads + threadIdx.x;
        const int j = c0 + x / kRefCols, v = v0 + x % kRefCols;
        if (j < num_t && v < m) pre[i] = __ldg(t2 + (size_t)j * m + v);
      }
    };
    float acc[TQ];
#pragma unroll
    for (int t = 0; t < TQ; ++t) acc[t] = 0.0f;
    fetch(0);
    for (int v0 = 0; v0 < m; v0 += kRefCols) {
      __syncthreads();  // the last columns are used (the first time: the envelopes are written)
#pragma unroll
      for (int i = 0; i < kRefCols; ++i) {
        const int x = i * kFilterThreads + threadIdx.x;
        tile[(x % kRefCols) * kRefStride + x / kRefCols] = pre[i];
      }
      __syncthreads();
      if (v0 + kRefCols < m) fetch(v0 + kRefCols);
      if (v0 + kRefCols <= m) {
#pragma unroll
        for (int u = 0; u < kRefCols; ++u) {
          const float2 p = tile[u * kRefStride + threadIdx.x];
#pragma unroll
          for (int t = 0; t < TQ; ++t) point(envv[t * m + v0 + u], p, acc[t]);
        }
      } else {
        for (int u = 0; v0 + u < m; ++u) {
          const float2 p = tile[u * kRefStride + threadIdx.x];
#pragma unroll
          for (int t = 0; t < TQ; ++t) point(envv[t * m + v0 + u], p, acc[t]);
        }
      }
    }
    const int j = c0 + threadIdx.x;
    if (j < num_t) {
#pragma unroll
      for (int t = 0; t < TQ; ++t) {
        if (q0 + t >= num_t) break;
        unsigned long long* keys = gkeys ? gkeys + (size_t)(q0 + t) * num_t : skeys + (size_t)t * num_t;
        // LCSS: descending ub -> ascending key
        keys[j] = pack_key(KIND == 1 ? -__fdiv_rn(acc[t], (float)min_len) : acc[t], j);
      }
    }
  }
  __syncthreads();
  __shared__ unsigned long long sel[64];
#pragma unroll 1
  for (int t = 0; t < TQ && q0 + t < num_t; ++t) {
    const unsigned long long* keys =
        gkeys ? gkeys + (size_t)(q0 + t) * num_t : skeys + (size_t)t * num_t;
    block_select_k(keys, num_t, K, sel, red);
    for (int k = threadIdx.x; k < K; k += blockDim.x)
      pairs[(size_t)(q0 + t) * K + k] = make_int2(q0 + t, key_index(sel[k]));
    __syncthreads();
  }
}

// kind 0/2: min of refined distances; 1: max of count / min(n, m).
template <int KIND>
__global__ void ref_reduce_kernel(const float* __restrict__ vals, int num_t, int K, int n, int m,
                                  float* __restrict__ out) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= num_t) return;
  if (KIND == 1) {
    float best = -1.0f;
    const int min_len = min(n, m);
    for (int k = 0; k < K; ++k) {
      float sim = __fdiv_rn(vals[(size_t)q * K + k], (float)min_len);
      if (sim > best) best = sim;
    }
    out[q] = best;
  } else {
    float best = kRefBig;
    for (int k = 0; k < K; ++k) {
      float v = vals[(size_t)q * K + k];
      if (v < best) best = v;
    }
    out[q] = best;
  }
}

__global__ void fixed_offsets_kernel(int64_t* off1, int len1, int64_t* off2, int len2, int count) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i <= count) {
    off1[i] = (int64_t)i * len1;
    off2[i] = (int64_t)i * len2;
  }
}

}  // namespace

// Scratch of one reference-semantics batch call, carved from one block.
size_t ref_scratch_bytes(int num_t, int m, bool* keys_in_smem) {
  const int K = std::min(10, num_t);
  const size_t env_bytes = (size_t)m * sizeof(float4);
  const size_t key_bytes = (size_t)num_t * sizeof(unsigned long long);
  const bool in_smem = env_bytes + key_bytes <= kRefSmemCap;
  if (keys_in_smem) *keys_in_smem = in_smem;
  return align256(sizeof(int2) * num_t * K) + align256(sizeof(float) * num_t * K) +
         2 * align256(sizeof(int64_t) * (num_t + 1)) + (in_smem ? 0 : align256(key_bytes * num_t));
}

int ref_batch_core(tsim_ctx* ctx, int measure, const float2* d_t1, const float2* d_t2, int num_t,
                   int n, int m, float eps, float* d_out, char* scratch) {
  const int K = std::min(10, num_t);
  // shared memory: m envelopes + keys when they fit, else keys in scratch
  const size_t env_bytes = (size_t)m * sizeof(float4);
  const size_t key_bytes = (size_t)num_t * sizeof(unsigned long long);
  TSIM_CHECK_ARG(env_bytes <= kRefSmemCap, "candidate length too large for the envelope filter");
  bool keys_in_smem = false;
  ref_scratch_bytes(num_t, m, &keys_in_smem);
  char* p = scratch;
  auto take = [&p](size_t bytes) {
    char* q = p;
    p += align256(bytes);
    return q;
  };
  int2* pairs = reinterpret_cast<int2*>(take(sizeof(int2) * num_t * K));
  float* vals = reinterpret_cast<float*>(take(sizeof(float) * num_t * K));
  int64_t* qoff = reinterpret_cast<int64_t*>(take(sizeof(int64_t) * (num_t + 1)));
  int64_t* coff = reinterpret_cast<int64_t*>(take(sizeof(int64_t) * (num_t + 1)));
  unsigned long long* gkeys =
      keys_in_smem ? nullptr : reinterpret_cast<unsigned long long*>(take(key_bytes * num_t));

  stage_begin(ctx, TSIM_STAGE_REF);
  // two queries a CTA where two CTAs per SM are left and their keys fit
  const size_t one = env_bytes + (keys_in_smem ? key_bytes : 0);
  const int tq = num_t >= 4 * ctx->num_sms && 2 * one + kRefTileBytes <= 100 * 1024 ? 2 : 1;
  const size_t smem = tq * one + kRefTileBytes;
  auto launch_filter = [&](auto kern) -> int {
    TSIM_CUDA(allow_dynamic_smem(kern, smem));
    kern<<<(num_t + tq - 1) / tq, kFilterThreads, smem, ctx->stream>>>(d_t1, d_t2, num_t, n, m, eps,
                                                                       K, gkeys, pairs);
    TSIM_CUDA(cudaGetLastError());
    launched(ctx);
    return TSIM_OK;
  };
  int kind;
  if (measure == TSIM_DTW) {
    TSIM_TRY(tq == 2 ? launch_filter(ref_filter_kernel<0, 2>) : launch_filter(ref_filter_kernel<0, 1>));
    kind = DP_DTW_REF;
  } else if (measure == TSIM_LCSS) {
    TSIM_TRY(tq == 2 ? launch_filter(ref_filter_kernel<1, 2>) : launch_filter(ref_filter_kernel<1, 1>));
    kind = DP_LCSS;
  } else {
    TSIM_TRY(tq == 2 ? launch_filter(ref_filter_kernel<2, 2>) : launch_filter(ref_filter_kernel<2, 1>));
    kind = DP_FRECHET_REF;
  }
  fixed_offsets_kernel<<<(num_t + 256) / 256, 256, 0, ctx->stream>>>(qoff, n, coff, m, num_t);
  TSIM_CUDA(cudaGetLastError());
  launched(ctx);

  DpArgs a{};
  a.qpts = d_t1;
  a.qoff = qoff;
  a.cpts = d_t2;
  a.coff = coff;
  a.pairs = pairs;
  a.npairs = num_t * K;
  a.out = vals;
  a.thr = nullptr;
  a.band_pct = -1;
  a.delta = -1;
  a.eps = eps;
  a.max_n = n;
  // The reference's square roots make a lone warp's step long, and a strip's
  // time hardly depends on the warps beside it: one pair more than the SMs hold
  // doubles the launch.  Round-striped, whose pairs stage no points, from there
  // on: where an SM holds eight pairs for any number (2,440 pairs of 2,040 points
  // 10.9 ms, 17.8 on strips, 3,700 of them 18.6 and 24.2; 1,000 7.8 and 6.3), else
  // as long as it does not take turns itself (of 1,000 points 2,440 2.8 ms and 3.3,
  // 3,300 4.4 and 3.6).
  const int held = strip_pairs_per_sm(n, m);
  const bool turns = a.npairs > held * ctx->num_sms && std::max(n, m) <= strip_max_cols() &&
                     (held <= 8 || a.npairs <= 20 * ctx->num_sms);
  if (strip_kind(kind) && turns) {
    TSIM_TRY(launch_dp(ctx, kind, 32, 8, a, m));
  } else if (strip_kind(kind) && std::min(n, m) <= strip_max_cols()) {
    TSIM_TRY(launch_dp_strip(ctx, kind, a, n, m, nullptr, nullptr));
  } else {
    int G, R;
    dp_shape(kind, n, m, -1, G, R);
    TSIM_TRY(launch_dp(ctx, kind, G, R, a, m));
  }

  const int tb = 128;
  if (measure == TSIM_LCSS)
    ref_reduce_kernel<1><<<(num_t + tb - 1) / tb, tb, 0, ctx->stream>>>(vals, num_t, K, n, m, d_out);
  else
    ref_reduce_kernel<0><<<(num_t + tb - 1) / tb, tb, 0, ctx->stream>>>(vals, num_t, K, n, m, d_out);
  TSIM_CUDA(cudaGetLastError());
  launched(ctx);
  stage_end(ctx);
  return TSIM_OK;
}

int ref_batch(tsim_ctx* ctx, int measure, const float2* d_t1, const float2* d_t2, int num_t, int n,
              int m, float eps, float* d_out) {
  TSIM_TRY(arena_reserve(ctx, ref_scratch_bytes(num_t, m, nullptr)));
  char* scratch = arena_take<char>(ctx, ref_scratch_bytes(num_t, m, nullptr));
  return ref_batch_core(ctx, measure, d_t1, d_t2, num_t, n, m, eps, d_out, scratch);
}

}  // namespace tsim

extern "C" int tsim_ref_batch(tsim_ctx* ctx, int measure, const tsim_point* d_t1,
                              const tsim_point* d_t2, int num_t, int n, int m, float epsilon,
                              float* d_out) {
  TSIM_CHECK_ARG(ctx != nullptr, "ctx is NULL");
  TSIM_CHECK_ARG(measure == TSIM_DTW || measure == TSIM_LCSS || measure == TSIM_FRECHET,
                 "measure must be DTW, LCSS or Frechet");
  TSIM_CHECK_ARG(num_t >= 1 && n >= 1 && m >= 1, "num_t, n and m must be >= 1");
  TSIM_CHECK_ARG(d_t1 && d_t2 && d_out, "NULL device pointer");
  TSIM_CUDA(cudaSetDevice(ctx->device));
  return tsim::ref_batch(ctx, measure, reinterpret_cast<const float2*>(d_t1),
                         reinterpret_cast<const float2*>(d_t2), num_t, n, m, epsilon, d_out);
}
