// pairwise.cu -- tiled pairwise-distance reductions: symmetric Hausdorff
// (max-min), lock-step Euclidean (sum), and the bounding-box candidate
// generator that stands in for the reference's Boost R-tree.
#include "debug_bounds.cuh"
#include "hausdorff.cuh"
#include "topk.cuh"
#include "tsim_internal.cuh"

namespace tsim {

namespace {

// One CTA per query, its top_k candidates in two passes (the reference's
// hausdorff_tiled_rtree_kernel takes them in turn, CudaRuntime1/hausdorff.cu:
// 84-122).  First a warp per candidate bounds the symmetric Hausdorff^2 from
// below by 32 points of either side; then the candidate with the smallest
// bound is computed, each direction's points dealt over half of the warps, and
// the others only where their bound is still below the best: a warp per
// candidate, or, where they are fewer than the warps, the whole CTA for each (a
// candidate's long sides on a warp or two left the others idle: 4 queries of
// 8,192 points, two candidates, 24.8 ms, 13.7 on 256 threads a candidate, 6.7
// now).  A lone candidate needs no bound.
// Minima and maxima are exact in any order, so the value is the sequential
// loop's.  Bound by the FP32 pipe (hausdorff.cuh); 1,024 queries of 128
// points, ten candidates: 69 us computing every candidate on 256 threads a
// query, 36 now.
constexpr int kMaxCandSlots = 1024;  // bounds kept in shared memory at a time
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
    hausdorff_cands_kernel(const float2* __restrict__ t1, int n, const float2* __restrict__ t2,
                           int num_t2, int m, const int* __restrict__ cand, int top_k,
                           float* __restrict__ out) {
  constexpr int kWarps = THREADS / 32, kHalf = kWarps / 2;
  __shared__ __align__(16) float targets[kWarps][haus::kStageFloats];
  __shared__ float bound[kMaxCandSlots];
  __shared__ unsigned best_bits;  // of a non-negative float: ordered as unsigned
  __shared__ float part[kWarps];
  __shared__ int first;
  const int q = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* sm = targets[warp];
  const float2* A = t1 + (size_t)q * n;
  long long pairs = 0;
  // the candidate in slot k by the whole CTA: this warp's points of its direction
  auto together = [&](int k, float stop) {
    const float2* B = t2 + (size_t)cand[(size_t)q * top_k + k] * m;
    const bool back = warp >= kHalf;
    const float2 *S = back ? B : A, *D = back ? A : B;
    const int ns = back ? m : n, w = back ? warp - kHalf : warp;
    const int r0 = (int)((long long)w * ns / kHalf), r1 = (int)((long long)(w + 1) * ns / kHalf);
    const float v = r1 > r0 ? haus::warp_directed<false>(S + r0, r1 - r0, D, back ? n : m, 0.0f,
                                                         stop, sm, false, &pairs)
                            : 0.0f;
    if (lane == 0) part[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
      float h = part[0];
#pragma unroll
      for (int i = 1; i < kWarps; ++i) h = fmaxf(h, part[i]);
      best_bits = min(best_bits, __float_as_uint(h));
    }
    __syncthreads();
  };
  if (threadIdx.x == 0) best_bits = __float_as_uint(TSIM_INF);
  for (int k0 = 0; k0 < top_k; k0 += kMaxCandSlots) {
    const int kn = min(kMaxCandSlots, top_k - k0);
    __syncthreads();
    for (int k = warp; k < kn; k += kWarps) {
      const int c = cand[(size_t)q * top_k + k0 + k];
      float v = TSIM_INF;  // out-of-range candidate slots are ignored
      if (c >= 0 && c < num_t2) {
        const float2* B = t2 + (size_t)c * m;
        v = 0.0f;
        if (kn > 1) {
          v = haus::warp_directed<false>(A, n, B, m, 0.0f, TSIM_INF, sm, true, &pairs);
          v = haus::warp_directed<false>(B, m, A, n, v, TSIM_INF, sm, true, &pairs);
        }
      }
      if (lane == 0) bound[k] = v;
    }
    __syncthreads();
    if (warp == 0) {  // the smallest bound
      float b = TSIM_INF;
      int at = -1;
      for (int k = lane; k < kn; k += 32)
        if (bound[k] < b) b = bound[k], at = k;
      for (int o = 16; o; o >>= 1) {
        const float b2 = __shfl_xor_sync(0xffffffffu, b, o);
        const int a2 = __shfl_xor_sync(0xffffffffu, at, o);
        if (a2 >= 0 && (b2 < b || at < 0)) b = b2, at = a2;
      }
      if (lane == 0) first = at;
    }
    __syncthreads();
    const int f = first;
    if (f >= 0 && bound[f] < __uint_as_float(best_bits))  // uniform over the CTA, as below
      together(k0 + f, TSIM_INF);
    if (kn <= kWarps) {
      for (int k = 0; k < kn; ++k) {
        const float best = __uint_as_float(best_bits);
        if (k != f && bound[k] < best) together(k0 + k, best);
      }
      continue;
    }
    for (int k = warp; k < kn; k += kWarps) {
      const float best = __uint_as_float(*(volatile unsigned*)&best_bits);
      if (k == f || !(bound[k] < best)) continue;
      const float2* B = t2 + (size_t)cand[(size_t)q * top_k + k0 + k] * m;
      float v = haus::warp_directed<false>(A, n, B, m, 0.0f, best, sm, false, &pairs);
      if (v < best) v = haus::warp_directed<false>(B, m, A, n, v, best, sm, false, &pairs);
      if (lane == 0) atomicMin(&best_bits, __float_as_uint(v));
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) out[q] = __fsqrt_rn(__uint_as_float(best_bits));
}

// ---- lock-step Euclidean -----------------------------------------------------
constexpr int kEuThreads = 128;

// TwoSum: s + e == a + b exactly (Knuth)
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// Warp per query (the reference's block per query, CudaRuntime1/euclidean.cu:
// 17-73).  First its CSR entries four at a time, 8 lanes each: compensated
// FP32 sums of squared point differences (TwoSum per lane, a compensated
// butterfly over the 8); their order does not matter, since they only pick
// the candidates whose sum lies within its rigorous error margin of the
// smallest.  Those are re-scored in FP64 left to right exactly like
// calc_exact_dist_sq (euclidean.cpp:27-40): the lanes compute 32 terms
// dx^2 + dy^2 at a time, and every lane adds them to the running sum in
// point order; out = (float)sqrt of the best.
__global__ void __launch_bounds__(kEuThreads)
    euclid_cands_kernel(const float2* __restrict__ t1, const float2* __restrict__ t2,
                        const int* __restrict__ cand, const int* __restrict__ off, int num_t, int n,
                        int total, float* __restrict__ s32, float* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q >= num_t) return;
  // clamp caller offsets into [0, total] so a malformed CSR cannot read out of bounds
  const int b = min(max(off[q], 0), total), e = max(min(off[q + 1], total), b);
  const float2* A = t1 + (size_t)q * n;
  const int grp = lane >> 3, gl = lane & 7;
  float mn = TSIM_INF;
  for (int base = b; base < e; base += 4) {
    const int idx = base + grp;
    const int ce = idx < e ? cand[idx] : -1;
    const bool ok = ce >= 0 && ce < num_t;  // out-of-range candidates never win
    const float2* B = t2 + (size_t)(ok ? ce : 0) * n;
    float sum = 0.0f, c = 0.0f;
    for (int i = gl; i < n; i += 8) {
      const float2 p = A[i], r = B[i];
      const float dx = p.x - r.x, dy = p.y - r.y;
      float ns, err;
      two_sum(sum, fmaf(dy, dy, dx * dx), ns, err);
      sum = ns;
      c += err;
    }
    for (int o = 4; o; o >>= 1) {
      const float s2 = __shfl_xor_sync(0xffffffffu, sum, o);
      const float c2 = __shfl_xor_sync(0xffffffffu, c, o);
      float ns, err;
      two_sum(sum, s2, ns, err);
      sum = ns;
      c = c + c2 + err;
    }
    const float tot = ok ? sum + c : TSIM_INF;
    if (gl == 0 && idx < e) s32[idx] = tot;
    mn = fminf(mn, tot);
  }
  for (int o = 16; o >= 8; o >>= 1) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
  __syncwarp();
  // |s32 - exact| <= g * exact with g = 2^-20 (terms 2u, TwoSum chain ~2u,
  // final fold ~2u, n*u^2 negligible for n < 2^20)
  const double g = 1.0 / (1 << 20);
  const double thr = (double)mn * (1.0 + g) / (1.0 - g);
  double best = 1.7976931348623157e308;
  for (int base = b; base < e; base += 32) {
    const int idx = base + lane;
    bool need = false;
    if (idx < e) need = (double)s32[idx] <= thr && cand[idx] >= 0 && cand[idx] < num_t;
    unsigned todo = __ballot_sync(0xffffffffu, need);
    while (todo) {
      const int l = __ffs(todo) - 1;
      todo &= todo - 1;
      const float2* B = t2 + (size_t)cand[base + l] * n;
      double s = 0.0;
      for (int k0 = 0; k0 < n; k0 += 32) {
        double t = 0.0;
        if (k0 + lane < n) {
          const double dx = (double)A[k0 + lane].x - (double)B[k0 + lane].x;
          const double dy = (double)A[k0 + lane].y - (double)B[k0 + lane].y;
          t = __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy));
        }
        const int cnt = min(32, n - k0);
        for (int u = 0; u < cnt; ++u) s = __dadd_rn(s, __shfl_sync(0xffffffffu, t, u));
      }
      best = s < best ? s : best;
    }
  }
  if (lane == 0) out[q] = __double2float_rn(__dsqrt_rn(best));
}

// ---- bounding boxes and box nearest neighbours --------------------------------
__global__ void boxes_kernel(const float2* __restrict__ t, int count, int len,
                             float4* __restrict__ box) {
  const int lane = threadIdx.x & 31;
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= count) return;
  const float2* p = t + (size_t)w * len;
  // sequential min/max semantics do not matter for the value of a min/max
  float x0 = TSIM_INF, y0 = TSIM_INF, x1 = -TSIM_INF, y1 = -TSIM_INF;
  for (int i = lane; i < len; i += 32) {
    float2 v = p[i];
    x0 = fminf(x0, v.x);
    x1 = fmaxf(x1, v.x);
    y0 = fminf(y0, v.y);
    y1 = fmaxf(y1, v.y);
  }
  for (int o = 16; o; o >>= 1) {
    x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
    y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
    y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
  }
  if (lane == 0) box[w] = make_float4(x0, y0, x1, y1);
}

__device__ __forceinline__ float smaxf(float a, float b) { return (a < b) ? b : a; }

__device__ __forceinline__ float box_box_d2(float4 a, float4 b) {
  float dx = smaxf(0.0f, smaxf(__fsub_rn(a.x, b.z), __fsub_rn(b.x, a.z)));
  float dy = smaxf(0.0f, smaxf(__fsub_rn(a.y, b.w), __fsub_rn(b.y, a.w)));
  return __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
}

constexpr int kSelThreads = 256;

__global__ void __launch_bounds__(kSelThreads)
    mbr_knn_kernel(const float4* __restrict__ qbox, const float4* __restrict__ cbox, int num_t2,
                   int k, unsigned long long* __restrict__ gkeys, int* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ SelScratch red;
  const int q = blockIdx.x;
  unsigned long long* keys =
      gkeys ? gkeys + (size_t)q * num_t2 : reinterpret_cast<unsigned long long*>(smem_raw);
  unsigned long long* sel =
      reinterpret_cast<unsigned long long*>(smem_raw + (gkeys ? 0 : (size_t)num_t2 * 8));
  const float4 a = qbox[q];
  for (int j = threadIdx.x; j < num_t2; j += kSelThreads) keys[j] = pack_key(box_box_d2(a, cbox[j]), j);
  __syncthreads();
  block_select_k(keys, num_t2, min(k, num_t2), sel, red);
  const int got = min(k, num_t2);
  for (int e = threadIdx.x; e < k; e += kSelThreads)
    out[(size_t)q * k + e] = e < got ? key_index(sel[e]) : (got > 0 ? key_index(sel[got - 1]) : 0);
}

}  // namespace

int hausdorff_cands(tsim_ctx* ctx, const float2* t1, int num_t1, int n, const float2* t2, int num_t2,
                    int m, const int* cand, int top_k, float* out) {
  TSIM_CHECK_ARG(sizeof(float2) * ((size_t)n + m) <= 200 * 1024,
                 "trajectories too long for the Hausdorff kernel");
  // eight warps a query where four leave the GPU half empty (200 queries of 2,048
  // points, four candidates: 2.3 ms on four, 1.0)
  if (num_t1 <= 2 * ctx->num_sms)
    hausdorff_cands_kernel<256><<<num_t1, 256, 0, ctx->stream>>>(t1, n, t2, num_t2, m, cand, top_k,
                                                                 out);
  else
    hausdorff_cands_kernel<128><<<num_t1, 128, 0, ctx->stream>>>(t1, n, t2, num_t2, m, cand, top_k,
                                                                 out);
  TSIM_CUDA(cudaGetLastError());
  return TSIM_OK;
}

int euclid_cands(tsim_ctx* ctx, const float2* t1, const float2* t2, const int* cand, const int* off,
                 int num_t, int n, int total, float* out) {
  TSIM_TRY(arena_reserve(ctx, align256(sizeof(float) * std::max(total, 1))));
  float* s32 = arena_take<float>(ctx, std::max(total, 1));
  const int warps = kEuThreads / 32;
  euclid_cands_kernel<<<(num_t + warps - 1) / warps, kEuThreads, 0, ctx->stream>>>(
      t1, t2, cand, off, num_t, n, total, s32, out);
  TSIM_CUDA(cudaGetLastError());
  return TSIM_OK;
}

int mbr_knn(tsim_ctx* ctx, const float2* t1, int num_t1, int n, const float2* t2, int num_t2, int m,
            int k, int* out) {
  size_t key_bytes = sizeof(unsigned long long) * (size_t)num_t2;
  bool in_smem = key_bytes + 64 * sizeof(unsigned long long) <= 200 * 1024;
  size_t need = align256(sizeof(float4) * num_t1) + align256(sizeof(float4) * num_t2) +
                (in_smem ? 0 : align256(key_bytes * num_t1) + align256((size_t)k * 4 * num_t1));
  TSIM_TRY(arena_reserve(ctx, need));
  float4* qb = arena_take<float4>(ctx, num_t1);
  float4* cb = arena_take<float4>(ctx, num_t2);
  unsigned long long* gkeys = in_smem ? nullptr : arena_take<unsigned long long>(ctx, (size_t)num_t2 * num_t1);
  boxes_kernel<<<(num_t1 + 3) / 4, 128, 0, ctx->stream>>>(t1, num_t1, n, qb);
  boxes_kernel<<<(num_t2 + 3) / 4, 128, 0, ctx->stream>>>(t2, num_t2, m, cb);
  size_t smem = (in_smem ? key_bytes : 0) + 64 * sizeof(unsigned long long);
  TSIM_CUDA(cudaFuncSetAttribute(mbr_knn_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  mbr_knn_kernel<<<num_t1, kSelThreads, smem, ctx->stream>>>(qb, cb, num_t2, k, gkeys, out);
  TSIM_CUDA(cudaGetLastError());
  return TSIM_OK;
}

}  // namespace tsim

extern "C" {

int tsim_hausdorff_cands(tsim_ctx* ctx, const tsim_point* d_t1, int num_t1, int n,
                         const tsim_point* d_t2, int num_t2, int m, const int* d_cand, int top_k,
                         float* d_out) {
  TSIM_CHECK_ARG(ctx != nullptr, "ctx is NULL");
  TSIM_CHECK_ARG(num_t1 >= 1 && num_t2 >= 1 && n >= 1 && m >= 1 && top_k >= 1, "sizes must be >= 1");
  TSIM_CHECK_ARG(d_t1 && d_t2 && d_cand && d_out, "NULL device pointer");
  TSIM_CUDA(cudaSetDevice(ctx->device));
  return tsim::hausdorff_cands(ctx, (const float2*)d_t1, num_t1, n, (const float2*)d_t2, num_t2, m,
                               d_cand, top_k, d_out);
}

int tsim_euclid_cands(tsim_ctx* ctx, const tsim_point* d_t1, const tsim_point* d_t2,
                      const int* d_cand, const int* d_off, int num_t, int n, int total,
                      float* d_out) {
  TSIM_CHECK_ARG(ctx != nullptr, "ctx is NULL");
  TSIM_CHECK_ARG(num_t >= 1 && n >= 1 && total >= 0, "bad sizes");
  TSIM_CHECK_ARG(d_t1 && d_t2 && d_off && d_out && (total == 0 || d_cand), "NULL device pointer");
  TSIM_CUDA(cudaSetDevice(ctx->device));
  return tsim::euclid_cands(ctx, (const float2*)d_t1, (const float2*)d_t2, d_cand, d_off, num_t, n,
                            total, d_out);
}

int tsim_mbr_knn(tsim_ctx* ctx, const tsim_point* d_t1, int num_t1, int n, const tsim_point* d_t2,
                 int num_t2, int m, int k, int* d_out) {
  TSIM_CHECK_ARG(ctx != nullptr, "ctx is NULL");
  TSIM_CHECK_ARG(num_t1 >= 1 && num_t2 >= 1 && n >= 1 && m >= 1 && k >= 1 && k <= 64,
                 "sizes must be >= 1 and k <= 64");
  TSIM_CHECK_ARG(d_t1 && d_t2 && d_out, "NULL device pointer");
  TSIM_CUDA(cudaSetDevice(ctx->device));
  return tsim::mbr_knn(ctx, (const float2*)d_t1, num_t1, n, (const float2*)d_t2, num_t2, m, k, d_out);
}

}  // extern "C"
