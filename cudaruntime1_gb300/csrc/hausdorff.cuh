// hausdorff.cuh -- the directed Hausdorff distance (squared) by a warp,
// shared by the exact kNN refine (pairwise_knn.cu) and the given-candidate
// call (pairwise.cu).
//
// A lane holds up to 8 points of one side in registers; the other side passes
// through shared memory, x and y apart, so that a packed instruction takes
// two points, and each lane keeps its points' minimum squared distances.
// What bounds it is the FP32 pipe: four operations a point pair (two
// differences, a multiply, an FMA; the minima are a half instruction on
// another pipe).
#pragma once
#include "debug_bounds.cuh"
#include "f32x2.cuh"
#include "tsim_internal.cuh"

namespace tsim {
namespace haus {

constexpr int kTargets = 512;  // targets staged at a time, per warp: x, then y
constexpr int kStageFloats = 2 * kTargets;

// points T[t0 .. t0 + len) to the warp's shared memory, padded to a multiple
// of four with the last one
__device__ __forceinline__ void stage_targets(const float2* T, int t0, int len, float* sm) {
  const int lane = threadIdx.x & 31;
  __syncwarp();  // the last targets are used
  for (int j = lane; j < ((len + 3) & ~3); j += 32) {
    const float2 p = __ldg(T + t0 + min(j, len - 1));
    sm[TSIM_SIDX(j, kTargets)] = p.x;
    sm[kTargets + TSIM_SIDX(j, kTargets)] = p.y;
  }
  __syncwarp();
}

// dx^2 + dy^2 of two point pairs: FMA = true one FMA (the kNN path's
// arithmetic), else every operation rounded (the reference CPU's,
// hausdorff.cpp:77-79; the sums are scalar, since a packed product and a packed
// sum come back fused from the assembler)
template <bool FMA>
__device__ __forceinline__ float2 sq2(float2 dx, float2 dy) {
  if (FMA) return fma2(dy, dy, mul2(dx, dx));
  const float2 x = mul2(dx, dx), y = mul2(dy, dy);
  return make_float2(__fadd_rn(x.x, y.x), __fadd_rn(x.y, y.y));
}

// The largest of the minimum squared distances of 32 R points of S to T's;
// lane's point u is S[row(u)] (a row past the end repeats one of the others).
template <bool FMA, int R, class Row>
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
      const float4 X = *reinterpret_cast<const float4*>(sm + TSIM_SIDX(j, kTargets));
      const float4 Y = *reinterpret_cast<const float4*>(sm + kTargets + TSIM_SIDX(j, kTargets));
#pragma unroll
      for (int u = 0; u < R; ++u) {
        const float2 d = sq2<FMA>(sub2(make_float2(X.x, X.y), sx[u]), sub2(make_float2(Y.x, Y.y), sy[u]));
        const float2 e = sq2<FMA>(sub2(make_float2(X.z, X.w), sx[u]), sub2(make_float2(Y.z, Y.w), sy[u]));
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
// only, spread over it.
template <bool FMA>
__device__ float warp_directed(const float2* S, int ns, const float2* T, int nt, float run,
                               float stop, float* sm, bool sample, long long* pairs) {
  const int lane = threadIdx.x & 31;
  if (nt <= kTargets) stage_targets(T, 0, nt, sm);
  if (sample) {
    *pairs += 32ll * nt;
    return fmaxf(run, rows_max_min<FMA, 1>(S, T, nt, sm, [&](int) {
                   return (int)((2 * lane + 1) * (long long)ns >> 6);
                 }));
  }
  for (int base = 0; base < ns;) {
    // as many points a lane as the rest fills
    const int r = (ns - base + 31) >> 5;
    const int take = r >= 8 ? 8 : r >= 4 ? 4 : r >= 2 ? 2 : 1;
    auto row = [&](int u) { return min(base + u * 32 + lane, ns - 1); };
    const float loc = take == 8   ? rows_max_min<FMA, 8>(S, T, nt, sm, row)
                      : take == 4 ? rows_max_min<FMA, 4>(S, T, nt, sm, row)
                      : take == 2 ? rows_max_min<FMA, 2>(S, T, nt, sm, row)
                                  : rows_max_min<FMA, 1>(S, T, nt, sm, row);
    *pairs += (long long)min(32 * take, ns - base) * nt;
    run = fmaxf(run, loc);
    if (run > stop) return run;
    base += 32 * take;
  }
  return run;
}

}  // namespace haus
}  // namespace tsim
