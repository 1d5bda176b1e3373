// dp_strip.cu -- full-matrix DP (no band): a warp per (query, candidate)
// pair, the pair's rows in strips of 32 R, lane l holding rows l R .. l R + R
// - 1 of the strip in registers.  At step s lane l computes column s - l of
// its R rows, top to bottom; the row above comes from the lane above by one
// shuffle (its bottom row, one step earlier).  A strip of r rows and c
// columns takes c + 31 steps, so a step's fixed work (one inner point from
// shared memory, the shuffle, the loop) is shared by R cells, and no cell is
// masked: the inner trajectory is staged with points at infinity on both
// sides, whose cells cost +inf, which is what the cells outside the matrix
// must hold.  Strips of one pair are joined by a shared-memory row (the last
// lane's bottom row, read by the first lane of the next strip).
//
// Rows and columns are whichever side makes the pair cheaper (the measures
// are symmetric under the transpose and a minimum of three values is exact
// in any order, so values are the same bits as the other kernels').
//
// What bounds it: FP32 and ALU issue -- five instructions a cell (a packed
// subtraction, multiply, FMA, three-operand minimum, add) and about twelve a
// step, so R is as large as the pair's rows fill (8 for 4-byte values).
// 131,072 DTW pairs of 128 x 128 points: 0.62 ms, 3,450 GCUPS (1,610 on a
// lane per pair), 27.6 of the FP32 probe's 77 TFLOP/s at 8 flops a cell.
//
// Early abandon: every warping path crosses the frontier of the cells done
// so far -- each lane's current column, the value it received from the lane
// above last, and (with strips still to come) any cell of the strip's bottom
// row -- and values never decrease along a path, so a frontier whose
// smallest value exceeds the threshold ends the pair.  Tested every 16 steps
// of the first strip and after every strip.
//
// Reference kernels replaced: dtw_refine_kernel (CudaRuntime1/dtw.cu:41-96)
// and frechet_refine_kernel_m (CudaRuntime1/frechet.cu:44-117).
#include <type_traits>

#include "debug_bounds.cuh"
#include "dp_policies.cuh"

namespace tsim {
namespace {
using namespace dp;

constexpr int kStripThreads = 128;
constexpr int kStripPad = 32;       // staged points at infinity on each side
constexpr int kStripMaxCols = 2048;  // longest inner trajectory

// rows per lane of the widest strip: 8 for 4-byte values, 4 for pairs and
// 64-bit ones (registers)
template <class P>
constexpr int strip_rmax() {
  return sizeof(typename P::V) > 4 ? 4 : 8;
}

// Policies whose cost takes a square root test whether the lane's column is
// inside the matrix instead: the square root of an infinite cost leaves the
// fast path, for the whole warp, on every step that has a lane outside.
// Compensated Frechet too: a pair's cost at infinity is no number, and among
// three cells that are none (a point at infinity on the matrix's edge) the
// maximum passes over them.
template <class P>
constexpr bool strip_guard() {
  return std::is_same<P, PolDtwRef>::value || std::is_same<P, PolFrechetRef>::value ||
         std::is_same<P, PolDtwEu>::value || std::is_same<P, PolDtwEuC>::value ||
         std::is_same<P, PolFrechetSqC>::value;
}

// a cell from packed points where the policy has that form
template <class P, class V>
__device__ __forceinline__ auto strip_cell(float2 q, float2 c, V up, V lf, V dg, float aux, int)
    -> decltype(P::cellp(q, c, up, lf, dg, aux)) {
  return P::cellp(q, c, up, lf, dg, aux);
}
template <class P, class V>
__device__ __forceinline__ V strip_cell(float2 q, float2 c, V up, V lf, V dg, float aux, long) {
  return P::cell(q.x, q.y, c.x, c.y, up, lf, dg, aux);
}

template <class V>
__device__ __forceinline__ V shfl_above(V v) {
  return __shfl_up_sync(0xffffffffu, v, 1);
}
__device__ __forceinline__ df shfl_above(df v) {
  return df{__shfl_up_sync(0xffffffffu, v.hi, 1), __shfl_up_sync(0xffffffffu, v.lo, 1)};
}

// issue slots of a pair with `rows` outer rows: strips x steps x step cost
__device__ __forceinline__ int strip_cost(int rows, int cols, int rmax, int& R) {
  R = 2;
  while (R < rmax && rows > 32 * R) R *= 2;
  const int strips = (rows + 32 * R - 1) / (32 * R);
  return strips * (cols + 31) * (6 * R + 12);
}

#define PT(j) pts[TSIM_SIDX((j) + kStripPad, cap + 2 * kStripPad)]
#define ROWBUF(j) buf[TSIM_SIDX((j) + kStripPad, bufcap)]

// One pair on the warp.  MULTI: rows in several strips.
template <class P, int R, bool MULTI>
__device__ __forceinline__ void strip_pair(const DpArgs& a, const int pid, const float2* O,
                                           const int rows, const int cols, const float thr,
                                           const float aux, const float2* pts,
                                           typename P::V* buf, const int cap, const int bufcap) {
  using V = typename P::V;
  const int lane = threadIdx.x & 31;
  const int nstrips = MULTI ? (rows + 32 * R - 1) / (32 * R) : 1;
  const bool check = a.thr != nullptr;
  if (MULTI) {  // the row above the matrix: D(-1,-1) = origin, +inf elsewhere
    for (int j = lane - kStripPad; j < cols + kStripPad; j += 32)
      ROWBUF(j) = j == -1 ? P::origin() : P::border();
    __syncwarp();
  }
  bool alive = true;
  long long cells = 0;
  V left[R];
  int lres = 0;
  for (int st = 0; st < nstrips; ++st) {
    const int r0 = st * 32 * R;
    const bool last = st == nstrips - 1;
    float2 o[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      o[k] = __ldg(O + min(r0 + lane * R + k, rows - 1));  // rows past the end: never used
      left[k] = P::border();
    }
    V prev_up = lane == 0 ? (MULTI ? ROWBUF(-1) : P::origin()) : P::border();
    V bottom = P::border();
    float bmin = TSIM_INF;  // MULTI: smallest value of this lane's bottom row
    if (last) lres = (rows - 1 - r0) / R;
    const int nsteps = cols + (last ? lres : 31);
    auto step = [&](const int s) __attribute__((always_inline)) {
      const float2 c = PT(s - lane);
      const V sh = shfl_above(bottom);
      const V above = MULTI ? ROWBUF(s) : P::border();
      const V upv = lane == 0 ? above : sh;
      if (!strip_guard<P>() || (unsigned)(s - lane) < (unsigned)cols) {
        V up = upv, dg = prev_up;
#pragma unroll
        for (int k = 0; k < R; ++k) {
          const V lf = left[k];
          up = strip_cell<P>(o[k], c, up, lf, dg, aux, 0);
          dg = lf;
          left[k] = up;
        }
        bottom = up;
      }
      prev_up = upv;
      if (MULTI) {
        bmin = fminf(bmin, vf(bottom));
        if (lane == 31) ROWBUF(s - 31) = bottom;
      }
    };
    // the odd steps first, then straight-line blocks of 8
    int s = 0;
    for (; s < (nsteps & 7); ++s) step(s);
    for (; s < nsteps; s += 8) {
#pragma unroll
      for (int u = 0; u < 8; ++u) step(s + u);
      if (check && st == 0 && (s & 8)) {
        float mn = fminf(vf(prev_up), MULTI && lane == 31 ? bmin : TSIM_INF);
#pragma unroll
        for (int k = 0; k < R; ++k) mn = fminf(mn, vf(left[k]));
        if (__uint_as_float(__reduce_min_sync(0xffffffffu, __float_as_uint(mn))) > thr) {
          alive = false;
          s += 8;
          break;
        }
      }
    }
    if (MULTI) {
      __syncwarp();  // the strip's bottom row is written before the next strip reads it
      if (check && alive && !last && __shfl_sync(0xffffffffu, bmin, 31) > thr) alive = false;
    }
    if (a.cells) {  // this lane's rows and columns of the strip
      const int nr = min(max(rows - (r0 + lane * R), 0), R);
      cells += (long long)nr * min(max(s - lane, 0), cols);
    }
    if (!alive) break;
  }
  if (a.cells) {
    for (int o = 16; o; o >>= 1) cells += __shfl_xor_sync(0xffffffffu, cells, o);
    if (lane == 0) atomicAdd(a.cells, (unsigned long long)cells);
  }
  if (!alive) {
    if (lane == 0) store_result(a, pid, P::border());
  } else if (lane == lres) {  // the last row's value after its last column
    V r = left[0];
#pragma unroll
    for (int k = 1; k < R; ++k)
      if ((rows - 1) % R == k) r = left[k];
    store_result(a, pid, r);
  }
}

template <class P>
__global__ void __launch_bounds__(kStripThreads)
    dp_strip_kernel(DpArgs a, int cap, int multi, int* spill, int* nspill) {
  using V = typename P::V;
  static_assert(P::kMin, "the strip kernel serves the minimum measures");
  extern __shared__ __align__(16) float2 strip_smem[];
  constexpr int RM = strip_rmax<P>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kWarps = kStripThreads / 32;
  float2* pts = strip_smem + (size_t)warp * (cap + 2 * kStripPad);
  // the row between strips: there only where the launch's longest pair needs it
  const int bufcap = multi ? cap + 2 * kStripPad : 0;
  V* buf = reinterpret_cast<V*>(strip_smem + (size_t)kWarps * (cap + 2 * kStripPad)) +
           (size_t)warp * bufcap;
  const int slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nslots = (gridDim.x * blockDim.x) >> 5;
  const int npairs = a.npairs_dev ? min(*a.npairs_dev, a.npairs) : a.npairs;
  for (int wk = slot; wk < npairs; wk += nslots) {
    const int pid = a.order ? a.order[wk] : wk;
    const int2 pr = a.pairs[pid];
    if (pr.y < 0) continue;
    const int64_t qo = a.qoff[pr.x], co = a.coff[pr.y];
    const int n = (int)(a.qoff[pr.x + 1] - qo), m = (int)(a.coff[pr.y + 1] - co);
    if (n < 1 || m < 1) {  // an empty trajectory: no path
      if (lane == 0) store_result(a, pid, P::border());
      continue;
    }
    // rows on the side that makes the pair cheaper
    int Rq, Rc;
    const int cq = m <= cap ? strip_cost(n, m, RM, Rq) : 0x7fffffff;
    const int cc = n <= cap ? strip_cost(m, n, RM, Rc) : 0x7fffffff;
    if (min(cq, cc) == 0x7fffffff) {  // both sides longer than the staging
      if (lane == 0) spill[atomicAdd(nspill, 1)] = pid;
      continue;
    }
    const bool tr = cc < cq;
    const int rows = tr ? m : n, cols = tr ? n : m, R = tr ? Rc : Rq;
    if (rows > 32 * RM && !multi) {  // longer than max_n and max_m: no row to join its strips
      if (lane == 0) spill[atomicAdd(nspill, 1)] = pid;
      continue;
    }
    const float2* O = tr ? a.cpts + co : a.qpts + qo;
    const float2* I = tr ? a.qpts + qo : a.cpts + co;
    const float thr = a.thr ? a.thr[pr.x] : TSIM_INF;
    const float aux = a.aux ? (float)a.aux[pid] : a.eps;
    __syncwarp();  // the previous pair's reads are done
    for (int j = lane - kStripPad; j < cols + kStripPad; j += 32)
      PT(j) = (unsigned)j < (unsigned)cols ? __ldg(I + j) : make_float2(TSIM_INF, TSIM_INF);
    __syncwarp();
    if (rows > 32 * RM)
      strip_pair<P, RM, true>(a, pid, O, rows, cols, thr, aux, pts, buf, cap, bufcap);
    else if (R == 2)
      strip_pair<P, 2, false>(a, pid, O, rows, cols, thr, aux, pts, buf, cap, bufcap);
    else if (R == 4)
      strip_pair<P, 4, false>(a, pid, O, rows, cols, thr, aux, pts, buf, cap, bufcap);
    else
      strip_pair<P, RM, false>(a, pid, O, rows, cols, thr, aux, pts, buf, cap, bufcap);
  }
}

#undef PT
#undef ROWBUF

// Two pairs a warp, 16 lanes and 16 R rows each, for launches whose pairs
// all have a side of at most 16 R points: 15 steps of ramp for a strip
// instead of 31 (128 x 128: 143 steps of 8 rows for two pairs against 159 of
// 4 rows for one: 8,192 such pairs 61 -> 57 us, and the reference's
// square-root cost, 1,024 x 10 pairs of them, 131 us, striped 178).  The halves'
// pairs differ in length, so a lane outside
// its matrix sits the step out; its last values stay for the result.
#define HPT(j) pts[TSIM_SIDX(j, cap)]
template <class P, int R>
__global__ void __launch_bounds__(kStripThreads)
    dp_half_kernel(DpArgs a, int cap, int* spill, int* nspill) {
  using V = typename P::V;
  static_assert(P::kMin, "the strip kernel serves the minimum measures");
  extern __shared__ __align__(16) float2 strip_smem[];
  const int sl = threadIdx.x & 15, half = (threadIdx.x >> 4) & 1;
  float2* pts = strip_smem + (size_t)(threadIdx.x >> 4) * cap;
  const int slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nslots = (gridDim.x * blockDim.x) >> 5;
  const int npairs = a.npairs_dev ? min(*a.npairs_dev, a.npairs) : a.npairs;
  const bool check = a.thr != nullptr;
  for (int base = 2 * slot; base < npairs; base += 2 * nslots) {
    const int wk = base + half;
    const int pid = wk < npairs ? (a.order ? a.order[wk] : wk) : 0;
    const int2 pr = wk < npairs ? a.pairs[pid] : make_int2(0, -1);
    bool has = pr.y >= 0;
    int rows = 1, cols = 0;
    float thr = TSIM_INF, aux = 0.0f;
    float2 o[R];
    V left[R];
    __syncwarp();  // the previous pairs' reads are done
    if (has) {
      const int64_t qo = a.qoff[pr.x], co = a.coff[pr.y];
      const int n = (int)(a.qoff[pr.x + 1] - qo), m = (int)(a.coff[pr.y + 1] - co);
      // rows: the longer side where it fits the lanes, else the shorter
      const int lo = min(n, m), hi = max(n, m);
      rows = hi <= 16 * R ? hi : lo;
      cols = hi <= 16 * R ? lo : hi;
      if (lo < 1) {  // an empty trajectory: no path
        if (sl == 0) store_result(a, pid, P::border());
        has = false;
      } else if (rows > 16 * R || cols > cap) {
        if (sl == 0) spill[atomicAdd(nspill, 1)] = pid;
        has = false;
      }
      if (has) {
        const bool tr = rows != n;
        const float2* O = tr ? a.cpts + co : a.qpts + qo;
        const float2* I = tr ? a.qpts + qo : a.cpts + co;
        if (check) thr = a.thr[pr.x];
        aux = a.aux ? (float)a.aux[pid] : a.eps;
        for (int j = sl; j < cols; j += 16) HPT(j) = __ldg(I + j);
#pragma unroll
        for (int k = 0; k < R; ++k) o[k] = __ldg(O + min(sl * R + k, rows - 1));
      }
    }
    if (!has) {
      rows = 1;
      cols = 0;
#pragma unroll
      for (int k = 0; k < R; ++k) o[k] = make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int k = 0; k < R; ++k) left[k] = P::border();
    __syncwarp();
    const int lres = (rows - 1) / R;
    int end = has ? cols + lres : 0;  // this half's steps
    int nsteps = (int)__reduce_max_sync(0xffffffffu, (unsigned)end);
    V prev_up = sl == 0 ? P::origin() : P::border();
    V bottom = P::border();
    bool alive = true;
    int done = 0;  // steps this half ran before it was abandoned (else end)
    for (int s = 0; s < nsteps;) {
      const int e = min(nsteps, s + 16);
#pragma unroll 4
      for (; s < e; ++s) {
        const V sh = __shfl_up_sync(0xffffffffu, bottom, 1, 16);
        const V upv = sl == 0 ? P::border() : sh;
        if ((unsigned)(s - sl) < (unsigned)cols) {
          const float2 c = HPT(s - sl);
          V up = upv, dg = prev_up;
#pragma unroll
          for (int k = 0; k < R; ++k) {
            const V lf = left[k];
            up = strip_cell<P>(o[k], c, up, lf, dg, aux, 0);
            dg = lf;
            left[k] = up;
          }
          bottom = up;
          prev_up = upv;
        }
      }
      if (check) {  // the frontier, as on the strips of a warp
        float mn = vf(prev_up);
#pragma unroll
        for (int k = 0; k < R; ++k) mn = fminf(mn, vf(left[k]));
        for (int d = 8; d; d >>= 1) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, d, 16));
        if (alive && s < end && mn > thr) {
          alive = false;
          done = s;
          end = 0;
          cols = 0;
        }
        nsteps = (int)__reduce_max_sync(0xffffffffu, (unsigned)end);
      }
    }
    if (a.cells) {
      const int nr = min(max(rows - sl * R, 0), R);
      const int cl = alive ? cols : done;  // columns of this lane's rows
      long long cells = has ? (long long)nr * (alive ? cl : min(max(cl - sl, 0), cl)) : 0;
      for (int d = 8; d; d >>= 1) cells += __shfl_xor_sync(0xffffffffu, cells, d, 16);
      if (sl == 0 && cells) atomicAdd(a.cells, (unsigned long long)cells);
    }
    if (has && !alive) {
      if (sl == 0) store_result(a, pid, P::border());
    } else if (has && sl == lres) {
      V r = left[0];
#pragma unroll
      for (int k = 1; k < R; ++k)
        if ((rows - 1) % R == k) r = left[k];
      store_result(a, pid, r);
    }
  }
}
#undef HPT

template <class P>
int launch_half(tsim_ctx* ctx, const DpArgs& a, int cap, int* spill, int* nspill) {
  auto kern = dp_half_kernel<P, 8>;
  const size_t smem = (size_t)(kStripThreads / 16) * cap * sizeof(float2);
  int per_sm = 0;
  TSIM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kStripThreads, smem));
  if (per_sm < 1) return fail(TSIM_ERR_UNSUPPORTED, "strip kernel does not fit on an SM");
  const long long per_cta = kStripThreads / 16;
  const long long blocks = std::min<long long>((a.npairs + per_cta - 1) / per_cta,
                                               (long long)per_sm * ctx->num_sms);
  kern<<<(unsigned)std::max(blocks, 1ll), kStripThreads, smem, ctx->stream>>>(a, cap, spill, nspill);
  TSIM_CUDA(cudaGetLastError());
  launched(ctx);
  return TSIM_OK;
}

template <class P>
int launch_strip_one(tsim_ctx* ctx, const DpArgs& a, int max_n, int max_m, int* spill,
                     int** nspill_io) {
  if (nspill_io) TSIM_TRY(fresh_counter(ctx, *nspill_io, nspill_io));
  int* nspill = nspill_io ? *nspill_io : nullptr;
  if (a.npairs <= 0) return TSIM_OK;
  // the inner side can always be one of at most the smaller of the longest
  // lengths, so staging is sized for that (with unknown query lengths, for
  // the candidates)
  const int shorter = max_n > 0 ? std::min(max_n, max_m) : max_m;
  const int cap = std::min((shorter + 1) & ~1, kStripMaxCols);
  const int longer = max_n > 0 ? std::max(max_n, max_m) : 0x7fffffff;
  if constexpr (sizeof(typename P::V) == 4 && !std::is_same<P, PolFrechetWin>::value) {
    // two pairs a warp: every pair has a side of at most 128 points, at
    // least one wave of warps is left (below it a pair's own latency counts,
    // and a step of 8 rows takes longer than one of 4), and inner points of
    // up to 512 staged for eight pairs a CTA
    if (shorter > 32 && shorter <= 128 && longer <= 512 && a.npairs >= 8 * ctx->num_sms)
      return launch_half<P>(ctx, a, longer <= 128 ? cap : (longer + 1) & ~1, spill, nspill);
  }
  const int multi = longer > 32 * strip_rmax<P>() ? 1 : 0;
  auto kern = dp_strip_kernel<P>;
  const size_t smem = (size_t)(kStripThreads / 32) * (cap + 2 * kStripPad) *
                      (sizeof(float2) + (multi ? sizeof(typename P::V) : 0));
  if (smem > 48 * 1024)
    TSIM_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int per_sm = 0;
  TSIM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kStripThreads, smem));
  if (per_sm < 1) return fail(TSIM_ERR_UNSUPPORTED, "strip kernel does not fit on an SM");
  const long long warps = kStripThreads / 32;
  const long long blocks = std::min<long long>((a.npairs + warps - 1) / warps,
                                               (long long)per_sm * ctx->num_sms);
  kern<<<(unsigned)std::max(blocks, 1ll), kStripThreads, smem, ctx->stream>>>(a, cap, multi, spill,
                                                                              nspill);
  TSIM_CUDA(cudaGetLastError());
  launched(ctx);
  return TSIM_OK;
}

// Exact FP64 Frechet values without a DP where one cell decides.  The FP64
// optimum is the FP64 cost of some cell whose FP32 cost lies in the window
// around the pair's FP32 optimum (PolFrechetWin), so when all the window's
// cells have one FP64 cost, that is the value: a scan of the costs, no
// dependency between cells, five instructions each.  Of 2,560 pairs of up to
// 256 x 1,024 points about one in twelve holds two different costs in its
// window (64 2^-24 wide) and goes on to the DP.  A CTA per pair, a warp every
// fourth column of 256 rows at a time (a row block's points in registers).
constexpr int kWinRows = 8;
__global__ void __launch_bounds__(kStripThreads)
    frechet_window_kernel(DpArgs a, int* rest, int* nrest) {
  constexpr int kWarps = kStripThreads / 32;
  __shared__ double wval[kWarps];
  __shared__ int wstate[kWarps];  // 0: no window cell, 1: one cost, 2: several
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int npairs = a.npairs_dev ? min(*a.npairs_dev, a.npairs) : a.npairs;
  for (int wk = blockIdx.x; wk < npairs; wk += gridDim.x) {
    const int pid = a.order ? a.order[wk] : wk;
    const int2 pr = a.pairs[pid];
    if (pr.y < 0) continue;  // uniform over the CTA, as below
    const int64_t qo = a.qoff[pr.x], co = a.coff[pr.y];
    const int n = (int)(a.qoff[pr.x + 1] - qo), m = (int)(a.coff[pr.y + 1] - co);
    const float v32 = (float)a.aux[pid];
    if (!(v32 >= 1e-20f) || !(v32 < 1e38f)) {  // the relative window does not hold there
      if (threadIdx.x == 0) rest[atomicAdd(nrest, 1)] = pid;
      continue;
    }
    // costs strictly between lo and hi, as positive floats' bit patterns
    const unsigned lo = __float_as_uint(__fmul_rd(v32, 1.0f - 32.0f / 16777216.0f));
    const unsigned span = __float_as_uint(__fmul_ru(v32, 1.0f + 32.0f / 16777216.0f)) - lo - 1;
    const float2* A = a.qpts + qo;
    const float2* B = a.cpts + co;
    double val = 0.0;
    int state = 0;
    for (int base = 0; base < n; base += 32 * kWinRows) {
      float2 p[kWinRows];
#pragma unroll
      for (int k = 0; k < kWinRows; ++k) p[k] = __ldg(A + min(base + k * 32 + lane, n - 1));
#pragma unroll 2
      for (int j = warp; j < m; j += kWarps) {
        const float2 c = __ldg(B + j);
        unsigned first = 0xffffffffu;
        float d[kWinRows];
#pragma unroll
        for (int k = 0; k < kWinRows; ++k) {
          const float2 t = sub2(p[k], c);
          d[k] = fmaf(t.y, t.y, t.x * t.x);
          first = min(first, __float_as_uint(d[k]) - lo - 1u);
        }
        if (first < span) {  // some cost of this lane's is inside
#pragma unroll
          for (int k = 0; k < kWinRows; ++k)
            if (__float_as_uint(d[k]) - lo - 1u < span) {
              const double x = d2_64(p[k].x, p[k].y, c.x, c.y);
              if (state == 0) {
                val = x;
                state = 1;
              } else if (x != val) {
                state = 2;
              }
            }
        }
      }
    }
    // the lanes', then the warps' costs together
    auto meet = [](double& v, int& s, double v2, int s2) {
      if (s2 == 0) return;
      if (s == 0) v = v2, s = s2;
      else if (s2 == 2 || v2 != v) s = 2;
    };
    for (int o = 16; o; o >>= 1) {
      const double v2 = __shfl_xor_sync(0xffffffffu, val, o);
      const int s2 = __shfl_xor_sync(0xffffffffu, state, o);
      meet(val, state, v2, s2);
    }
    __syncthreads();  // the previous pair's states are read
    if (lane == 0) wval[warp] = val, wstate[warp] = state;
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < kWarps; ++w) meet(val, state, wval[w], wstate[w]);
      if (state == 1)
        a.out64[pid] = val;
      else
        rest[atomicAdd(nrest, 1)] = pid;
    }
  }
}

// The value of a pair with several costs in its window, by deciding which of
// them is the optimum: the smallest cost c for which the cells of cost at most
// c join the first cell to the last.  Joined or not is one bit a cell, so a
// column of up to 1,024 rows is a 32-bit word per lane of one warp: a cell is
// reached from the column before (its row or the row above) or from the row
// above in its own, and the runs of free cells below the reached ones come
// from one addition over the column, whose carry ripples through exactly the
// ones of a run, across the lanes by a second addition on the words' generate
// and propagate ballots.  The window's costs (at most 64 distinct ones) are
// found and ordered first; a binary search then takes one pass over the matrix
// for two costs, six for 64.  The other seven warps turn points into the bits
// of the next 32 columns meanwhile.
//
// What bounds it: the pass's chain of columns, about 80 cycles each, on the one
// pair in twelve that gets here (a CTA for each).  The DP's chain is as long
// but takes four cells of 64-bit minima and maxima a step and eight strips for
// 1,024 rows: the pairs left of 2,560 of up to 256 x 1,024 points 602 -> 52 us.
// Pairs this cannot take (more rows or costs, a window that does not hold) are
// left for the DP.
constexpr int kDecideThreads = 256;
constexpr int kDecideRows = 1024;
constexpr int kDecideCosts = 64;
__global__ void __launch_bounds__(kDecideThreads, 4)
    frechet_decide_kernel(DpArgs a, int* rest, int* nrest) {
  __shared__ float2 row[kDecideRows];
  __shared__ unsigned fw[2][32][33];  // free bits of 32 columns: [column][word of rows]
  __shared__ double found[kDecideCosts], cost[kDecideCosts];
  __shared__ int nfound;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int npairs = a.npairs_dev ? min(*a.npairs_dev, a.npairs) : a.npairs;
  for (int wk = blockIdx.x; wk < npairs; wk += gridDim.x) {
    const int pid = a.order ? a.order[wk] : wk;
    const int2 pr = a.pairs[pid];
    if (pr.y < 0) continue;  // uniform over the CTA, as below
    const int64_t qo = a.qoff[pr.x], co = a.coff[pr.y];
    const int n = (int)(a.qoff[pr.x + 1] - qo), m = (int)(a.coff[pr.y + 1] - co);
    const int rows = min(n, m), cols = max(n, m);
    const float2* O = n <= m ? a.qpts + qo : a.cpts + co;
    const float2* I = n <= m ? a.cpts + co : a.qpts + qo;
    const float v32 = (float)a.aux[pid];
    if (!(v32 >= 1e-20f) || !(v32 < 1e38f) || rows < 1 || rows > kDecideRows) {
      if (threadIdx.x == 0) rest[atomicAdd(nrest, 1)] = pid;
      continue;
    }
    // the window of frechet_window_kernel
    const unsigned lo = __float_as_uint(__fmul_rd(v32, 1.0f - 32.0f / 16777216.0f));
    const unsigned span = __float_as_uint(__fmul_ru(v32, 1.0f + 32.0f / 16777216.0f)) - lo - 1;
    const int W = (rows + 31) >> 5;
    auto d32 = [](float2 p, float2 c) {
      const float2 t = sub2(p, c);
      return __float_as_uint(fmaf(t.y, t.y, t.x * t.x));
    };

    __syncthreads();  // the previous pair's reads are done
    for (int i = threadIdx.x; i < 32 * W; i += kDecideThreads)
      row[i] = i < rows ? __ldg(O + i) : make_float2(TSIM_INF, TSIM_INF);  // never free
    if (threadIdx.x < kDecideCosts) found[threadIdx.x] = -1.0;
    if (threadIdx.x == 0) nfound = 0;
    __syncthreads();
    for (int j = threadIdx.x; j < cols; j += kDecideThreads) {
      const float2 c = __ldg(I + j);
      for (int i0 = 0; i0 < 32 * W; i0 += 8) {
        unsigned first = 0xffffffffu;
#pragma unroll
        for (int k = 0; k < 8; ++k) first = min(first, d32(row[i0 + k], c) - lo - 1u);
        if (first >= span) continue;
        for (int k = 0; k < 8; ++k) {
          if (d32(row[i0 + k], c) - lo - 1u >= span) continue;
          const double x = d2_64(row[i0 + k].x, row[i0 + k].y, c.x, c.y);
          // (a cost written by another thread meanwhile may be listed twice)
          bool have = false;
          const int have_n = min(*(volatile int*)&nfound, kDecideCosts);
          for (int t = 0; t < have_n; ++t) have = have || *(volatile double*)&found[t] == x;
          if (have) continue;
          const int at = atomicAdd(&nfound, 1);
          if (at < kDecideCosts) *(volatile double*)&found[at] = x;
        }
      }
    }
    __syncthreads();
    const int nc = nfound;
    if (nc < 1 || nc > kDecideCosts) {
      if (threadIdx.x == 0) rest[atomicAdd(nrest, 1)] = pid;
      continue;
    }
    if (threadIdx.x < nc) {
      const double x = found[threadIdx.x];
      int r = 0;
      for (int t = 0; t < nc; ++t) r += found[t] < x || (found[t] == x && t < (int)threadIdx.x);
      cost[r] = x;
    }
    __syncthreads();

    // free bits of columns 32 ch .. into fw[ch & 1], words w0, w0 + dw, ..
    auto fill = [&](int ch, double lim, int w0, int dw) {
      const int j = ch * 32 + lane;
      const float2 c = j < cols ? __ldg(I + j) : make_float2(TSIM_INF, TSIM_INF);
      for (int w = w0; w < W; w += dw) {
        unsigned f = 0, in = 0;
#pragma unroll 8
        for (int r = 0; r < 32; ++r) {
          const unsigned d = d32(row[w * 32 + r], c);
          if (d <= lo) f |= 1u << r;
          if (d - lo - 1u < span) in |= 1u << r;
        }
        while (in) {
          const int r = __ffs(in) - 1;
          in &= in - 1;
          const float2 p = row[w * 32 + r];
          if (d2_64(p.x, p.y, c.x, c.y) <= lim) f |= 1u << r;
        }
        fw[ch & 1][lane][w] = f;
      }
    };
    const int nch = (cols + 31) >> 5;
    int t0 = 0, t1 = nc - 1;  // the optimum is one of cost[t0 .. t1]
    while (t0 < t1) {
      const int mid = (t0 + t1) >> 1;
      const double lim = cost[mid];
      unsigned reach = 0;  // warp 0: this lane's 32 rows of the last column done
      bool joined = false;
      fill(0, lim, warp, kDecideThreads / 32);
      __syncthreads();
      for (int ch = 0; ch < nch; ++ch) {
        if (warp == 0) {
          const int w = min(cols - ch * 32, 32);
#pragma unroll 4
          for (int c = 0; c < w; ++c) {
            const unsigned f = lane < W ? fw[ch & 1][c][lane] : 0u;
            const unsigned tops = __ballot_sync(0xffffffffu, reach >> 31);
            unsigned from = reach | (reach << 1) | (((tops << 1) >> lane) & 1u);
            if (ch == 0 && c == 0) from = lane == 0 ? 1u : 0u;
            const unsigned s = f & from;
            const unsigned t = f + s;
            const unsigned gen = __ballot_sync(0xffffffffu, t < f);
            const unsigned pass = __ballot_sync(0xffffffffu, t == 0xffffffffu);
            const unsigned carry = (((gen | pass) + gen) ^ pass) >> lane & 1u;
            reach = (((t + carry) ^ f) | s) & f;
          }
          joined = lane == (rows - 1) >> 5 && (reach >> ((rows - 1) & 31) & 1u);
        } else if (ch + 1 < nch) {
          fill(ch + 1, lim, warp - 1, kDecideThreads / 32 - 1);
        }
        if (!__syncthreads_or(warp == 0 && reach != 0)) break;  // nothing reached in this column
      }
      if (__syncthreads_or(joined))  // of the last column done: false after a break
        t1 = mid;
      else
        t0 = mid + 1;
    }
    if (threadIdx.x == 0) a.out64[pid] = cost[t0];
  }
}

}  // namespace

int launch_frechet_window(tsim_ctx* ctx, const DpArgs& a, int* rest, int** nrest_io) {
  TSIM_TRY(fresh_counter(ctx, *nrest_io, nrest_io));
  int* nrest = *nrest_io;
  if (a.npairs <= 0) return TSIM_OK;
  const int blocks = std::min(a.npairs, 16 * ctx->num_sms);
  frechet_window_kernel<<<blocks, kStripThreads, 0, ctx->stream>>>(a, rest, nrest);
  TSIM_CUDA(cudaGetLastError());
  launched(ctx);
  return TSIM_OK;
}

int launch_frechet_decide(tsim_ctx* ctx, const DpArgs& a, int* rest, int** nrest_io) {
  TSIM_TRY(fresh_counter(ctx, *nrest_io, nrest_io));
  int* nrest = *nrest_io;
  if (a.npairs <= 0) return TSIM_OK;
  const int blocks = std::min(a.npairs, 4 * ctx->num_sms);
  frechet_decide_kernel<<<blocks, kDecideThreads, 0, ctx->stream>>>(a, rest, nrest);
  TSIM_CUDA(cudaGetLastError());
  launched(ctx);
  return TSIM_OK;
}

bool strip_kind(int kind) {
  return kind == DP_DTW_REF || kind == DP_FRECHET_REF || kind == DP_DTW_SQ || kind == DP_DTW_EU ||
         kind == DP_FRECHET_SQ || kind == DP_DTW_SQC || kind == DP_DTW_EUC ||
         kind == DP_FRECHET_SQC || kind == DP_FRECHET_WIN;
}

int strip_max_cols() { return kStripMaxCols; }

int strip_pairs_per_sm(int max_n, int max_m) {
  const int cap = std::min((std::min(max_n, max_m) + 1) & ~1, kStripMaxCols);
  constexpr int kWarps = kStripThreads / 32;
  const int cta = kWarps * (cap + 2 * kStripPad) * (int)(sizeof(float2) + sizeof(float)) + 1024;
  return kWarps * (228 * 1024 / cta);
}

int launch_dp_strip(tsim_ctx* ctx, int kind, const DpArgs& a, int max_n, int max_m, int* spill,
                    int** nspill) {
  switch (kind) {
    case DP_DTW_REF: return launch_strip_one<PolDtwRef>(ctx, a, max_n, max_m, spill, nspill);
    case DP_FRECHET_REF: return launch_strip_one<PolFrechetRef>(ctx, a, max_n, max_m, spill, nspill);
    case DP_DTW_SQ: return launch_strip_one<PolDtwSq>(ctx, a, max_n, max_m, spill, nspill);
    case DP_DTW_EU: return launch_strip_one<PolDtwEu>(ctx, a, max_n, max_m, spill, nspill);
    case DP_FRECHET_SQ: return launch_strip_one<PolFrechetSq>(ctx, a, max_n, max_m, spill, nspill);
    case DP_DTW_SQC: return launch_strip_one<PolDtwSqC>(ctx, a, max_n, max_m, spill, nspill);
    case DP_DTW_EUC: return launch_strip_one<PolDtwEuC>(ctx, a, max_n, max_m, spill, nspill);
    case DP_FRECHET_SQC: return launch_strip_one<PolFrechetSqC>(ctx, a, max_n, max_m, spill, nspill);
    case DP_FRECHET_WIN: return launch_strip_one<PolFrechetWin>(ctx, a, max_n, max_m, spill, nspill);
  }
  return fail(TSIM_ERR_UNSUPPORTED, "no strip kernel for this DP kind");
}

}  // namespace tsim
