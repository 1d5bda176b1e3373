// dp_lcss.cu -- windowed LCSS by bit vectors: a warp per (query, candidate)
// pair, for index windows |i - j| <= delta of at most 63 rows.
//
// The rows of a column differ from their neighbour above by 0 or 1, so a
// column of the LCSS matrix is one bit per row, V (bit 1: no increment), and
// a column with match bits M follows from the last one by
//     V = (V + (V & M)) | (V & ~M)
// (Crochemore, Iliopoulos, Pinzon and Reid, "A fast and practical bit-vector
// algorithm for the longest common subsequence problem", 2001).  With an
// index window only rows j - delta .. j + delta can match column j: rows
// below no longer change, rows above still equal the window's last row (bits
// 1, into which a carry runs out), so 64 bits sliding with the column hold
// all that matters, and the zeros that slide out are counted.  Counts are
// the DP's, exactly.
//
// What is left to do per cell is the match test, and few columns need it: a
// column whose point lies outside the eps-inflated box of its window's rows
// (built once per query by the caller, optional) matches nothing.  The warp
// tests 32 columns' boxes at a time, queues those that pass, and whenever 32
// are queued each lane builds one column's M over the 2 delta + 1 rows, read
// through L1 (the pairs of one query, neighbours in a list, share them; staging
// them per warp held the kernel to 20 warps an SM: 692 us below).  Columns with
// M = 0 leave V as it is; the others (a handful per pair of random walks) are
// applied in order by the whole warp.
//
// What bounds it: issue, five instructions a tested cell (load, packed
// subtraction, two comparisons, set bit), seven at the matrix's ends.  Against
// the lane-per-pair DP, which runs eleven instructions on every cell of the
// window and masks a quarter of its slots: 283,000 pairs of lognormal lengths
// (median 200), delta 20, 1,864 -> 612 us.
//
// Reference kernel replaced: lcss_refine_kernel_m_1 (CudaRuntime1/lcss.cu:46-111).
#include "debug_bounds.cuh"
#include "dp_policies.cuh"

namespace tsim {
namespace {
using namespace dp;

constexpr int kLcssThreads = 128;
constexpr int kLcssMaxDelta = 31;  // 2 delta + 1 rows in 64 bits
constexpr int kLcssQueue = 64;     // queued columns: at most 31 kept, 32 added

__global__ void __launch_bounds__(kLcssThreads) lcss_window_kernel(DpArgs a) {
  constexpr int kWarps = kLcssThreads / 32;
  __shared__ float2 s_qpt[kWarps * kLcssQueue];  // queued columns' points
  __shared__ int s_qcol[kWarps * kLcssQueue];    // and indices
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#define QPT(i) s_qpt[warp * kLcssQueue + TSIM_SIDX(i, kLcssQueue)]
#define QCOL(i) s_qcol[warp * kLcssQueue + TSIM_SIDX(i, kLcssQueue)]
  const int slot = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nslots = (gridDim.x * blockDim.x) >> 5;
  const int npairs = a.npairs_dev ? min(*a.npairs_dev, a.npairs) : a.npairs;
  const int delta = a.delta;
  const float eps = a.eps;
  const unsigned long long wmask = (2ull << (2 * delta)) - 1;  // 2 delta + 1 bits
  const int chunks = (2 * delta + 8) >> 3;                     // of 8 rows
  // a warp takes runs of up to 8 consecutive pairs: one query's, mostly
  const int run = max(1, min(8, npairs / (2 * nslots)));
  int left = 0;
  for (int wk = slot * run - 1, next = slot * run;;) {
    if (left == 0) {  // the next run
      wk = next;
      next += nslots * run;
      left = run;
    } else {
      ++wk;
    }
    --left;
    if (wk >= npairs) break;
    const int pid = a.order ? a.order[wk] : wk;
    const int2 pr = a.pairs[pid];
    if (pr.y < 0) continue;
    const int64_t qo = a.qoff[pr.x], co = a.coff[pr.y];
    const int n = (int)(a.qoff[pr.x + 1] - qo), m = (int)(a.coff[pr.y + 1] - co);
    if (n < 1 || m < 1) {
      if (lane == 0) store_result(a, pid, 0);
      continue;
    }
    const int mc = min(m, n + delta);  // columns whose window holds a row
    const float2* A = a.qpts + qo;
    const float2* B = a.cpts + co;
    // the windows' boxes of this query's columns: max_n + delta + 1 of them
    const float4* E = a.qtab ? a.qtab + (size_t)pr.x * (a.max_n + delta + 1) : nullptr;
    const int ecols = a.max_n + delta + 1;
    __syncwarp();
    unsigned long long V = ~0ull;  // bit b: row vcol - delta + b of column vcol
    int vcol = 0, zeros = 0;
    int queued = 0;
    // the first `k` queued columns: their match bits, then V through them
    auto apply = [&](int k) {
      unsigned long long M = 0;
      int j = 0;
      float2 p = make_float2(0.0f, 0.0f);
      if (lane < k) {
        j = QCOL(lane);
        p = QPT(lane);
      }
      const int r0 = j - delta;
      const bool inner = lane >= k || (r0 >= 0 && r0 + 8 * chunks <= n);
      // rows ch0 .. of 8, to ch1
      auto bits = [&](int ch0, int ch1, auto row) {
        for (int ch = ch0; ch < ch1; ++ch) {
          unsigned w = 0;
#pragma unroll
          for (int u = 0; u < 8; ++u) {
            const float2 d = sub2(row(r0 + ch * 8 + u), p);
            if (fabsf(d.x) < eps && fabsf(d.y) < eps) w |= 1u << u;
          }
          M |= (unsigned long long)w << (8 * ch);
        }
        M &= wmask;  // rows past the window (its chunks of 8)
      };
      if (__all_sync(0xffffffffu, inner)) {
        if (lane < k) bits(0, chunks, [&](int r) { return __ldg(A + r); });
      } else {  // some window reaches over an end of the query: the rows that exist
        const int e0 = max(0, -r0), e1 = min(2 * delta, n - 1 - r0);
        if (lane < k)
          bits(e0 >> 3, (e1 >> 3) + 1, [&](int r) { return __ldg(A + min(max(r, 0), n - 1)); });
        // rows -r0 .. n-1-r0 of the window exist (a column with none: mc)
        M &= (~0ull << e0) & ((2ull << e1) - 1);
        if (lane >= k) M = 0;
      }
      unsigned todo = __ballot_sync(0xffffffffu, M != 0);
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        const unsigned long long Mj = __shfl_sync(0xffffffffu, M, src);
        const int jj = __shfl_sync(0xffffffffu, j, src);
        const int g = jj - vcol;  // rows that slide out of the window
        if (g >= 64) {
          zeros += __popcll(~V);
          V = ~0ull;
        } else if (g > 0) {
          zeros += __popcll(~V & ((1ull << g) - 1));
          V = (V >> g) | ~(~0ull >> g);
        }
        vcol = jj;
        V = (V + (V & Mj)) | (V & ~Mj);
      }
    };
    for (int j0 = 0; j0 < mc; j0 += 32) {
      const int j = j0 + lane;
      bool pass = j < mc;
      float2 p = make_float2(0.0f, 0.0f);
      if (pass) {
        p = __ldg(B + j);
        if (E && j < ecols) {
          const float4 bx = __ldg(E + j);
          pass = p.x >= bx.x && p.x <= bx.z && p.y >= bx.y && p.y <= bx.w;
        }
      }
      const unsigned ball = __ballot_sync(0xffffffffu, pass);
      if (pass) {
        const int at = queued + __popc(ball & ((1u << lane) - 1));
        QCOL(at) = j;
        QPT(at) = p;
      }
      queued += __popc(ball);
      __syncwarp();
      if (queued >= 32) {
        apply(32);
        __syncwarp();
        queued -= 32;
        int cj = 0;
        float2 cp = make_float2(0.0f, 0.0f);
        if (lane < queued) cj = QCOL(32 + lane), cp = QPT(32 + lane);
        __syncwarp();
        if (lane < queued) QCOL(lane) = cj, QPT(lane) = cp;
        __syncwarp();
      }
    }
    if (queued) apply(queued);
    __syncwarp();  // the queue is free for the next pair
    if (lane == 0) store_result(a, pid, zeros + __popcll(~V));
    if (a.cells) {  // the window's cells
      long long cells = 0;
      for (int j = lane; j < mc; j += 32) cells += min(n - 1, j + delta) - max(0, j - delta) + 1;
      for (int o = 16; o; o >>= 1) cells += __shfl_xor_sync(0xffffffffu, cells, o);
      if (lane == 0) atomicAdd(a.cells, (unsigned long long)cells);
    }
  }
#undef QPT
#undef QCOL
}

}  // namespace

// The bit vectors' time grows with the columns that match: 262,144 pairs of 64
// to 512 points, every column tested, took 476 / 642 / 1,418 / 1,834 us for windows
// of 5, 11, 41 and 63 rows with few matches and 3,865 / 4,055 / 4,918 / 5,403
// with a match in every column; a lane a pair 782 / 947 / 1,890 / 2,513 either
// way. With columns outside their box skipped they meet where about 0.17, 0.21,
// 0.37 and 0.46 of the columns match. A query's threshold, the k-th best count
// so far, says how many do in the pairs whose bound still reaches it. With
// every round on the bit vectors, 64 queries against 16,384 trajectories that
// match everywhere took 8.0 ms (11 rows) and 10.1 (41); now 2.3 and 3.8.
float lcss_dense_from(int delta) { return 0.15f + 0.01f * delta; }

bool lcss_window_kind(int kind, int delta) {
  return kind == DP_LCSS && delta >= 0 && delta <= kLcssMaxDelta;
}

int launch_lcss_window(tsim_ctx* ctx, const DpArgs& a) {
  if (a.npairs <= 0) return TSIM_OK;
  int per_sm = 0;
  TSIM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lcss_window_kernel, kLcssThreads,
                                                          0));
  const long long warps = kLcssThreads / 32;
  const long long blocks = std::min<long long>((a.npairs + warps - 1) / warps,
                                               (long long)std::max(per_sm, 1) * ctx->num_sms);
  lcss_window_kernel<<<(unsigned)std::max(blocks, 1ll), kLcssThreads, 0, ctx->stream>>>(a);
  TSIM_CUDA(cudaGetLastError());
  launched(ctx);
  return TSIM_OK;
}

}  // namespace tsim
