// Grouped FP64 GEMM on the FP64 tensor pipe (DMMA, mma.sync m8n8k4 f64).
//
// C_p (+)= alpha_p * A_p * B_p^T for every problem p of a launch: all
// problems whose shape suits one kernel are one launch over a flat list of
// work items, an output tile each and, for problems with long K and few
// outputs, one K range of it (split-K): those write raw partial sums to a
// workspace that a second kernel reduces in a fixed order, so results are
// deterministic.  Operands are read through generic element strides, which
// covers the transposed forms of local_contraction.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "bodies.cuh"
#include "common.h"
#include "launch.h"
#include "program.h"

namespace cg = cooperative_groups;

namespace gbx {

namespace {
constexpr int kRedThreads = dev::kRedThreads;
constexpr int kThinN = 32, kThinK = 64, kThinMinWide = 16384;
constexpr int kSmallK = dev::kSmallK;
constexpr int kSmallKElems = dev::kSmallKElems;  // output elements per CTA
constexpr int kSmallOutDim = dev::kSmallOutDim;  // small outputs: at most 16 x 16 ...
constexpr int kSmallOutMinK = 4096;  // ... with at least this K
constexpr int kSmallOutChunk = 2048;  // K per work item
constexpr int kGemvDim = dev::kGemvDim;  // matrix-vector problems: one side at most this ...
constexpr int kGemvMinK = 64;         // ... with K above this
constexpr int kGemvItems = 152 * 4;   // work items that keep every SM busy
constexpr int kGemvMinChunk = 1024;   // smallest K range of a split
constexpr int kSms = 152;
constexpr int kQuarters = 4 * kSms;   // FP64 pipes: one per SM quarter

int ceil_div(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }
}  // namespace

// Variant 0 (tile_gemm_f64_kernel) takes any shape.  K <= 8 (outer products)
// runs with one thread per output element (variant 6).  Thin problems (one
// side at most 32) run with one thread per row (4) or column (5) of C, exact
// in the thin side, where enough rows keep the 152 SMs evenly busy: the tile
// kernel computes whole 8 x 8 x 4 blocks, so the thin kernel is taken when
// its waves of 152 CTAs are fuller than the blocks are real (times 0.9, what
// the tile kernel reaches on such shapes).  Measured, tile / thin kernel:
// 5000 x 6 x 30 12 / 23 us, 100000 x 6 x 30 78 / 54, 40000 x 24 x 64 143 /
// 207, 100000 x 24 x 64 306 / 320, 300000 x 24 x 64 883 / 825.  K beyond one
// stage only where the rows are very many: a thread walks K alone, and few
// CTAs have too few loads in flight for that (13000 x 3 x 75 23 / 39 us, 16000
// x 3 x 100 31 / 44, 14000 x 3 x 2000 431 / 1033).
// Before either, variant 7: outputs of at most 16 x 16 with long K, one CTA
// per K chunk holding the whole output (reduced in a fixed order), and 8:
// matrix-vector shapes (one side <= 2, K > 64), one warp per output of the
// wide side, the wide operand's rows read once and coalesced.
static int variant_of(int m, int n, int k, int gemv_min_k) {
  if (k <= kSmallK) return 6;
  if (m <= kSmallOutDim && n <= kSmallOutDim && k >= kSmallOutMinK) return 7;
  if (k > gemv_min_k && ((m <= kGemvDim && n > kSmallOutDim) || (n <= kGemvDim && m > kSmallOutDim))) return 8;
  const bool rows = n <= kThinN && m >= 4 * n, cols = m <= kThinN && n >= 4 * m;
  if (rows || cols) {
    const int wide = rows ? m : n, thin = rows ? n : m;
    const int ctas = ceil_div(wide, 256);
    const double filled = (double)ctas / ((double)kSms * ceil_div(ctas, kSms));
    const double real = (double)thin / (8.0 * ceil_div(thin, 8)) * (double)k / (4.0 * ceil_div(k, 4));
    if ((k <= kThinK || wide >= kThinMinWide) && filled > 0.9 * real) return rows ? 4 : 5;
  }
  return 0;
}
int f64_variant(int m, int n, int k) { return variant_of(m, n, k, kGemvMinK); }

// One thread per row (variant 4) or per column (variant 5) of C; the thin
// operand (at most kThinN rows) is staged through shared memory kThinK
// columns at a time, so K is unbounded.  Each output is a k-ordered FMA
// chain, so results are deterministic.
template <bool kRows>
__device__ __forceinline__ void thin_body(const GemmProblem* __restrict__ probs, int nprob,
                                          const int* __restrict__ block_first, int total_blocks, double* Ts) {
  for (int blk = blockIdx.x; blk < total_blocks; blk += gridDim.x) {
    int lo = 0, hi = nprob - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (block_first[mid] <= blk) lo = mid; else hi = mid - 1;
    }
    const GemmProblem& p = probs[lo];
    const int64_t i0 = (int64_t)(blk - block_first[lo]) * 256;
    // thin operand: B (N x K) for row mode, A (M x K) for column mode
    const int tn = kRows ? p.n : p.m;
    const double* T = kRows ? p.B : p.A;
    const int64_t trs = kRows ? p.b_rs : p.a_rs, tcs = kRows ? p.b_cs : p.a_cs;
    const int64_t i = i0 + threadIdx.x;
    const int64_t wide = kRows ? p.m : p.n;
    const double* W = kRows ? p.A + i * p.a_rs : p.B + i * p.b_rs;
    const int64_t wcs = kRows ? p.a_cs : p.b_cs;
    double acc[kThinN];
#pragma unroll
    for (int j = 0; j < kThinN; ++j) acc[j] = 0.0;
    for (int k0 = 0, kc; k0 < p.k; k0 += kc) {
      kc = min(kThinK, (k0 < p.twice ? p.twice : p.k) - k0);  // a stage ends with the columns that count twice
      __syncthreads();
      for (int e = threadIdx.x; e < tn * kc; e += 256)
        Ts[e] = __ldg(T + (int64_t)(e / kc) * trs + (int64_t)(k0 + e % kc) * tcs);
      __syncthreads();
      if (i < wide) {
        for (int k = 0; k < kc; ++k) {
          const double w = __ldg(W + (int64_t)(k0 + k) * wcs);
#pragma unroll
          for (int j = 0; j < kThinN; ++j)
            if (j < tn) acc[j] = fma(w, Ts[j * kc + k], acc[j]);
        }
      }
      if (k0 + kc == p.twice) {
#pragma unroll
        for (int j = 0; j < kThinN; ++j)
          if (j < tn) acc[j] = __dadd_rn(acc[j], acc[j]);
      }
    }
    if (i < wide) {
#pragma unroll
      for (int j = 0; j < kThinN; ++j) {
        if (j >= tn) break;
        double* c = kRows ? p.C + i * p.c_rs + j : p.C + (int64_t)j * p.c_rs + i;
        const double v = __dmul_rn(p.alpha, acc[j]);
        *c = p.accumulate ? __dadd_rn(*c, v) : v;
      }
    }
  }
}

template <bool kRows>
__global__ void __launch_bounds__(256) thin_gemm_f64_kernel(const GemmProblem* __restrict__ probs, int nprob,
                                                            const int* __restrict__ block_first, int total_blocks) {
  begin_dependent();
  __shared__ double Ts[kThinN * kThinK];
  thin_body<kRows>(probs, nprob, block_first, total_blocks, Ts);
}

// Matrix-vector shapes (variant 8): dev::gemv_body.
template <bool kTwice>
__global__ void __launch_bounds__(256) gemv_f64_kernel(const GemmProblem* __restrict__ probs, int nprob,
                                                       const int* __restrict__ block_first, int total_blocks) {
  begin_dependent();
  dev::gemv_body<false, kTwice>(probs, nprob, block_first, total_blocks, blockIdx.x, gridDim.x);
}

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c[0]), "+d"(c[1])
               : "d"(a), "d"(b));
}

// ---- tile kernel (variant 0) -------------------------------------------------
//
// The FP64 pipe bounds this kernel and nothing else comes near: a DMMA
// m8n8k4 occupies its quarter of the SM for 512 cycles (1.047 TFLOP/s over
// 152 SMs, DMMA and DFMA alike, measured), against 256 bytes of operands.
// So the operands go from L1 / L2 straight into the fragments -- no shared
// memory stages, no barriers in the K loop -- and everything is spent on
// keeping all 608 quarters busy to the end: output tiles of 16 x 16 or
// 8 x 8, of which only the 8 x 8 blocks that hold real outputs are issued.
// Very many tiles go one to a warp; else the K steps of a tile are dealt to
// the four warps of a CTA (one per quarter) and, when the tiles are few, to a
// cluster of up to eight CTAs, whose sums are added in a fixed order through
// (distributed) shared memory.  Longer K still is cut into ranges that write
// partial sums (splitk_reduce_kernel).
constexpr int kTileWarps = 4;
constexpr int kTileThreads = 32 * kTileWarps;
constexpr int kTileUnroll = 4;  // K steps (of 4) per register stage, two stages

struct TileSmem {
  double part[kTileWarps][256];
  double sum[256];
};

// Adds K steps [s0, s1) of the range [kbeg, kend) to MB x NB blocks of 8 x 8.
template <int MB, int NB>
__device__ __forceinline__ void tile_steps(const GemmProblem& p, int m0, int n0, int kbeg, int kend, int s0, int s1,
                                           double (&acc)[MB][NB][2]) {
  const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
  const int64_t acs = p.a_cs, bcs = p.b_cs;
  const double* pa[MB];
  const double* pb[NB];
  const int64_t k0 = kbeg + 4 * (int64_t)s0 + q;
  // rows past the end repeat the last one: they only reach outputs that are not stored
#pragma unroll
  for (int i = 0; i < MB; ++i) pa[i] = p.A + (int64_t)min(m0 + 8 * i + r, p.m - 1) * p.a_rs + k0 * acs;
#pragma unroll
  for (int j = 0; j < NB; ++j) pb[j] = p.B + (int64_t)min(n0 + 8 * j + r, p.n - 1) * p.b_rs + k0 * bcs;
  double a[2][kTileUnroll][MB], b[2][kTileUnroll][NB];
  auto load = [&](int buf, int s) {
#pragma unroll
    for (int u = 0; u < kTileUnroll; ++u) {
      const bool in = s + u < s1 && kbeg + 4 * (s + u) + q < kend;
      const int64_t d = 4 * (int64_t)(s - s0 + u);
#pragma unroll
      for (int i = 0; i < MB; ++i) a[buf][u][i] = in ? __ldg(pa[i] + d * acs) : 0.0;
#pragma unroll
      for (int j = 0; j < NB; ++j) b[buf][u][j] = in ? __ldg(pb[j] + d * bcs) : 0.0;
    }
  };
  auto mma = [&](int buf, int s) {
#pragma unroll
    for (int u = 0; u < kTileUnroll; ++u) {
      if (s + u >= s1) break;
#pragma unroll
      for (int i = 0; i < MB; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j) dmma884(acc[i][j], a[buf][u][i], b[buf][u][j]);
    }
  };
  if (s0 < s1) load(0, s0);
  for (int s = s0; s < s1; s += 2 * kTileUnroll) {
    if (s + kTileUnroll < s1) load(1, s + kTileUnroll);
    mma(0, s);
    if (s + 2 * kTileUnroll < s1) load(0, s + 2 * kTileUnroll);
    if (s + kTileUnroll < s1) mma(1, s + kTileUnroll);
  }
}

// K steps of the range [kbeg, kend): with kTwice those of its columns that
// count twice, then the others (no step holds both).
__device__ __forceinline__ int steps_twice(const GemmProblem& p, int kbeg, int kend) {
  return (max(min(kend, p.twice) - kbeg, 0) + 3) / 4;
}
template <bool kTwice>
__device__ __forceinline__ int k_steps(const GemmProblem& p, int kbeg, int kend) {
  if (!kTwice) return (max(kend - kbeg, 0) + 3) / 4;
  return steps_twice(p, kbeg, kend) + (max(kend - max(kbeg, p.twice), 0) + 3) / 4;
}

// MB x NB blocks of 8 x 8 over K steps [s0, s1) of the range [kbeg, kend);
// out(row, col, two sums) takes the results, rows and columns within the tile.
template <int MB, int NB, bool kTwice, class Out>
__device__ __forceinline__ void tile_loop(const GemmProblem& p, int m0, int n0, int kbeg, int kend, int s0, int s1,
                                          Out&& out) {
  const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
  double acc[MB][NB][2];
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  if constexpr (!kTwice) {
    tile_steps<MB, NB>(p, m0, n0, kbeg, kend, s0, s1, acc);
  } else {
    const int n2 = steps_twice(p, kbeg, kend);
#pragma unroll 1
    for (bool dbl = s0 < n2;; dbl = false) {
      tile_steps<MB, NB>(p, m0, n0, dbl ? kbeg : max(kbeg, p.twice), dbl ? min(kend, p.twice) : kend,
                         dbl ? s0 : max(s0 - n2, 0), dbl ? min(s1, n2) : max(s1 - n2, 0), acc);
      if (!dbl) break;
      // what counts twice: the sums so far, doubled exactly
#pragma unroll
      for (int i = 0; i < MB; ++i)
#pragma unroll
        for (int j = 0; j < NB; ++j) {
          acc[i][j][0] = __dadd_rn(acc[i][j][0], acc[i][j][0]);
          acc[i][j][1] = __dadd_rn(acc[i][j][1], acc[i][j][1]);
        }
    }
  }
#pragma unroll
  for (int i = 0; i < MB; ++i)
#pragma unroll
    for (int j = 0; j < NB; ++j) out(8 * i + r, 8 * j + 2 * q, acc[i][j][0], acc[i][j][1]);
}

// The 8 x 8 blocks of a 16 x 16 tile that hold real outputs.
template <bool kTwice, class Out>
__device__ __forceinline__ void tile_blocks(const GemmProblem& p, bool m2, bool n2, int m0, int n0, int kbeg, int kend,
                                            int s0, int s1, Out&& out) {
  if (m2 && n2) tile_loop<2, 2, kTwice>(p, m0, n0, kbeg, kend, s0, s1, out);
  else if (m2) tile_loop<2, 1, kTwice>(p, m0, n0, kbeg, kend, s0, s1, out);
  else if (n2) tile_loop<1, 2, kTwice>(p, m0, n0, kbeg, kend, s0, s1, out);
  else tile_loop<1, 1, kTwice>(p, m0, n0, kbeg, kend, s0, s1, out);
}

// Work item `local` of problem p when every warp has a 16 x 16 tile of its own.
template <bool kTwice>
__device__ __forceinline__ void warp_tile_item(const GemmProblem& p, int64_t local) {
  const int ntn = (p.n + 15) / 16, ntm = (p.m + 15) / 16;
  const int64_t t = local * kTileWarps + (threadIdx.x >> 5);
  if (t >= (int64_t)ntm * ntn) return;
  const int m0 = (int)(t / ntn) * 16, n0 = (int)(t % ntn) * 16;
  const auto store = [&](int i, int j, double x, double y) {
    const int64_t gm = m0 + i, gn = n0 + j;
    if (gm >= p.m) return;
    double* c = p.C + gm * p.c_rs + gn;
    if (gn < p.n) c[0] = p.accumulate ? __dadd_rn(c[0], __dmul_rn(p.alpha, x)) : __dmul_rn(p.alpha, x);
    if (gn + 1 < p.n) c[1] = p.accumulate ? __dadd_rn(c[1], __dmul_rn(p.alpha, y)) : __dmul_rn(p.alpha, y);
  };
  tile_blocks<kTwice>(p, p.m - m0 > 8, p.n - n0 > 8, m0, n0, 0, p.k, 0, k_steps<kTwice>(p, 0, p.k), store);
}

// One work item of problem p: output tile of edge TS (16 or 8) and K range
// `local`.
template <int TS, bool kTwice>
__device__ __forceinline__ void cluster_tile_item(const GemmProblem& p, int64_t local, TileSmem& sm) {
  constexpr int ts = TS;
  const cg::cluster_group cl = cg::this_cluster();
  const int csize = (int)cl.num_blocks(), crank = (int)cl.block_rank();
  const int warp = threadIdx.x >> 5;
  const int ntn = (p.n + ts - 1) / ts, ntm = (p.m + ts - 1) / ts;
  const int64_t per_k = (int64_t)ntm * ntn;
  const int kc = (int)(local / per_k);
  const int t = (int)(local - kc * per_k);
  const int m0 = t / ntn * ts, n0 = (t % ntn) * ts;
  const int kbeg = kc * p.kchunk, kend = min(p.k, kbeg + p.kchunk);
  const int steps = k_steps<kTwice>(p, kbeg, kend);
  const int per = (steps + csize * kTileWarps - 1) / (csize * kTileWarps);
  const int s0 = min(steps, (crank * kTileWarps + warp) * per), s1 = min(steps, s0 + per);
  const bool m2 = ts == 16 && p.m - m0 > 8, n2 = ts == 16 && p.n - n0 > 8;
  double* part = sm.part[warp];
  const auto keep = [&](int i, int j, double x, double y) {
    *reinterpret_cast<double2*>(part + i * 16 + j) = make_double2(x, y);
  };
  if constexpr (TS == 8) tile_loop<1, 1, kTwice>(p, m0, n0, kbeg, kend, s0, s1, keep);
  else tile_blocks<kTwice>(p, m2, n2, m0, n0, kbeg, kend, s0, s1, keep);
  __syncthreads();
  const int rows = min(ts, p.m - m0), cols = min(ts, p.n - n0);
  const auto add = [&](int e) {
    double v = sm.part[0][e];
#pragma unroll
    for (int w = 1; w < kTileWarps; ++w) v = __dadd_rn(v, sm.part[w][e]);
    return v;
  };
  const auto store = [&](int e, double v) {
    const int i = e >> 4, j = e & 15;
    const int64_t gm = m0 + i, gn = n0 + j;
    if (p.ksplit > 1) {
      p.partial[(int64_t)kc * p.m * p.n + gm * p.n + gn] = v;
    } else {
      double* c = p.C + gm * p.c_rs + gn;
      v = __dmul_rn(p.alpha, v);
      *c = p.accumulate ? __dadd_rn(*c, v) : v;
    }
  };
  const auto real = [&](int e) { return (e >> 4) < rows && (e & 15) < cols; };
  if (csize == 1) {
    for (int e = threadIdx.x; e < 256; e += kTileThreads)
      if (real(e)) store(e, add(e));
    return;
  }
  for (int e = threadIdx.x; e < 256; e += kTileThreads)
    if (real(e)) sm.sum[e] = add(e);
  cl.sync();
  // output e is summed over the cluster, in rank order, by rank e % csize
  for (int e = (int)threadIdx.x * csize + crank; e < 256; e += kTileThreads * csize)
    if (real(e)) {
      double v = *cl.map_shared_rank(&sm.sum[e], 0);
      for (int c = 1; c < csize; ++c) v = __dadd_rn(v, *cl.map_shared_rank(&sm.sum[e], c));
      store(e, v);
    }
  cl.sync();  // no CTA leaves while another reads its sums
}

// Work item `local` of problem p; TS 0: a tile per warp.
template <int TS, bool kTwice>
__device__ __forceinline__ void tile_item(const GemmProblem& p, int64_t local, TileSmem& sm) {
  if constexpr (TS == 0) warp_tile_item<kTwice>(p, local);
  else cluster_tile_item<TS, kTwice>(p, local, sm);
}

// All problems of a launch, one work item per cluster: the item's problem is
// found by a 32-way search of the first-item table.
template <int TS, bool kTwice>
__global__ void __launch_bounds__(kTileThreads, TS == 8 ? 8 : 4)
    tile_gemm_f64_kernel(const GemmProblem* __restrict__ probs, int nprob, const int* __restrict__ first) {
  begin_dependent();
  __shared__ TileSmem sm;
  const int item = (int)(blockIdx.x / cg::this_cluster().num_blocks());
  int lo = 0, n = nprob;
  while (n > 1) {
    const int step = (n + 31) / 32, at = lo + (int)(threadIdx.x & 31) * step;
    const unsigned le = __ballot_sync(0xffffffffu, at < lo + n && __ldg(first + min(at, nprob - 1)) <= item);
    const int hit = 31 - __clz(le);  // the first entry of the range is always <= item
    const int nlo = lo + hit * step;
    n = min(step, lo + n - nlo);
    lo = nlo;
  }
  tile_item<TS, kTwice>(probs[lo], item - first[lo], sm);
}

// A one-problem launch with its descriptor in the kernel's arguments: nothing to upload, no search.
struct OneProblem {
  GemmProblem p;
  int zero;            // the problem's first work item
  int red_prob;        // split-K reduction: problem index (0)
  uint32_t red_first;  // and its first chunk (0)
};

template <int TS>
__global__ void __launch_bounds__(kTileThreads, TS == 8 ? 8 : 4)
    tile_one_f64_kernel(const __grid_constant__ OneProblem a) {
  begin_dependent();
  __shared__ TileSmem sm;
  tile_item<TS, false>(a.p, blockIdx.x / cg::this_cluster().num_blocks(), sm);
}

// K <= 8 (dev::small_k_body).
__global__ void __launch_bounds__(256) small_k_gemm_f64_kernel(const GemmProblem* __restrict__ probs, int nprob,
                                                               const int* __restrict__ block_first, int total_blocks) {
  begin_dependent();
  dev::small_k_body<false>(probs, nprob, block_first, total_blocks, blockIdx.x, gridDim.x);
}

// Small output, long K (variant 7, dev::small_out_body).
__global__ void __launch_bounds__(256) small_out_gemm_f64_kernel(const GemmProblem* __restrict__ probs, int nprob,
                                                                 const int* __restrict__ item_first, int total) {
  begin_dependent();
  __shared__ dev::SmallOutSmem sm;
  dev::small_out_body<false>(probs, nprob, item_first, total, blockIdx.x, gridDim.x, sm);
}

// Fixed-order reduction of split-K partials into C.
__global__ void __launch_bounds__(kRedThreads) splitk_reduce_kernel(const GemmProblem* __restrict__ probs,
                                                                    const int* __restrict__ red_prob,
                                                                    const uint32_t* __restrict__ red_first, int nred,
                                                                    uint32_t nchunks) {
  begin_dependent();
  __shared__ double red[kRedThreads];
  dev::splitk_reduce_body<false>(probs, red_prob, red_first, nred, nchunks, blockIdx.x, gridDim.x, red);
}

// The one-problem forms of the kernels above.
template <bool kRows>
__global__ void __launch_bounds__(256) thin_one_f64_kernel(const __grid_constant__ OneProblem a, int total) {
  begin_dependent();
  __shared__ double Ts[kThinN * kThinK];
  thin_body<kRows>(&a.p, 1, &a.zero, total, Ts);
}
__global__ void __launch_bounds__(256) small_k_one_f64_kernel(const __grid_constant__ OneProblem a, int total) {
  begin_dependent();
  dev::small_k_body<false>(&a.p, 1, &a.zero, total, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(256) gemv_one_f64_kernel(const __grid_constant__ OneProblem a, int total) {
  begin_dependent();
  dev::gemv_body<false>(&a.p, 1, &a.zero, total, blockIdx.x, gridDim.x);
}
__global__ void __launch_bounds__(256) small_out_one_f64_kernel(const __grid_constant__ OneProblem a, int total) {
  begin_dependent();
  __shared__ dev::SmallOutSmem sm;
  dev::small_out_body<false>(&a.p, 1, &a.zero, total, blockIdx.x, gridDim.x, sm);
}
__global__ void __launch_bounds__(kRedThreads) splitk_reduce_one_kernel(const __grid_constant__ OneProblem a,
                                                                        uint32_t nchunks) {
  begin_dependent();
  __shared__ double red[kRedThreads];
  dev::splitk_reduce_body<false>(&a.p, &a.red_prob, &a.red_first, 1, nchunks, blockIdx.x, gridDim.x, red);
}

void F64Gemm::release() {
  auto fr = [&](void* q) {
    if (!q) return;
    if (async_stream_set) cudaFreeAsync(q, async_stream); else dev_free(q);
  };
  for (auto& sb : subs) {
    fr(sb.d_probs);
    fr(sb.d_first);
  }
  subs.clear();
  fr(d_all);
  fr(d_partial);
  fr(d_red_prob);
  fr(d_red_first);
  d_all = nullptr;
  d_partial = nullptr;
  d_red_prob = nullptr;
  d_red_first = nullptr;
  nprob = nred = 0;
  red_chunks = 0;
}

namespace {

// Schedule of one launch of the tile kernel: the tile edge (0: a 16 x 16
// tile per warp) and the cluster size.  16 x 16 tiles read half the operand
// bytes per product of 8 x 8 ones, but only many tiles keep the last wave
// short: a tile per warp where the waves of warps are many or full (no
// reduction through shared memory: 300000 x 32 x 30 722 -> 612 us), 16 x 16
// per CTA from twelve per SM on, else 8 x 8 (500 x 500 x 100: 57 us, 65 with
// 16 x 16).  While those leave fewer than two CTAs per SM, clusters share a
// tile's K steps, at least six for every warp (64 x 64 x 432: 10.3 us without,
// 8.3 with four; 192 x 192 x 192, 576 tiles: 17.2 without, 18.7 with two).
// Work that fills every quarter for longer than K ranges cost takes those
// alone: single CTAs spread evenly, clusters of eight do not (below).
// 64 x 48 x 96 takes 3.9 us on the GPU so (one 64 x 64 tile: 125), 1021 x 765
// x 1531 2.29 ms, 1.045 TFLOP/s (64 x 64 tiles: 2.36 ms).
struct TilePlan {
  int ts = 16, cluster = 1;
};

int64_t tile_count(const GemmProblem& q, int ts) { return (int64_t)ceil_div(q.m, ts) * ceil_div(q.n, ts); }

int64_t dmma_count(const GemmProblem& q) { return tile_count(q, 8) * ceil_div(q.k, 4); }

// least: DMMAs of a warp that K ranges have to be worth (tile_ksplit).
TilePlan tile_plan(const std::vector<const GemmProblem*>& probs, int least, bool warp_tiles = true) {
  TilePlan t;
  int64_t n16 = 0, n8 = 0, dmmas = 0;
  int kmax = 0;
  for (const GemmProblem* q : probs) {
    n16 += tile_count(*q, 16);
    n8 += tile_count(*q, 8);
    kmax = std::max(kmax, q->k);
    dmmas += dmma_count(*q);
  }
  const int64_t waves = (n16 + kQuarters - 1) / kQuarters;
  if (!warp_tiles) t.ts = 16;
  else if (waves >= 16 || (waves >= 4 && n16 >= 0.92 * (double)(waves * kQuarters))) t.ts = 0;
  if (t.ts == 0 || n16 >= 12 * kSms) return t;
  t.ts = 8;
  if (dmmas / kQuarters >= 2 * least) return t;
  while (t.cluster < 8 && n8 * t.cluster <= kSms && ceil_div(kmax, 4) >= 48 * t.cluster) t.cluster *= 2;
  return t;
}

// Clusters that get SMs of their own side by side: sixteen of eight CTAs did
// not (32 x 32 x 20000: 94 us, fifteen tiles of 17 x 40 half as long per
// product).
int clusters_apart(int cluster) { return cluster == 8 ? 15 : cluster == 4 ? 36 : kSms / cluster; }

// K ranges of one problem: cut where one CTA's share of a tile would outlast
// an even share of the whole launch (of `dmmas` DMMAs) and `least` DMMAs per
// warp, the cost that the partial sums and their reduction have to be worth.
// A problem that is most of its launch also counts how often its clusters
// come round to an SM, and is cut to even that out (planned, tiles cut by
// their share alone / so: 32 x 32 x 10^6 4422 / 1872 us, 100 x 100 x 50000 1774 /
// 1041, 110 x 110 x 2000 74 / 53, 28 x 3 x 17508 43 / 18).
void tile_ksplit(GemmProblem& q, const TilePlan& t, int64_t dmmas, int least) {
  const int steps = ceil_div(q.k, 4), workers = 4 * t.cluster;
  if (t.ts == 0) return;
  const int64_t blocks = t.ts == 16 ? std::min(2, ceil_div(q.m, 8)) * std::min(2, ceil_div(q.n, 8)) : 1;
  const int64_t item = blocks * ceil_div(steps, workers);
  const int64_t share = std::max<int64_t>(dmmas / kQuarters, least);
  const int64_t most = std::max(1, steps / (8 * workers));
  int64_t ks = std::max<int64_t>(1, std::min<int64_t>((item + share / 2) / share, most));
  if (2 * dmma_count(q) >= dmmas) {
    // the DMMAs of the SM quarter with the most (clusters beyond two rounds
    // share the SMs about evenly)
    const auto load = [&](int64_t k) {
      const int64_t n = tile_count(q, t.ts) * k, apart = clusters_apart(t.cluster);
      const int64_t each = blocks * ceil_div(ceil_div(steps, k), workers);
      return t.cluster > 1 && n > 2 * apart ? n * each / apart : ceil_div(n, apart) * each;
    };
    if (2 * load(1) >= 3 * (dmmas / kQuarters) && load(1) >= least) {
      const int64_t to = std::min(most, 8 * std::max<int64_t>(ks, 2));
      int64_t best = load(ks);
      for (int64_t k = ks; k <= to; ++k) best = std::min(best, load(k));
      while (ks < to && 20 * load(ks) > 21 * best) ++ks;
    }
  }
  const int chunk = 4 * ceil_div(steps, ks);
  q.ksplit = std::max(1, ceil_div(q.k, std::max(chunk, 4)));
  q.kchunk = std::max(chunk, 4);
}

// A tile that one warp would walk long after the others of its launch are
// done: more than twice their average DMMAs, and more than a quarter of an
// even share of the launch.  Such problems get a launch of their own, with
// their K shared (10000 products of 32 x 32 x 32 and one of 32 x 32 x 10^6:
// 317 ms in one launch, 2.5 so; with one of 32 x 32 x 10^5 32 and 0.85).
bool outlasts(const GemmProblem& q, int64_t dmmas, int64_t tiles) {
  const int64_t item = std::min(2, ceil_div(q.m, 8)) * std::min(2, ceil_div(q.n, 8)) * ceil_div(q.k, 4);
  return item > 2 * dmmas / tiles && item > dmmas / kQuarters / 4;
}

// Small outputs: K chunks that give every SM four of all problems' `total_k`,
// of at least 64.
int small_out_chunk(int64_t total_k) { return (int)std::max<int64_t>(64, total_k / (4 * kSms) / 64 * 64); }

// Matrix-vector problems: K ranges when the outputs are few.
void gemv_ksplit(GemmProblem& q) {
  const int64_t wide = q.m <= kGemvDim && q.m <= q.n ? q.n : q.m;
  const int64_t groups = (wide + 7) / 8;
  int ks = 1;
  if (groups < kGemvItems && q.k > 2 * kGemvMinChunk)
    ks = (int)std::min<int64_t>((kGemvItems + groups - 1) / groups, ceil_div(q.k, kGemvMinChunk));
  q.kchunk = ceil_div(ceil_div(q.k, ks), 32) * 32;
  q.ksplit = std::max(1, ceil_div(q.k, q.kchunk));
}

constexpr int kPlannedLeast = 96;   // about 25 us of one quarter: two reduction launches
constexpr int kOneShotLeast = 512;  // a one-shot call also allocates the partial sums

constexpr int kLongTiles = 1;  // variant number of tile-kernel problems with a launch of their own

// Variant, K ranges and tile schedule of every problem (tp[1]: of those with
// kLongTiles); partial sums are numbered from 0 in q.partial (offset + 1, 0 =
// none).  Returns their count.
int64_t f64_schedule(std::vector<GemmProblem>& probs, const std::vector<int>& want, TilePlan (&tp)[2]) {
  std::vector<const GemmProblem*> tiles, long_tiles;
  int64_t dmmas = 0, long_dmmas = 0, small_k = 0;
  for (size_t i = 0; i < probs.size(); ++i) {
    GemmProblem& q = probs[i];
    q.pad_ = want[i] >= 0 ? want[i] : f64_variant(q.m, q.n, q.k);
    if (q.pad_ == 0) {
      tiles.push_back(&q);
      dmmas += dmma_count(q);
    }
    if (q.pad_ == 7) small_k += q.k;
  }
  tp[0] = tile_plan(tiles, kPlannedLeast);
  if (tp[0].ts == 0) {
    int64_t n16 = 0;
    for (const GemmProblem* q : tiles) n16 += tile_count(*q, 16);
    for (GemmProblem& q : probs)
      if (q.pad_ == 0 && outlasts(q, dmmas, n16)) {
        q.pad_ = kLongTiles;
        long_tiles.push_back(&q);
        long_dmmas += dmma_count(q);
      }
    tp[1] = tile_plan(long_tiles, kPlannedLeast, false);
  }
  // small outputs: chunks of up to 2048, shorter where all problems together
  // would leave CTAs without one
  const int chunk7 = std::min(kSmallOutChunk, small_out_chunk(small_k));
  int64_t part = 0;
  for (GemmProblem& q : probs) {
    q.ksplit = 1;
    q.kchunk = std::max(q.k, 4);
    q.partial = nullptr;
    if (q.pad_ == 7) {
      q.ksplit = std::max(1, ceil_div(q.k, chunk7));
      q.kchunk = chunk7;
    } else if (q.pad_ == 8) {
      gemv_ksplit(q);
    } else if (q.pad_ == 0) {
      tile_ksplit(q, tp[0], dmmas, kPlannedLeast);
    } else if (q.pad_ == kLongTiles) {
      tile_ksplit(q, tp[1], long_dmmas, kPlannedLeast);
    }
    if (q.ksplit > 1) {
      q.partial = (double*)(intptr_t)(part + 1);
      part += (int64_t)q.ksplit * q.m * q.n;
    }
  }
  return part;
}

// Work items of a problem's variant.
int64_t f64_items(const GemmProblem& q, int ts) {
  switch (q.pad_) {
    case 4: return ceil_div(q.m, 256);
    case 5: return ceil_div(q.n, 256);
    case 6: return ((int64_t)q.m * q.n + kSmallKElems - 1) / kSmallKElems;
    case 7: return q.ksplit;
    case 8: return (int64_t)ceil_div(q.m <= kGemvDim && q.m <= q.n ? q.n : q.m, 8) * q.ksplit;
    default: return ts == 0 ? (tile_count(q, 16) + kTileWarps - 1) / kTileWarps : tile_count(q, ts) * q.ksplit;
  }
}

uint64_t red_chunks_of(const GemmProblem& q) {
  const int per = q.ksplit >= dev::kRedDeep ? dev::kRedDeepChunk : dev::kRedChunk;
  return ((uint64_t)q.m * q.n + per - 1) / per;
}

// Launch of a tile kernel over `items` work items, one cluster each.
template <class K, class... A>
int launch_tiles(K kernel, const TilePlan& t, int64_t items, cudaStream_t st, const A&... args) {
  if (items * t.cluster >= (1ll << 31)) return fail(GBX_EUNSUPPORTED, "FP64 GEMM has too many work items");
  return launch_dependent(kernel, (unsigned)(items * t.cluster), kTileThreads, st, (unsigned)t.cluster, 0, args...);
}

}  // namespace

int64_t f64_partial_elems(const std::vector<GemmProblem>& in) {
  std::vector<GemmProblem> probs;
  for (auto& q : in)
    if (q.m > 0 && q.n > 0) probs.push_back(q);
  TilePlan tp[2];
  return f64_schedule(probs, std::vector<int>(probs.size(), -1), tp);
}

int F64Gemm::build(const std::vector<GemmProblem>& in, bool async, cudaStream_t st, const std::vector<int>* variants) {
  release();
  async_stream_set = async;
  async_stream = st;
  std::vector<GemmProblem> probs;
  std::vector<int> want;
  for (size_t i = 0; i < in.size(); ++i) {
    const GemmProblem& q = in[i];
    if (q.m <= 0 || q.n <= 0) continue;
    probs.push_back(q);
    int v = variants && i < variants->size() ? (*variants)[i] : -1;
    if (v < -1 || (v > 0 && v < 4) || v > 8) return fail(GBX_EINVAL, "FP64 variant %d", v);
    // the thin kernels need their shape limits
    if ((v == 4 && q.n > kThinN) || (v == 5 && q.m > kThinN) || (v == 6 && q.k > kSmallK) ||
        (v == 7 && (q.m > kSmallOutDim || q.n > kSmallOutDim)) || (v == 8 && q.m > kGemvDim && q.n > kGemvDim))
      return fail(GBX_EINVAL, "FP64 variant %d does not fit %d x %d x %d", v, q.m, q.n, q.k);
    want.push_back(v);
  }
  nprob = (int)probs.size();
  if (nprob == 0) return GBX_OK;
  TilePlan tp[2];
  const int64_t part_elems = f64_schedule(probs, want, tp);
  std::vector<int> red;
  std::vector<uint32_t> red_first;
  uint64_t rc = 0;
  for (int i = 0; i < nprob; ++i)
    if (probs[i].ksplit > 1) {
      red.push_back(i);
      red_first.push_back((uint32_t)rc);
      rc += red_chunks_of(probs[i]);
    }
  if (rc >= (1ull << 31)) return fail(GBX_EUNSUPPORTED, "grouped GEMM has too many partial sums");
  nred = (int)red.size();
  red_chunks = (uint32_t)rc;
  auto alloc = [&](void** q, size_t bytes) -> int {
    if (bytes == 0) {
      *q = nullptr;
      return GBX_OK;
    }
    if (async) {
      GBX_CUDA(cudaMallocAsync(q, bytes, st));
      return GBX_OK;
    }
    return dev_alloc(q, bytes);
  };
  auto copy = [&](void* dst, const void* src, size_t bytes) -> int {
    if (bytes == 0) return GBX_OK;
    if (async) GBX_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
    else GBX_CUDA(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice));
    return GBX_OK;
  };
  GBX_TRY(alloc((void**)&d_partial, sizeof(double) * part_elems));
  for (auto& q : probs)
    if (q.partial) q.partial = d_partial + ((intptr_t)q.partial - 1);
  // one launch per kernel
  for (int v : {0, kLongTiles, 4, 5, 6, 7, 8}) {
    const TilePlan& t = tp[v == kLongTiles ? 1 : 0];
    std::vector<GemmProblem> vp;
    bool twice = false;
    std::vector<int> first;
    int64_t tiles = 0;
    for (auto& q : probs) {
      if (q.pad_ != v) continue;
      vp.push_back(q);
      twice = twice || q.twice > 0;
      first.push_back((int)tiles);
      tiles += f64_items(q, t.ts);
      if (tiles >= (1ll << 31)) return fail(GBX_EUNSUPPORTED, "grouped GEMM has too many work items");
    }
    if (vp.empty()) continue;
    Sub sb;
    sb.variant = v;
    sb.nprob = (int)vp.size();
    sb.total_tiles = (int)tiles;
    sb.ts = t.ts;
    sb.cluster = t.cluster;
    sb.twice = twice;
    GBX_TRY(alloc((void**)&sb.d_probs, sizeof(GemmProblem) * vp.size()));
    GBX_TRY(alloc((void**)&sb.d_first, sizeof(int) * vp.size()));
    GBX_TRY(copy(sb.d_probs, vp.data(), sizeof(GemmProblem) * vp.size()));
    GBX_TRY(copy(sb.d_first, first.data(), sizeof(int) * vp.size()));
    sb.first = first;
    sb.first.push_back((int)tiles);
    subs.push_back(sb);
  }
  if (nred) {
    GBX_TRY(alloc((void**)&d_all, sizeof(GemmProblem) * nprob));
    GBX_TRY(copy(d_all, probs.data(), sizeof(GemmProblem) * nprob));
    GBX_TRY(alloc((void**)&d_red_prob, sizeof(int) * nred));
    GBX_TRY(alloc((void**)&d_red_first, sizeof(uint32_t) * nred));
    GBX_TRY(copy(d_red_prob, red.data(), sizeof(int) * nred));
    GBX_TRY(copy(d_red_first, red_first.data(), sizeof(uint32_t) * nred));
  }
  workspace_bytes = (double)part_elems * 8.0;
  return GBX_OK;
}

int F64Gemm::run(cudaStream_t st) const {
  if (nprob == 0) return GBX_OK;
  if (ProgRecorder* rec = prog_recording()) {
    // the CUDA-core shapes become records of the persistent program (static
    // schedule over their work items); the tile and thin kernels keep their own launches
    for (const Sub& sb : subs) {
      if (sb.twice) return fail(GBX_EUNSUPPORTED, "columns that count twice in a program");
      const int kind = sb.variant == 6 ? PK_SMALLK : sb.variant == 7 ? PK_SMALLOUT : sb.variant == 8 ? PK_GEMV : -1;
      if (kind >= 0) {
        ProgArgs a;
        a.gemm = {sb.d_probs, sb.d_first, sb.nprob, sb.total_tiles};
        GBX_TRY(prog_mem(rec, kind, (uint32_t)std::min(sb.total_tiles, 152 * 8), a, {}));
        continue;
      }
      const Sub* psb = &sb;
      GBX_TRY(prog_ext(rec, [psb](cudaStream_t s2) { return run_sub(*psb, s2); }, {}));
    }
    if (nred) {
      ProgArgs a;
      a.kred = {d_all, d_red_prob, d_red_first, nred, red_chunks};
      GBX_TRY(prog_mem(rec, PK_SPLITKRED, std::min<uint32_t>(red_chunks, 152u * 8u), a, {}));
    }
    return GBX_OK;
  }
  for (const Sub& sb : subs) GBX_TRY(run_sub(sb, st));
  if (nred) {
    int rg = (int)std::min<uint32_t>(red_chunks, 152u * 8u);
    GBX_TRY(launch(splitk_reduce_kernel, (unsigned)rg, kRedThreads, st, d_all, d_red_prob, d_red_first, nred,
                   red_chunks));
  }
  return GBX_OK;
}

namespace {
// The kernel of variant v over problems [probs, probs + nprob) and their `tiles` work items.
int launch_variant(int v, const GemmProblem* probs, int nprob, const int* first, int tiles, const TilePlan& tp,
                   bool twice, cudaStream_t st) {
  const int grid = std::min(tiles, kSms * 8);
  switch (v) {
    case 0:
    case kLongTiles:
      if (twice)
        return launch_tiles(tp.ts == 8 ? tile_gemm_f64_kernel<8, true> : tp.ts ? tile_gemm_f64_kernel<16, true>
                                                                              : tile_gemm_f64_kernel<0, true>,
                            tp, tiles, st, probs, nprob, first);
      return launch_tiles(tp.ts == 8 ? tile_gemm_f64_kernel<8, false> : tp.ts ? tile_gemm_f64_kernel<16, false>
                                                                             : tile_gemm_f64_kernel<0, false>,
                          tp, tiles, st, probs, nprob, first);
    case 4: return launch(thin_gemm_f64_kernel<true>, (unsigned)grid, 256, st, probs, nprob, first, tiles);
    case 6: return launch(small_k_gemm_f64_kernel, (unsigned)grid, 256, st, probs, nprob, first, tiles);
    case 7: return launch(small_out_gemm_f64_kernel, (unsigned)grid, 256, st, probs, nprob, first, tiles);
    case 8:
      return launch(twice ? gemv_f64_kernel<true> : gemv_f64_kernel<false>, (unsigned)grid, 256, st, probs, nprob, first, tiles);
    default: return launch(thin_gemm_f64_kernel<false>, (unsigned)grid, 256, st, probs, nprob, first, tiles);
  }
}
}  // namespace

int F64Gemm::run_sub(const Sub& sb, cudaStream_t st) {
  TilePlan tp;
  tp.ts = sb.ts;
  tp.cluster = sb.cluster;
  return launch_variant(sb.variant, sb.d_probs, sb.nprob, sb.d_first, sb.total_tiles, tp, sb.twice, st);
}

int F64Gemm::run_each(cudaStream_t st) const {
  if (nprob == 0) return GBX_OK;
  for (const Sub& sb : subs) {
    // d_first[0] is 0: problem i is launched as a one-problem group whose
    // first-work-item table is that zero
    for (int i = 0; i < sb.nprob; ++i)
    {
      TilePlan tp;
      tp.ts = sb.ts;
      tp.cluster = sb.cluster;
      GBX_TRY(launch_variant(sb.variant, sb.d_probs + i, 1, sb.d_first, sb.first[i + 1] - sb.first[i], tp, sb.twice, st));
    }
  }
  if (nred) {
    int rg = (int)std::min<uint32_t>(red_chunks, 152u * 8u);
    GBX_TRY(launch(splitk_reduce_kernel, (unsigned)rg, kRedThreads, st, d_all, d_red_prob, d_red_first, nred,
                   red_chunks));
  }
  return GBX_OK;
}

// Kernel of a one-call product: a planned one's, but for the shapes whose few
// outputs and short K the tile kernel's clusters finish first (the kernels for
// long K add their K ranges' partial sums in a launch of their own, and
// matrix-vector warps walk short K one after another), and for the K up to 128
// that leave a matrix-vector warp little but its reduction.  Tile kernel /
// matrix-vector or small-output kernel, one call of many: 2000 x 1 x 2000 73 /
// 22 us, 5000 x 2 x 5000 447 / 113 (150 with the wide operand stored down its
// columns), 700 x 1 x 300 9.1 / 4.9, 20 x 1 x 200000 156 / 31, 1 x 1 x 10^6
// 159 / 45, 12 x 9 x 10^5 122 / 36; the other way round 20 x 1 x 2000 8.4 /
// 16, 300 x 2 x 1200 12.5 / 15, 1 x 1 x 4096 12.9 / 16.6, and against the thin
// kernel 100000 x 2 x 100 99 / 169, 50000 x 1 x 70 30 / 43.
int one_call_variant(int m, int n, int k) {
  const int v = variant_of(m, n, k, 2 * kGemvMinK);
  if (v == 7 && m == 1 && n == 1 && k < 6144) return 0;
  if (v == 8 && k < 4608) {
    const int wide = std::max(m, n);
    if (wide < 400 || (int64_t)ceil_div(wide, 8) * ceil_div(k, 4) < 5000) return 0;
  }
  return v;
}

namespace {
// Stream-ordered temporaries of one-call products, from a pool of their own
// that keeps up to kTempKeep bytes of a device between calls: the default pool
// gives its memory back at every synchronisation, and a call after one then
// waits 150 us for the driver (16 x 16 x 5000 alone: 181 us, 24 so).  The
// pool is the CUDA runtime's, safe with any number of threads and streams.
constexpr uint64_t kTempKeep = 32ull << 20;

int temp_alloc(double** p, size_t bytes, cudaStream_t st) {
  static std::mutex mu;
  static cudaMemPool_t pools[256] = {nullptr};
  int dev = 0;
  GBX_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) return fail(GBX_EUNSUPPORTED, "device ordinal %d out of range", dev);
  cudaMemPool_t pool;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!pools[dev]) {
      cudaMemPoolProps props = {};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      // (also in the first call of a capture, this thread's or another's)
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
      GBX_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
      cudaError_t e = cudaMemPoolCreate(&pool, &props);
      uint64_t keep = kTempKeep;
      if (e == cudaSuccess) e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
      cudaThreadExchangeStreamCaptureMode(&mode);
      if (e != cudaSuccess) return cuda_fail(e, "pool of one-call temporaries", __FILE__, __LINE__);
      pools[dev] = pool;
    }
    pool = pools[dev];
  }
  GBX_CUDA(cudaMallocFromPoolAsync((void**)p, bytes, pool, st));
  return GBX_OK;
}
}  // namespace

// One problem, one call: the descriptor travels in the kernel's arguments.
// The partial sums of long K with few outputs come from `scratch` (at most
// scratch_elems) when given, else from a stream-ordered temporary.
int run_f64_one(const GemmProblem& in, cudaStream_t st, double* scratch, int64_t scratch_elems) {
  OneProblem a;
  std::memset(&a, 0, sizeof(a));
  GemmProblem& q = a.p;
  q = in;
  if (q.m <= 0 || q.n <= 0) return GBX_OK;
  q.pad_ = one_call_variant(q.m, q.n, q.k);
  q.ksplit = 1;
  q.kchunk = std::max(q.k, 4);
  q.partial = nullptr;
  const TilePlan tp = tile_plan({&q}, kOneShotLeast);
  double* own = nullptr;
  if (q.pad_ == 0) {
    tile_ksplit(q, tp, dmma_count(q), kOneShotLeast);
  } else if (q.pad_ == 7) {
    q.kchunk = small_out_chunk(q.k);
    q.ksplit = ceil_div(q.k, q.kchunk);
  } else if (q.pad_ == 8) {
    gemv_ksplit(q);
  }
  if (scratch && (int64_t)q.ksplit * q.m * q.n > scratch_elems) {
    const int64_t ks = std::max<int64_t>(1, scratch_elems / ((int64_t)q.m * q.n));
    q.kchunk = 4 * ceil_div(ceil_div(q.k, 4), ks);
    q.ksplit = std::max(1, ceil_div(q.k, q.kchunk));
  }
  if (q.ksplit > 1) {
    if (!scratch) GBX_TRY(temp_alloc(&own, sizeof(double) * q.ksplit * q.m * q.n, st));
    q.partial = scratch ? scratch : own;
  }
  const int64_t items = f64_items(q, tp.ts);
  if (items >= (1ll << 31)) return fail(GBX_EUNSUPPORTED, "FP64 GEMM has too many work items");
  const int grid = (int)std::min<int64_t>(items, kSms * 8);
  int rc = GBX_OK;
  switch (q.pad_) {
    case 0:
      rc = launch_tiles(tp.ts == 8 ? tile_one_f64_kernel<8> : tp.ts ? tile_one_f64_kernel<16> : tile_one_f64_kernel<0>, tp,
                        items, st, a);
      break;
    case 4: rc = launch(thin_one_f64_kernel<true>, (unsigned)grid, 256, st, a, (int)items); break;
    case 6: rc = launch(small_k_one_f64_kernel, (unsigned)grid, 256, st, a, (int)items); break;
    case 7: rc = launch(small_out_one_f64_kernel, (unsigned)grid, 256, st, a, (int)items); break;
    case 8: rc = launch(gemv_one_f64_kernel, (unsigned)grid, 256, st, a, (int)items); break;
    default: rc = launch(thin_one_f64_kernel<false>, (unsigned)grid, 256, st, a, (int)items); break;
  }
  if (rc == GBX_OK && q.ksplit > 1) {
    const uint32_t chunks = (uint32_t)red_chunks_of(q);
    rc = launch(splitk_reduce_one_kernel, std::min<uint32_t>(chunks, kSms * 8u), kRedThreads, st, a, chunks);
  }
  if (own) cudaFreeAsync(own, st);
  return rc;
}
}  // namespace gbx

// ---- allocation-free local contraction ----------------------------------
//
// Some callers cannot let a library allocate device memory: a framework that
// has handed nearly all of the device's memory to its own caching pool (a
// library cudaMalloc then fails, or forces the pool to give memory back), and
// latency-bound loops that keep other streams busy (cudaFree synchronises the
// device and stalls them).  For them gbx_local_contraction_noalloc runs the
// same FP64 GEMM with its split-K partial sums in one file-scope device
// array of kNoAllocBytes, which every GPU that loads the library holds until
// the process exits; the descriptor travels in the kernel's arguments.
// Nothing of the array needs clearing: every split-K range overwrites its
// slab in full before the reduction reads it.
namespace gbx {
namespace {
constexpr size_t kNoAllocBytes = 32ull << 20;  // split-K partial sums
constexpr int64_t kNoAllocMaxElems = (int64_t)(kNoAllocBytes / sizeof(double));
}  // namespace

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// Device address of the scratch array, looked up once per device (the host
// symbol is only a stand-in for it).
static int noalloc_scratch(unsigned char** out) {
  static std::mutex mu;
  static unsigned char* addr[256] = {nullptr};
  int dev = 0;
  GBX_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 256) return fail(GBX_EUNSUPPORTED, "device ordinal %d out of range", dev);
  std::lock_guard<std::mutex> lk(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)", __FILE__, __LINE__);
    addr[dev] = (unsigned char*)p;
  }
  *out = addr[dev];
  return GBX_OK;
}

}  // namespace gbx

extern "C" int gbx_local_contraction_noalloc(int n_a, int n_b, int n_k, const double* d_A, const double* d_B,
                                             double* d_C, int at, int bt, double alpha, void* stream) {
  using namespace gbx;
  if (n_a < 0 || n_b < 0 || n_k < 0) return fail(GBX_EINVAL, "negative extent");
  if (n_a == 0 || n_b == 0) return GBX_OK;
  if ((int64_t)n_a * n_b > kNoAllocMaxElems)
    return fail(GBX_EINVAL, "output of %lld elements exceeds the allocation-free workspace (max %lld elements)",
                (long long)n_a * n_b, (long long)kNoAllocMaxElems);
  unsigned char* scratch = nullptr;
  GBX_TRY(noalloc_scratch(&scratch));
  GemmProblem p;
  std::memset(&p, 0, sizeof(p));
  p.A = d_A;
  p.B = d_B;
  p.C = d_C;
  p.a_rs = at ? 1 : n_k;
  p.a_cs = at ? n_a : 1;
  p.b_rs = bt ? n_k : 1;
  p.b_cs = bt ? 1 : n_b;
  p.c_rs = n_b;
  p.m = n_a;
  p.n = n_b;
  p.k = n_k;
  p.alpha = alpha;
  p.accumulate = 1;
  return run_f64_one(p, (cudaStream_t)stream, (double*)scratch, kNoAllocMaxElems);
}
