// Split-precision FP64 GEMM on the tcgen05 tensor cores.
//
// C = A * B^T with A (M x K) and B (N x K) row-major FP64.
//
// Split.  Row i of A is scaled by 2^-e_i, e_i the smallest exponent with
// max_k |A_ik| < 2^e_i, and the scaled row is rounded to a fixed-point
// integer X = round(A_ik 2^(F - e_i)), F = 7 + 8 (S - 1).  X is cut into S
// balanced base-256 digits d_1..d_S (d_1 in [-128, 128], the rest in
// [-128, 127]) so that A_ik ~ 2^e_i sum_s d_s 2^-(7 + 8 (s - 1)).  Every digit
// is an integer that bf16 holds exactly.  The split is pure integer
// arithmetic on the FP64 bit pattern (no FP64 instructions); subnormal
// inputs count as zero.  B is split by rows the same way (exponents f_j).
//
// Products.  C_ij = 2^(e_i + f_j - 14) sum_l 2^(-8 l) X_l with
// X_l = sum_{s + t - 2 = l} (D^A_s D^B_t^T)_ij, kept for levels l <= S - 1
// (S (S + 1) / 2 slice products).  Each product runs on tcgen05.mma
// (kind::f16, bf16 operands from TMA-loaded 128B-swizzled shared memory,
// FP32 accumulator in TMEM).  |d_A d_B| <= 2^14, so a TMEM accumulation over
// at most 1024 K-elements stays below 2^24 and is exact; the kernel drains
// the accumulator after every such chunk into int32 registers (exact), folds
// the int32 sums into an FP64 Horner accumulator at each level change
// (acc = acc * 2^-8 + X, levels from S - 1 down to 0), and writes
// 2^(e_i + f_j - 14) * acc.  Only the fold and the final scale are FP64.
//
// Kernel roles (one or two CTAs per SM, persistent over 128 x BN output
// tiles of all problems): warp 0 issues TMA loads into a ring of shared-
// memory stages, warp 1 allocates TMEM and issues the MMAs (one elected
// lane), the drain warps (one per TMEM lane quarter and 64 columns) empty
// the accumulators.  Two to eight TMEM accumulator buffers let the drain of
// one chunk overlap the MMAs of the next.  Every mbarrier wait is bounded (about a second); on timeout the
// kernel records an error, stops issuing work, waits (bounded) for its own
// TMA copies and MMAs in flight, frees its TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <utility>

#include "bodies.cuh"
#include "launch.h"
#include "program.h"
#include "split.h"
#include "split_dev.h"

namespace gbx {

namespace {

constexpr int BM = 128;
constexpr int BK = 64;             // bf16 elements per 128-byte swizzled row
constexpr int kChunkKb = 16;       // k-blocks per exact FP32 chunk (16 * 64 = 1024; half with doubled digits)
constexpr int kFoldChunks = 127;   // int32 drain sums fold into FP64 before overflow

constexpr long long kWaitCycles = 2000000000ll;  // ~1 s at 2 GHz
constexpr int kSplitFill = 152 * 2;  // work items that keep every SM busy

using dev::kMidRow;
using dev::kShortRow;
using dev::kSplitChunk;

struct GemmParams {
  const DevProblem* probs;
  const int* tile_first;
  const CUtensorMap* maps;  // 2 per problem: A, B
  int nprob, total_tiles, S, L;
  int* err;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait; false (and the error word set) when it ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* err, int code,
                                          long long limit = kWaitCycles) {
  if (mbar_try_wait(bar, parity)) return true;
  long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > limit) {
      atomicCAS(err, 0, code);
      return false;
    }
  }
  return true;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
      "[%2];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row atoms of
// 1024 bytes stacked along M/N (stride byte offset 1024).
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;              // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;    // stride byte offset
  d |= (uint64_t)1 << 46;              // descriptor version
  d |= (uint64_t)2 << 61;              // 128-byte swizzle
  return d;
}

// 64-byte swizzled rows (32 bf16 of K): 8-row groups 512 bytes apart
__device__ __forceinline__ uint64_t sdesc64(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;              // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(512 >> 4) << 32;     // stride byte offset
  d |= (uint64_t)1 << 46;              // descriptor version
  d |= (uint64_t)4 << 61;              // 64-byte swizzle
  return d;
}

template <int BN>
__device__ __forceinline__ constexpr uint32_t idesc_bf16() {
  return (1u << 4)                  // D: f32
         | (1u << 7)                // A: bf16
         | (1u << 10)               // B: bf16
         | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

// The same with the output width N (a multiple of 16, at most 256) as a value.
__device__ __forceinline__ constexpr uint32_t idesc_bf16_n(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(
          tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

struct TileInfo {
  int p, m0, n0, kb0, nkb, kc, dbl;
};

template <int BN>
__device__ __forceinline__ TileInfo decode_tile(const GemmParams& P, int tile) {
  TileInfo t;
  int p = 0, hi = P.nprob - 1;
  while (p < hi) {
    const int mid = (p + hi + 1) >> 1;
    if (P.tile_first[mid] <= tile) p = mid; else hi = mid - 1;
  }
  const DevProblem& pr = P.probs[p];
  int local = tile - P.tile_first[p];
  const int per_k = pr.tiles_m * pr.tiles_n;
  t.kc = local / per_k;
  local -= t.kc * per_k;
  t.p = p;
  t.m0 = (local / pr.tiles_n) * BM;
  t.n0 = (local % pr.tiles_n) * BN;
  t.kb0 = t.kc * pr.kb_per_split;
  t.nkb = min(pr.nkb, t.kb0 + pr.kb_per_split) - t.kb0;
  t.dbl = pr.dbl;
  return t;
}

// Number of slice pairs (s, t), 1 <= s, t <= S, on level l = s + t - 2.
__device__ __forceinline__ int level_pairs(int l, int S) {
  int lo = max(1, l + 2 - S), hi = min(S, l + 1);
  return hi >= lo ? hi - lo + 1 : 0;
}

template <int BN>
struct SplitCfg {
  static constexpr int kStageBytes = (BM + BN) * BK * 2;
  // narrow tiles: two CTAs per SM (half the shared memory each) and deeper
  // TMEM buffering, since their chunks are short and drains come often
  static constexpr int kCtasPerSm = BN <= 32 ? 2 : 1;
  static constexpr int kSmemBudget = (BN <= 32 ? 100 : 200) * 1024;
  static constexpr int kStages = (kSmemBudget / kStageBytes) < 8 ? (kSmemBudget / kStageBytes) : 8;
  static constexpr int kAccBufs = BN <= 32 ? 8 : 2;
  static constexpr uint32_t kTmemCols = (kAccBufs * BN <= 32) ? 32 : (kAccBufs * BN <= 64) ? 64
                                        : (kAccBufs * BN <= 128) ? 128 : (kAccBufs * BN <= 256) ? 256 : 512;
  // drain warps: 4 per 64 columns (one per TMEM lane quarter), at least 4
  static constexpr int kDrainWarps = BN >= 64 ? 4 * (BN / 64) : 4;
  static constexpr int kCols = BN >= 64 ? 64 : BN;  // columns per drain thread
  static constexpr int kThreads = 64 + 32 * kDrainWarps;
};

template <int BN>
struct Smem {
  alignas(1024) __nv_bfloat16 a[SplitCfg<BN>::kStages][BM * BK];
  alignas(1024) __nv_bfloat16 b[SplitCfg<BN>::kStages][BN * BK];
  uint64_t full[SplitCfg<BN>::kStages], empty[SplitCfg<BN>::kStages], accfull[SplitCfg<BN>::kAccBufs],
      accempty[SplitCfg<BN>::kAccBufs], done;
  uint32_t tmem_base;
};

// Warp roles: 0 TMA producer, 1 TMEM owner + MMA issuer, 2.. drain.  A drain
// thread owns one row (its TMEM lane) and up to 64 columns; its exact int32 sums
// fold into an FP64 Horner accumulator kept in the output tile itself (or the
// split-K partial), which stays in L2 between the few folds of a tile.
template <int BN>
__global__ void __launch_bounds__(SplitCfg<BN>::kThreads, SplitCfg<BN>::kCtasPerSm)
    split_gemm_kernel(const GemmParams P) {
  using Cfg = SplitCfg<BN>;
  constexpr int kAcc = Cfg::kAccBufs;
  constexpr int kStagesN = Cfg::kStages;
  constexpr int kCols = Cfg::kCols;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Smem<BN>& sm = *reinterpret_cast<Smem<BN>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  begin_dependent();
  constexpr uint32_t kTxBytes = (BM + BN) * BK * 2;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStagesN; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    for (int b = 0; b < kAcc; ++b) {
      mbar_init(&sm.accfull[b], 1);
      mbar_init(&sm.accempty[b], Cfg::kDrainWarps);
    }
    mbar_init(&sm.done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(Cfg::kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  const int S = P.S, L = P.L;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < P.total_tiles && ok; tile += gridDim.x) {
        const TileInfo ti = decode_tile<BN>(P, tile);
        const CUtensorMap* ma = P.maps + 2 * ti.p;
        const CUtensorMap* mb = P.maps + 2 * ti.p + 1;
        for (int l = L; l >= 0 && ok; --l)
          for (int s = max(1, l + 2 - S); s <= min(S, l + 1) && ok; ++s) {
            const int t = l + 2 - s;
            for (int kb = ti.kb0; kb < ti.kb0 + ti.nkb; ++kb) {
              if (!mbar_wait(&sm.empty[stage], phase ^ 1, P.err, 1)) {
                ok = false;
                break;
              }
              mbar_expect_tx(&sm.full[stage], kTxBytes);
              tma_load_3d(sm.a[stage], ma, &sm.full[stage], kb * BK, ti.m0, s - 1);
              tma_load_3d(sm.b[stage], mb, &sm.full[stage], kb * BK, ti.n0, t - 1);
              if (++stage == kStagesN) {
                stage = 0;
                phase ^= 1;
              }
            }
          }
      }
      // wait (bounded) for the copies this warp issued to land before leaving
      for (int i = 0; i < kStagesN; ++i) {
        if (--stage < 0) {
          stage = kStagesN - 1;
          phase ^= 1;
        }
        long long t0 = clock64();
        while (!mbar_try_wait(&sm.full[stage], phase) && !mbar_try_wait(&sm.empty[stage], phase)) {
          if (clock64() - t0 > kWaitCycles) {
            atomicCAS(P.err, 0, 5);
            break;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int stage = 0, buf = 0;
      uint32_t phase = 0, aphase = 0;
      bool ok = true;
      constexpr uint32_t idesc = idesc_bf16<BN>();
      for (int tile = blockIdx.x; tile < P.total_tiles && ok; tile += gridDim.x) {
        const TileInfo ti = decode_tile<BN>(P, tile);
        const int nkb = ti.nkb, chunk_kb = ti.dbl ? kChunkKb / 2 : kChunkKb;
        for (int l = L; l >= 0 && ok; --l) {
          const int items = level_pairs(l, S) * nkb;
          int item = 0;
          for (int s = max(1, l + 2 - S); s <= min(S, l + 1) && ok; ++s) {
            for (int kb = 0; kb < nkb && ok; ++kb, ++item) {
              const int in_chunk = item % chunk_kb;
              if (in_chunk == 0 && !mbar_wait(&sm.accempty[buf], aphase ^ 1, P.err, 2)) {
                ok = false;
                break;
              }
              if (!mbar_wait(&sm.full[stage], phase, P.err, 3)) {
                ok = false;
                break;
              }
              tc_fence_after();
              const uint32_t d = tmem + (uint32_t)(buf * BN);
              const uint64_t a0 = sdesc(smem_u32(sm.a[stage]));
              const uint64_t b0 = sdesc(smem_u32(sm.b[stage]));
#pragma unroll
              for (int k = 0; k < BK / 16; ++k)
                umma(d, a0 + (uint64_t)(k * 2), b0 + (uint64_t)(k * 2), idesc, (in_chunk > 0 || k > 0) ? 1u : 0u);
              umma_commit(&sm.empty[stage]);
              if (++stage == kStagesN) {
                stage = 0;
                phase ^= 1;
              }
              if (in_chunk == chunk_kb - 1 || item == items - 1) {
                umma_commit(&sm.accfull[buf]);
                if (++buf == kAcc) {
                  buf = 0;
                  aphase ^= 1;
                }
              }
            }
          }
        }
      }
      // all MMAs issued by this thread complete before TMEM is released
      umma_commit(&sm.done);
      mbar_wait(&sm.done, 0, P.err, 6);
    }
  } else {
    // ---------------- drain / fold (warps 2..) ----------------
    const int quarter = warp & 3;
    const int group = (warp - 2) >> 2;
    const int row_in_tile = quarter * 32 + lane;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const int col0 = group * kCols;
    int buf = 0;
    uint32_t aphase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < P.total_tiles && ok; tile += gridDim.x) {
      const TileInfo ti = decode_tile<BN>(P, tile);
      const DevProblem& pr = P.probs[ti.p];
      const int row = ti.m0 + row_in_tile;
      const bool row_ok = row < pr.M;
      double* crow = nullptr;
      double scale[1] = {0.0};
      if (row_ok) {
        crow = pr.ksplit > 1 ? pr.partial + ((int64_t)ti.kc * pr.M + row) * pr.N : pr.C + (int64_t)row * pr.ldc;
        scale[0] = (double)pr.eA[row];  // biased row exponent, combined per column below
      }
      int32_t X[kCols];
#pragma unroll
      for (int j = 0; j < kCols; ++j) X[j] = 0;
      bool first_fold = true;
      for (int l = L; l >= 0 && ok; --l) {
        const int items = level_pairs(l, S) * ti.nkb;
        const int chunk_kb = ti.dbl ? kChunkKb / 2 : kChunkKb;
        const int chunks = (items + chunk_kb - 1) / chunk_kb;
        bool scale_pending = l != L;  // Horner: acc = acc * 2^-8 + X_l at the first fold of level l
        int since_fold = 0;
        for (int c = 0; c < chunks; ++c) {
          // one lane waits, the warp follows (tcgen05.ld must stay warp-uniform)
          int w_ok = lane == 0 ? (int)mbar_wait(&sm.accfull[buf], aphase, P.err, 4) : 1;
          w_ok = __shfl_sync(0xffffffffu, w_ok, 0);
          if (!w_ok) {
            ok = false;
            break;
          }
          __syncwarp();
          tc_fence_after();
#pragma unroll
          for (int j0 = 0; j0 < kCols; j0 += 16) {
            uint32_t r[16];
            tmem_ld16(tmem + lane_addr + (uint32_t)(buf * BN + col0 + j0), r);
            tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < 16; ++q) X[j0 + q] += __float2int_rn(__uint_as_float(r[q]));
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.accempty[buf]);
          if (++buf == kAcc) {
            buf = 0;
            aphase ^= 1;
          }
          const bool last = (l == 0 && c == chunks - 1);
          if (++since_fold == kFoldChunks || c == chunks - 1) {
            if (row_ok) {
#pragma unroll
              for (int j = 0; j < kCols; ++j) {
                const int col = ti.n0 + col0 + j;
                if (col < pr.N) {
                  double acc = first_fold ? 0.0 : crow[col];
                  if (scale_pending) acc *= 0x1.0p-8;  // exact
                  acc += (double)X[j];
                  if (last) {
                    // row scale 2^(eA - 1022), column 2^(eB - 1022), digit weights 2^-14
                    int ex = (int)scale[0] + pr.eB[col] - 2 * 1022 - 14 + 1023;
                    ex = ex < 1 ? 1 : (ex > 2046 ? 2046 : ex);
                    acc *= __longlong_as_double((long long)ex << 52);
                  }
                  crow[col] = acc;
                }
              }
            }
#pragma unroll
            for (int j = 0; j < kCols; ++j) X[j] = 0;
            first_fold = false;
            scale_pending = false;
            since_fold = 0;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::kTmemCols));
  }
}

// x * 2^(ex - 1023), the exponent moved by an integer addition: a multiply is
// one of the FP64 instructions that bound the drains (an SM issues 1.8 a
// clock).  x is 0 or of magnitude 2^-60 .. 2^70, ex one of plain_exponent.
__device__ __forceinline__ double scaled(double x, int ex) {
  const int hi = __double2hiint(x);
  return __hiloint2double((hi & 0x7FFFFFFF) ? hi + (ex - 1023) * (1 << 20) : hi, __double2loint(x));
}
__device__ __forceinline__ bool plain_exponent(int ex) { return ex >= 64 && ex <= 1900; }

// T * 2^(ex - 1023), rounded to nearest even, without an FP64 instruction (the
// conversion is one): T normalised, its bits below the 53rd rounded off, the
// exponent set (plain_exponent(ex)).
__device__ __forceinline__ double scaled_int(long long T, int ex) {
  const unsigned long long u = (unsigned long long)(T < 0 ? -T : T);
  const int z = __clzll((long long)u);
  const unsigned long long n = (u << (z & 63)) & 0x7FFFFFFFFFFFFFFFull;  // without its leading 1
  const unsigned long long m = (n + (0x3FFull + ((uint32_t)(n >> 11) & 1u))) >> 11;  // a carry moves the exponent
  const uint32_t hi = (uint32_t)(m >> 32) + ((uint32_t)(ex + 63 - z) << 20);
  return __hiloint2double((int)((u ? hi : 0u) | ((uint32_t)(T >> 32) & 0x80000000u)), (int)(uint32_t)m);
}

// No scale of a warp's elements near the ends of the range: each lane's row
// exponent with each of the column exponents the lanes hold (ebl).  A zero
// row or column (exponent word 0) has sums of 0, which scaled() leaves alone.
__device__ __forceinline__ bool plain_exponents(int ea, int ebl, int offset) {
  const int emin = (int)__reduce_min_sync(0xffffffffu, ebl ? (uint32_t)ebl : 4000u);
  const int emax = (int)__reduce_max_sync(0xffffffffu, (uint32_t)ebl);
  return __all_sync(0xffffffffu, ea == 0 || emax == 0 ||
                                     (plain_exponent(ea + emin + offset) && plain_exponent(ea + emax + offset)));
}

// The 16 or 32 bytes at p (aligned so).
__device__ __forceinline__ void store_vec(double* p, const double (&v)[2]) {
  *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}
__device__ __forceinline__ void store_vec(double* p, const double (&v)[4]) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]), "d"(v[2]), "d"(v[3]) : "memory");
}

// ---- thin-K kernel: K <= 64, N <= 32 -----------------------------------
//
// One k-block per problem, so every slice is loaded once per 128-row tile
// and all S(S+1)/2 slice products go into per-level TMEM accumulators
// (level l at columns l*32 of a buffer; two buffers alternate between tiles).
// A level sums at most S products of 64 K-elements, below 2^24, so no drains
// are needed mid-tile: the drain warps read the levels and recombine them,
// in integers up to six slices, with FP64 Horner steps beyond.  The k-block is TBK = 64
// (128-byte swizzled rows) or, for K <= 32, TBK = 32 (64-byte rows): slices
// are padded to the k-block, so short K (a virtual block of ~30 orbitals)
// streams half the bytes with the narrow block.
constexpr int kThinBN = 32;
constexpr int kThinBufs = 3;        // accumulator buffers (at most; S (S <= 5) levels of 32 columns each)
constexpr int kThinDrainWarps = 4 * kThinBufs;  // one group of four (one per TMEM lane quarter) per buffer
constexpr int kThinThreads = 64 + 32 * kThinDrainWarps;

template <int TBK>
struct ThinSmem {
  static constexpr int kSlots = 10 * (BK / TBK);  // ring of (A slice, B slice) pairs, 200 KB of them
  alignas(1024) __nv_bfloat16 a[kSlots][BM * TBK];
  alignas(1024) __nv_bfloat16 b[kSlots][kThinBN * TBK];
  uint64_t full[kSlots], empty[kSlots], accfull[kThinBufs], accempty[kThinBufs], done;
  uint32_t tmem_base;
};

// Drain of one thin tile, first NC columns (NC covers ncol): Horner over the
// levels in exact int64 fixed point, Y = sum_l X_l 2^(8 (L - l)), from level
// 0 up (|X_l| <= 7 * 64 * 2^14 < 2^23, so |Y| < 2^63 for L <= 5; S = 7 keeps
// the FP64 recombination); the accumulator buffer is released before the
// results are rounded, scaled and stored (in integers, as in the k-stationary
// kernel: the nine thin launches of a CCSD iteration at o = 48, v = 240 take
// 546 us with a conversion and a multiply to each output, 475 so).
// ea: the row's exponent, ebl: the lane's column's, both loaded by the caller
// before it waited for the accumulator (their latency hidden behind the wait).
// Stores of one drained row: v[j] * 2^(its exponent), columns < ncol.  All
// lanes of the warp call it.
__device__ __forceinline__ double plain_value(long long x, int ex) { return scaled_int(x, ex); }
__device__ __forceinline__ double plain_value(double x, int ex) { return scaled(x, ex); }

template <int NC, typename T>
__device__ __forceinline__ void thin_store(const T (&v)[NC], int L, int ncol, const DevProblem& pr, int row,
                                           int ea, int ebl) {
  const int64_t ld = pr.ldc;
  double* crow = pr.C + (int64_t)row * ld;
  const int e0 = ea + 1023 - 2 * 1022 - 14 - (L <= 5 ? 8 * L : 0);  // the int64 path carries 2^(8L)
  const bool real = row < pr.M;
  if (plain_exponents(ea, ebl, e0 - ea)) {
    const bool pairs = (((uintptr_t)pr.C | (uintptr_t)(ld * 8)) & 15) == 0;
#pragma unroll
    for (int j = 0; j < NC; j += 2) {
      if (j >= ncol) break;
      const int ex0 = e0 + __shfl_sync(0xffffffffu, ebl, j), ex1 = e0 + __shfl_sync(0xffffffffu, ebl, j + 1);
      const double x[2] = {plain_value(v[j], ex0), plain_value(v[j + 1], ex1)};
      if (!real) continue;
      if (pairs && j + 1 < ncol) {
        store_vec(crow + j, x);
      } else {
        crow[j] = x[0];
        if (j + 1 < ncol) crow[j + 1] = x[1];
      }
    }
    return;
  }
#pragma unroll
  for (int j = 0; j < NC; ++j) {
    if (j >= ncol) break;
    int ex = e0 + __shfl_sync(0xffffffffu, ebl, j);
    ex = ex < 1 ? 1 : (ex > 2046 ? 2046 : ex);
    if (real) crow[j] = (double)v[j] * __longlong_as_double((long long)ex << 52);
  }
}

template <int NC>
__device__ __forceinline__ void thin_drain(uint32_t tb, int L, int ncol, const DevProblem& pr, int row,
                                           uint64_t* accempty, int lane, int ea, int ebl) {
  if (L <= 5) {
    long long Y[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) Y[j] = 0;
    if (NC == 8 && L <= 3) {
      // at most four levels of 8 columns (the usual thin tile: an occupied
      // block of about 6): every load issued, then one wait
      uint32_t rb[4][8];
#pragma unroll
      for (int l = 0; l < 4; ++l)
        if (l <= L) tmem_ld8(tb + (uint32_t)(l * kThinBN), rb[l]);
      tmem_wait_ld();
#pragma unroll
      for (int l = 0; l < 4; ++l)
        if (l <= L) {
#pragma unroll
          for (int j = 0; j < 8; ++j)
            if (j < ncol) Y[j] = Y[j] * 256 + (long long)__float2int_rn(__uint_as_float(rb[l][j]));
        }
    } else {
      for (int l = 0; l <= L; ++l) {
        uint32_t r[NC];
        if (NC == 8) {
          tmem_ld8(tb + (uint32_t)(l * kThinBN), r);
        } else {
#pragma unroll
          for (int h = 0; h < NC / 16; ++h)
            tmem_ld16(tb + (uint32_t)(l * kThinBN + 16 * h), *reinterpret_cast<uint32_t(*)[16]>(r + 16 * h));
        }
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < NC; ++j)
          if (j < ncol) Y[j] = Y[j] * 256 + (long long)__float2int_rn(__uint_as_float(r[j]));
      }
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(accempty);
    thin_store<NC>(Y, L, ncol, pr, row, ea, ebl);
  } else {
    double v[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) v[j] = 0.0;
    for (int l = L; l >= 0; --l) {
      uint32_t r[NC];
      if (NC == 8) {
        tmem_ld8(tb + (uint32_t)(l * kThinBN), r);
      } else {
#pragma unroll
        for (int h = 0; h < NC / 16; ++h)
          tmem_ld16(tb + (uint32_t)(l * kThinBN + 16 * h), *reinterpret_cast<uint32_t(*)[16]>(r + 16 * h));
      }
      tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < NC; ++j)
        if (j < ncol) v[j] = v[j] * 0x1.0p-8 + (double)__uint_as_float(r[j]);
    }
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(accempty);
    thin_store<NC>(v, L, ncol, pr, row, ea, ebl);
  }
}

template <int TBK>
__global__ void __launch_bounds__(kThinThreads, 1) split_thin_kernel(const GemmParams P) {
  static_assert(TBK == 32 || TBK == 64, "thin k-block");
  using Sm = ThinSmem<TBK>;
  constexpr int kThinSlots = Sm::kSlots;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  Sm& sm = *reinterpret_cast<Sm*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  begin_dependent();
  const int S = P.S, L = P.L;
  // a stage holds one tile's S (A slice, B slice) pairs, the B slices back
  // to back, behind one full and one empty barrier
  const int stages = kThinSlots / S;
  constexpr uint32_t kTx = (BM + kThinBN) * TBK * 2;
  constexpr uint32_t kCols = 512;
  if (threadIdx.x == 0) {
    for (int i = 0; i < stages; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], 1);
    }
    for (int b = 0; b < kThinBufs; ++b) {
      mbar_init(&sm.accfull[b], 1);
      mbar_init(&sm.accempty[b], 4);
    }
    mbar_init(&sm.done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;
  const uint32_t buf_cols = (uint32_t)(S * kThinBN);
  // accumulator buffers in the 512 columns: three for S <= 5, two above
  const int nbuf = min(kThinBufs, (int)(kCols / buf_cols));

  if (warp == 0) {
    if (lane == 0) {
      int st = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < P.total_tiles && ok; tile += gridDim.x) {
        const TileInfo ti = decode_tile<kThinBN>(P, tile);
        const CUtensorMap* ma = P.maps + 2 * ti.p;
        const CUtensorMap* mb = P.maps + 2 * ti.p + 1;
        if (!mbar_wait(&sm.empty[st], phase ^ 1, P.err, 11)) {
          ok = false;
          break;
        }
        mbar_expect_tx(&sm.full[st], (uint32_t)S * kTx);
        for (int s = 0; s < S; ++s) {
          tma_load_3d(sm.a[st * S + s], ma, &sm.full[st], 0, ti.m0, s);
          tma_load_3d(sm.b[st * S + s], mb, &sm.full[st], 0, ti.n0, s);
        }
        if (++st == stages) {
          st = 0;
          phase ^= 1;
        }
      }
      for (int i = 0; i < stages; ++i) {
        if (--st < 0) {
          st = stages - 1;
          phase ^= 1;
        }
        long long t0 = clock64();
        while (!mbar_try_wait(&sm.full[st], phase) && !mbar_try_wait(&sm.empty[st], phase)) {
          if (clock64() - t0 > kWaitCycles) {
            atomicCAS(P.err, 0, 15);
            break;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      int st = 0, buf = 0;
      uint32_t phase = 0, aphase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < P.total_tiles && ok; tile += gridDim.x) {
        if (!mbar_wait(&sm.full[st], phase, P.err, 13)) break;
        if (!mbar_wait(&sm.accempty[buf], aphase ^ 1, P.err, 12)) break;
        tc_fence_after();
        // one UMMA per A slice s and K step over B slices 1 .. S + 1 - s
        // (N = 32 (S + 1 - s)) with D at column 32 (s - 1): product (s, t)
        // lands in level s + t - 2's columns; the first (s = 1, k = 0) spans
        // every level and starts them from zero
        const int base = st * S;
        const uint32_t bs = smem_u32(sm.b[base]);
        const uint64_t b0 = TBK == 64 ? sdesc(bs) : sdesc64(bs);
        for (int s = 1; s <= S; ++s) {
          const uint32_t d = tmem + (uint32_t)buf * buf_cols + (uint32_t)((s - 1) * kThinBN);
          const uint32_t as = smem_u32(sm.a[base + s - 1]);
          const uint64_t a0 = TBK == 64 ? sdesc(as) : sdesc64(as);
          const uint32_t idesc = idesc_bf16_n(kThinBN * (S + 1 - s));
#pragma unroll
          for (int k = 0; k < TBK / 16; ++k)
            umma(d, a0 + (uint64_t)(k * 2), b0 + (uint64_t)(k * 2), idesc, (s == 1 && k == 0) ? 0u : 1u);
        }
        umma_commit(&sm.empty[st]);
        umma_commit(&sm.accfull[buf]);
        if (++st == stages) {
          st = 0;
          phase ^= 1;
        }
        if (++buf == nbuf) {
          buf = 0;
          aphase ^= 1;
        }
      }
      umma_commit(&sm.done);
      mbar_wait(&sm.done, 0, P.err, 16);
    }
  } else {
    // nbuf drain groups of four warps: group g drains this CTA's tiles g,
    // g + nbuf, g + 2 nbuf, ... -- always from accumulator buffer g -- so
    // that nbuf tiles drain at once (a drain, with its exponent loads, TMEM
    // reads and scattered row stores, takes longer than a tile's MMAs); a
    // group without a buffer (S > 5) has no tiles
    const int group = (warp - 2) >> 2;
    const int quarter = warp & 3;
    const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
    const int buf = group;
    uint32_t aphase = 0;
    for (int tile = blockIdx.x + group * (int)gridDim.x; group < nbuf && tile < P.total_tiles;
         tile += nbuf * (int)gridDim.x) {
      const TileInfo ti = decode_tile<kThinBN>(P, tile);
      const DevProblem& pr = P.probs[ti.p];
      // only the tile's real columns are read and combined: a drain sized
      // for 8, 16 or 32 columns (the thin problems of a block-sparse
      // contraction often have an occupied block of ~6 as N)
      const int ncol = min(kThinBN, pr.N - ti.n0);
      const int row = ti.m0 + quarter * 32 + lane;
      const int ea = row < pr.M ? pr.eA[row] : 0;
      const int ebl = lane < ncol ? pr.eB[lane] : 0;  // thin tiles start at column 0
      int w_ok = lane == 0 ? (int)mbar_wait(&sm.accfull[buf], aphase, P.err, 14) : 1;
      w_ok = __shfl_sync(0xffffffffu, w_ok, 0);
      if (!w_ok) break;
      __syncwarp();
      tc_fence_after();
      const uint32_t tb = tmem + lane_addr + (uint32_t)buf * buf_cols;
      if (ncol <= 8) thin_drain<8>(tb, L, ncol, pr, row, &sm.accempty[buf], lane, ea, ebl);
      else if (ncol <= 16) thin_drain<16>(tb, L, ncol, pr, row, &sm.accempty[buf], lane, ea, ebl);
      else thin_drain<32>(tb, L, ncol, pr, row, &sm.accempty[buf], lane, ea, ebl);
      aphase ^= 1;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
  }
}

// ---- k-stationary kernel: 64-column output tiles, any slice count -------------
//
// The pair-by-pair kernel above streams a k-block's A and B slices once per
// slice pair that uses them (2 S (S + 1) / 2 tile loads per k-block).  Here
// every k-block's S A slices and S B slices are loaded once and all
// S (S + 1) / 2 products are issued from there into per-level TMEM accumulators of 64 columns: B slices
// sit back to back in the stage, so one instruction of A slice s covers
// every level it contributes to (product (s, t) lands in level s + t - 2's
// columns when D starts at level s - 1's).
//
// What bounds it is shared memory: at S = 4 a K step of 16 reads 16 KB of A
// and 20 KB of B and TMA writes 24 KB, 60 KB at 128 bytes a clock against 320
// clocks of MMAs.  9216 x 768 x 4096 runs at 1483 TFLOP/s of slice products
// at S = 4 (66% of the tensor pipe; the bound above is 68%), 1366 at 5, 1332
// at 6 and 1190 at 7, where the pair-by-pair kernel reaches 940.
//
// A k-block is 64 elements up to four slices (two stages or more); beyond
// only one such stage would fit, so 32 (at S = 4 that took 453 us, and 64 took
// 441).
//
// TMEM holds eight such accumulators.  Level l sums l + 1 products of at
// most 2^14 per element, so 1024 / (l + 1) elements fit below 2^24 and are
// exact.  The high levels, which fill up first, have two buffers and are
// drained every few k-blocks behind the MMAs of the next ones; the low
// ones have one and are drained more rarely, the MMAs of a k-block starting
// with its high levels while they are.  S = 4: four high levels; 5: three
// and two low ones; 6: two and four; 7: one and six.
//
// The drains add the levels exactly into 64-bit sums (levels apart by 2^8;
// two sums 2^32 apart from six slices on), which become one FP64 value per
// output at the end of a tile.  That end is what bounds short K: an SM issues
// 1.8 FP64 instructions a clock, so each one to an output is 2.4 us of a
// tile.  So the values are rounded and scaled by integer instructions (from
// six slices on one FP64 multiply-add is left; near the ends of the FP64
// range the plain conversion and multiply), full rows of four go out in one
// store, and warps without real elements skip their part.  Conversions,
// multiplies and 8-byte stores / so, with the operand splits: 2000 x 2000 x 66
// 62.5 / 29.4 us at 4 slices and 99.6 / 42.4 at 6, 400 x 400 x 400 26.1 / 17.5
// and 44.5 / 27.8, 2000 x 2000 x 3200 279 / 248 and 578 / 529.
constexpr int kKsBN = 64;
constexpr int ks_bk(int S) { return S <= 4 ? 64 : 32; }  // elements of a k-block
constexpr int kKsDrainWarps = 8;     // 4 TMEM lane quarters x 2 column halves
constexpr int kKsThreads = 64 + 32 * kKsDrainWarps;
constexpr int kKsMinS = 2, kKsMaxS = 7;

template <int S>
struct KsCfg {
  static constexpr int L = S - 1;
  static constexpr int kHi = S <= 4 ? S : 8 - S;  // levels with two buffers
  static constexpr int kLo = S - kHi;             // levels with one (kLo + 2 kHi <= 8)
  static constexpr int kBK = ks_bk(S);
  // k-blocks of an accumulator (a doubled leading digit counts as a product more)
  static constexpr int kHiBlocks = 1024 / S / kBK, kHiBlocksDbl = 1024 / (S + 1) / kBK;
  static constexpr int kLoBlocks = kLo ? 1024 / (kLo ? kLo : 1) / kBK : 1, kLoBlocksDbl = kLo ? 1024 / (kLo + 1) / kBK : 1;
  static constexpr int kStageBytes = S * (BM + kKsBN) * kBK * 2;
  static constexpr int kStages = (220 * 1024 / kStageBytes) < 8 ? 220 * 1024 / kStageBytes : 8;
  static constexpr int kCut = S <= 5 ? 0 : S - 4;  // levels below this go to the upper sum
  // the drains' level loops: unrolled, their TMEM reads overlap the sums
  // before (S = 6: 978 instead of 1019 us, although at 168 registers it spills
  // 224 bytes and S = 7 60); at S = 4, faster without, it would spill too
  static constexpr int kUnroll = S <= 4 ? 1 : S;
};

template <int S>
struct KsSmem {
  using Cfg = KsCfg<S>;
  struct alignas(1024) Stage {
    __nv_bfloat16 a[S][BM * Cfg::kBK];
    __nv_bfloat16 b[S][kKsBN * Cfg::kBK];
  };
  Stage st[Cfg::kStages];
  uint64_t full[Cfg::kStages], empty[Cfg::kStages], hifull[2], hiempty[2], lofull, loempty, done;
  uint32_t tmem_base;
};

template <int S>
__global__ void __launch_bounds__(kKsThreads, 1) split_ks_kernel(const GemmParams P) {
  using Cfg = KsCfg<S>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  KsSmem<S>& sm = *reinterpret_cast<KsSmem<S>*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  begin_dependent();
  constexpr int L = Cfg::L, kStages = Cfg::kStages;
  constexpr uint32_t kCols = 512;
  // accumulator columns: the low levels, then the two buffers of the high ones
  constexpr uint32_t kHiCol = Cfg::kLo * kKsBN, kHiCols = Cfg::kHi * kKsBN;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(&sm.full[i], 1);
      mbar_init(&sm.empty[i], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.hifull[b], 1);
      mbar_init(&sm.hiempty[b], kKsDrainWarps);
    }
    mbar_init(&sm.lofull, 1);
    mbar_init(&sm.loempty, kKsDrainWarps);
    mbar_init(&sm.done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                 "r"(kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp == 0) {
    // ---------------- TMA producer: a k-block's slices ----------------
    if (lane == 0) {
      int st = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < P.total_tiles && ok; tile += gridDim.x) {
        const TileInfo ti = decode_tile<kKsBN>(P, tile);
        const CUtensorMap* ma = P.maps + 2 * ti.p;
        const CUtensorMap* mb = P.maps + 2 * ti.p + 1;
        for (int kb = ti.kb0; kb < ti.kb0 + ti.nkb; ++kb) {
          if (!mbar_wait(&sm.empty[st], phase ^ 1, P.err, 21)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&sm.full[st], (uint32_t)Cfg::kStageBytes);
#pragma unroll
          for (int s = 0; s < S; ++s) {
            tma_load_3d(sm.st[st].a[s], ma, &sm.full[st], kb * Cfg::kBK, ti.m0, s);
            tma_load_3d(sm.st[st].b[s], mb, &sm.full[st], kb * Cfg::kBK, ti.n0, s);
          }
          if (++st == kStages) {
            st = 0;
            phase ^= 1;
          }
        }
      }
      // wait (bounded) for the copies this warp issued to land before leaving
      for (int i = 0; i < kStages; ++i) {
        if (--st < 0) {
          st = kStages - 1;
          phase ^= 1;
        }
        long long t0 = clock64();
        while (!mbar_try_wait(&sm.full[st], phase) && !mbar_try_wait(&sm.empty[st], phase)) {
          if (clock64() - t0 > kWaitCycles) {
            atomicCAS(P.err, 0, 25);
            break;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int st = 0, hb = 0;
      uint32_t phase = 0, hphase = 0, lphase = 0;
      bool ok = true;
      // stage descriptors: stage 0's plus the stage offset in 16-byte units
      // (the address field holds shared-memory address / 16, below 2^14)
      const auto desc = [](const void* p) { return Cfg::kBK == 64 ? sdesc(smem_u32(p)) : sdesc64(smem_u32(p)); };
      const uint64_t ad0 = desc(sm.st[0].a), bd0 = desc(sm.st[0].b);
      constexpr uint64_t kStep = (uint64_t)sizeof(typename KsSmem<S>::Stage) >> 4;
      constexpr uint64_t kAStep = (uint64_t)(BM * Cfg::kBK * 2) >> 4, kBStep = (uint64_t)(kKsBN * Cfg::kBK * 2) >> 4;
      for (int tile = blockIdx.x; tile < P.total_tiles && ok; tile += gridDim.x) {
        const TileInfo ti = decode_tile<kKsBN>(P, tile);
        const int nkb = ti.nkb, hmax = ti.dbl ? Cfg::kHiBlocksDbl : Cfg::kHiBlocks,
                  lmax = ti.dbl ? Cfg::kLoBlocksDbl : Cfg::kLoBlocks;
        int hn = 0, ln = 0;  // k-blocks in the current accumulators
        for (int kb = 0; kb < nkb; ++kb) {
          if (hn == 0 && !mbar_wait(&sm.hiempty[hb], hphase ^ 1, P.err, 22)) {
            ok = false;
            break;
          }
          if (!mbar_wait(&sm.full[st], phase, P.err, 23)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t as = ad0 + (uint64_t)st * kStep, bs = bd0 + (uint64_t)st * kStep;
          // high levels kLo .. L: A slice s with B slices max(1, kLo + 2 - s) .. S + 1 - s
          const uint32_t hcol = tmem + kHiCol + (uint32_t)hb * kHiCols;
#pragma unroll
          for (int s = 1; s <= S; ++s) {
            const int l0 = s - 1 > Cfg::kLo ? s - 1 : Cfg::kLo;  // first high level of slice s
            const int t0 = l0 + 2 - s;
#pragma unroll
            for (int k = 0; k < Cfg::kBK / 16; ++k)
              umma(hcol + (uint32_t)((l0 - Cfg::kLo) * kKsBN), as + (uint64_t)(s - 1) * kAStep + (uint64_t)(k * 2),
                   bs + (uint64_t)(t0 - 1) * kBStep + (uint64_t)(k * 2), idesc_bf16_n(kKsBN * (S - l0)),
                   (s == 1 && k == 0 && hn == 0) ? 0u : 1u);
          }
          if (Cfg::kLo == 0) umma_commit(&sm.empty[st]);
          if (++hn == hmax || kb == nkb - 1) {
            umma_commit(&sm.hifull[hb]);
            hn = 0;
            if (++hb == 2) {
              hb = 0;
              hphase ^= 1;
            }
          }
          if constexpr (Cfg::kLo > 0) {
            if (ln == 0) {
              if (!mbar_wait(&sm.loempty, lphase ^ 1, P.err, 27)) {
                ok = false;
                break;
              }
              tc_fence_after();
            }
            // low levels 0 .. kLo - 1: A slice s with B slices 1 .. kLo + 1 - s,
            // at most 256 columns to an instruction
#pragma unroll
            for (int s = 1; s <= Cfg::kLo; ++s) {
              const int n = Cfg::kLo + 1 - s;
#pragma unroll
              for (int k = 0; k < Cfg::kBK / 16; ++k)
#pragma unroll
                for (int c = 0; c < n; c += 4)
                  umma(tmem + (uint32_t)((s - 1 + c) * kKsBN), as + (uint64_t)(s - 1) * kAStep + (uint64_t)(k * 2),
                       bs + (uint64_t)c * kBStep + (uint64_t)(k * 2), idesc_bf16_n(kKsBN * (n - c < 4 ? n - c : 4)),
                       (s == 1 && k == 0 && ln == 0) ? 0u : 1u);
            }
            if (++ln == lmax || kb == nkb - 1) {
              umma_commit(&sm.lofull);
              ln = 0;
              lphase ^= 1;
            }
            umma_commit(&sm.empty[st]);
          }
          if (++st == kStages) {
            st = 0;
            phase ^= 1;
          }
        }
      }
      umma_commit(&sm.done);
      mbar_wait(&sm.done, 0, P.err, 26);
    }
  } else {
    // ---------------- drain: exact 64-bit level recombination ----------------
    const int quarter = warp & 3;               // TMEM lanes this warp may read
    const int half = (warp - 2) >> 2;           // which 32 of the 64 columns
    const uint32_t base = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 32);
    int hb = 0;
    uint32_t hphase = 0, lphase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < P.total_tiles && ok; tile += gridDim.x) {
      const TileInfo ti = decode_tile<kKsBN>(P, tile);
      const int M = P.probs[ti.p].M, N = P.probs[ti.p].N;
      const int row = ti.m0 + quarter * 32 + lane, col0 = ti.n0 + half * 32;
      // a warp whose 32 x 32 elements lie outside the matrix only keeps the
      // accumulators turning
      const bool idle = ti.m0 + quarter * 32 >= M || col0 >= N;
      // the exponents, read ahead of the waits: the row's, and a column's to a lane
      const int ea = row < M ? P.probs[ti.p].eA[row] : 0;
      const int ebl = col0 + lane < N ? P.probs[ti.p].eB[col0 + lane] : 0;
      long long Y[32], U[Cfg::kCut ? 32 : 1];
#pragma unroll
      for (int j = 0; j < 32; ++j) Y[j] = 0;
      if (Cfg::kCut) {
#pragma unroll
        for (int j = 0; j < 32; ++j) U[Cfg::kCut ? j : 0] = 0;
      }
      // adds level l's 32 columns at col, weighted 2^(8 (L - l)) (below the
      // cut 2^(8 (kCut - 1 - l)) of the upper sum)
      auto add = [&](int l, uint32_t col) {
        if (idle) return;
        uint32_t r[2][16];
        tmem_ld16(base + col, r[0]);
        tmem_ld16(base + col + 16, r[1]);
        tmem_wait_ld();
        if (Cfg::kCut && l < Cfg::kCut) {
          const int w = 1 << (8 * (Cfg::kCut - 1 - l));
#pragma unroll
          for (int j = 0; j < 32; ++j)
            U[Cfg::kCut ? j : 0] += (long long)__float2int_rn(__uint_as_float(r[j >> 4][j & 15])) * w;
        } else {
          const long long w = 1ll << (8 * (L - l));
#pragma unroll
          for (int j = 0; j < 32; ++j) Y[j] += (long long)__float2int_rn(__uint_as_float(r[j >> 4][j & 15])) * w;
        }
      };
      auto wait = [&](uint64_t* bar, uint32_t parity) {
        int w_ok = lane == 0 ? (int)mbar_wait(bar, parity, P.err, 24) : 1;
        w_ok = __shfl_sync(0xffffffffu, w_ok, 0);
        __syncwarp();
        tc_fence_after();
        return w_ok != 0;
      };
      auto release = [&](uint64_t* bar) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar);
      };
      const int hmax = ti.dbl ? Cfg::kHiBlocksDbl : Cfg::kHiBlocks,
                  lmax = ti.dbl ? Cfg::kLoBlocksDbl : Cfg::kLoBlocks;
      int hn = 0, ln = 0;
      for (int kb = 0; kb < ti.nkb; ++kb) {
        if (++hn == hmax || kb == ti.nkb - 1) {
          if (!wait(&sm.hifull[hb], hphase)) {
            ok = false;
            break;
          }
#pragma unroll(Cfg::kUnroll)
          for (int l = Cfg::kLo; l <= L; ++l)
            add(l, kHiCol + (uint32_t)hb * kHiCols + (uint32_t)((l - Cfg::kLo) * kKsBN));
          release(&sm.hiempty[hb]);
          hn = 0;
          if (++hb == 2) {
            hb = 0;
            hphase ^= 1;
          }
        }
        if constexpr (Cfg::kLo > 0) {
          if (++ln == lmax || kb == ti.nkb - 1) {
            if (!wait(&sm.lofull, lphase)) {
              ok = false;
              break;
            }
#pragma unroll(Cfg::kUnroll)
            for (int l = 0; l < Cfg::kLo; ++l) add(l, (uint32_t)(l * kKsBN));
            release(&sm.loempty);
            ln = 0;
            lphase ^= 1;
          }
        }
      }
      if (!ok) break;
      if (idle) continue;
      const DevProblem& pr = P.probs[ti.p];
      const int64_t ld = pr.ksplit > 1 ? N : pr.ldc;
      double* cbase = (pr.ksplit > 1 ? pr.partial + (int64_t)ti.kc * M * N : pr.C) + col0;
      double* crow = cbase + (int64_t)row * ld;
      const uintptr_t at = (uintptr_t)cbase | (uintptr_t)(ld * 8);
      const int vec = (at & 31) == 0 ? 4 : (at & 15) == 0 ? 2 : 1;
      constexpr int kE = 1023 - 2 * 1022 - 14 - 8 * L;
      auto store = [&](auto is_plain) {
#pragma unroll
        for (int j0 = 0; j0 < 32; j0 += 4) {
          if (col0 + j0 >= N) break;
          double v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int j = j0 + i;
            int ex = ea + __shfl_sync(0xffffffffu, ebl, j) + kE;
            constexpr bool kPlain = decltype(is_plain)::value;
            if constexpr (kPlain && !Cfg::kCut) {
              v[i] = scaled_int(Y[j], ex);
            } else {
              double x;
              if constexpr (Cfg::kCut) {
                // U 2^32 + Y = V 2^32 + (2^52 + the low 32 bits of Y), the
                // bracket a double's bits as it stands; V is below 2^53
                const long long V = U[j] + (Y[j] >> 32) - (1 << 20);
                x = __fma_rn(kPlain ? scaled_int(V, 1023) : (double)V, 0x1.0p32,
                             __hiloint2double(0x43300000, (int)(uint32_t)Y[j]));
              } else {
                x = (double)Y[j];
              }
              if constexpr (kPlain) {
                v[i] = scaled(x, ex);
              } else {
                ex = ex < 1 ? 1 : (ex > 2046 ? 2046 : ex);
                v[i] = x * __longlong_as_double((long long)ex << 52);
              }
            }
          }
          if (row >= M) continue;
          if (vec == 4 && col0 + j0 + 4 <= N) {
            store_vec(crow + j0, v);
          } else if (vec == 2 && col0 + j0 + 4 <= N) {
            store_vec(crow + j0, {v[0], v[1]});
            store_vec(crow + j0 + 2, {v[2], v[3]});
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (col0 + j0 + i < N) crow[j0 + i] = v[i];
          }
        }
      };
      if (plain_exponents(ea, ebl, kE)) store(std::true_type());
      else store(std::false_type());
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
  }
}

// Fixed-order sum of the split-K partial contributions into C.
__global__ void __launch_bounds__(256) split_reduce_kernel(const DevProblem* __restrict__ probs,
                                                           const int* __restrict__ red_prob,
                                                           const int64_t* __restrict__ red_first, int nred,
                                                           int64_t total) {
  begin_dependent();
  dev::split_reduce_body<false>(probs, red_prob, red_first, nred, total, blockIdx.x, gridDim.x);
}

// Rows up to this length go a warp to a row in plans of few rows (both
// operands' rows fit one wave of the CTA-per-row kernel), up to kShortRow in
// others: a warp walks a long row 64 elements at a time (a plan of 975 rows
// of 900 at 4 slices: 52.1 us with a warp to a row, 45.8 with a CTA; 800 rows
// of 400: 35.5 and 33.5).
constexpr int64_t kFewRows = 152 * 8;
constexpr int64_t kFewShortRow = 128;

// Operand splits (dev::row_exponent_body, dev::digits_body, dev::short_rows_body).
__global__ void __launch_bounds__(256) row_exponent_kernel(const SplitRowSet* __restrict__ sets, int nsets,
                                                           int64_t first, int64_t end) {
  begin_dependent();
  __shared__ uint32_t red[8];
  dev::row_exponent_body<false>(sets, nsets, first, end, blockIdx.x, gridDim.x, red);
}

__global__ void __launch_bounds__(256) digits_kernel(const SplitRowSet* __restrict__ sets, int nsets,
                                                     int64_t first, int64_t end, int S) {
  begin_dependent();
  dev::digits_body<false>(sets, nsets, first, end, S, blockIdx.x, gridDim.x);
}

template <bool kFour>
__global__ void __launch_bounds__(256, kFour ? 3 : 4)
    split_rows_kernel(const SplitRowSet* __restrict__ sets, int nsets, int64_t first, int64_t end, int S) {
  begin_dependent();
  __shared__ uint32_t red[8];
  dev::split_rows_body<false, kFour>(sets, nsets, first, end, S, blockIdx.x, gridDim.x, red);
}

__global__ void __launch_bounds__(256) split_short_rows_kernel(const SplitRowSet* __restrict__ sets, int nsets,
                                                               int64_t first, int64_t end, int S, int lg) {
  begin_dependent();
  dev::short_rows_body<false>(sets, nsets, first, end, S, lg, blockIdx.x, gridDim.x);
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    cudaDriverEntryPointQueryResult q;
    void* p = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  }
  return fn;
}

int encode_slices(CUtensorMap* map, const __nv_bfloat16* base, int64_t S, int64_t rows, int64_t Kp, int box_rows,
                  int box_k = BK) {
  auto enc = get_encode();
  if (!enc) return fail(GBX_ECUDA, "cuTensorMapEncodeTiled unavailable");
  cuuint64_t dims[3] = {(cuuint64_t)Kp, (cuuint64_t)rows, (cuuint64_t)S};
  cuuint64_t strides[2] = {(cuuint64_t)(Kp * 2), (cuuint64_t)(rows * Kp * 2)};
  cuuint32_t box[3] = {(cuuint32_t)box_k, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, (void*)base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, box_k == BK ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(GBX_ECUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return GBX_OK;
}

}  // namespace

// Output tile width of a problem: 64 columns, the k-stationary kernel.
// gbx_split_set_width() and the autotuners may take another (the
// pair-by-pair kernel).
static int g_width_override = 0;

int choose_width() { return g_width_override ? g_width_override : kKsBN; }

// The k-stationary kernel's exact 64-bit sums: 2^(14 + 24) a level sum and
// element from four slices on, up to S products to a level, one bit more for
// doubled digits.
int64_t ks_max_k(int S) { return S <= 4 ? 1 << 24 : 1 << 22; }
// At five slices they are one sum each, 2^(14 + 32) an element: longer rows
// are cut into ranges (as rows are where output tiles are few).
constexpr int64_t kFiveRange = 1 << 15;

struct SplitLaunch {  // the problems of one output tile width
  int bn = 0;
  DevProblem* d_probs = nullptr;
  int* d_tile_first = nullptr;
  CUtensorMap* d_maps = nullptr;
  int nprob = 0, total_tiles = 0;
  // host copies (merged launches of the persistent iteration program)
  std::vector<DevProblem> hp;
  std::vector<CUtensorMap> hm;
  std::vector<int> hfirst;
};

struct SplitPlan {
  int S = 0, L = 0;
  std::vector<SplitProblem> host;
  std::vector<int> width;  // per problem
  std::vector<int> thin;  // per problem: 0, or the thin-K kernel with a 64 (1) or 32 (2) element k-block
  std::vector<int> kb;    // per problem: k-block
  unsigned char* d_persist = nullptr;    // slices and exponents of constant plan operands
  unsigned char* d_own_arena = nullptr;  // the per-run region when no arena was given
  // row sets of one kernel: those of the plan's packed A, then those of its
  // packed B (first_row counts on), so one launch covers either or both
  struct Rows {
    SplitRowSet* d = nullptr;
    int n[2] = {0, 0};
    int64_t items[2] = {0, 0};
  };
  Rows lng;   // (row, K chunk) work items
  Rows mid;   // one CTA per row
  Rows shrt;  // a warp or less per row
  bool mid_four = false;  // a medium row of 2049 .. 4096 elements
  int short_lg = 3;       // log2 of a short row's lanes: the longest row's elements in one step, or 5
  int nsets = 0;
  // exponent words of the long rows, reset before a split of A (1), B (2) or both (3)
  std::vector<std::pair<void*, size_t>> exp_ranges[4];
  std::vector<SplitLaunch> launches;
  DevProblem* d_all = nullptr;  // every problem, for the split-K reduction
  int* d_err = nullptr;
  int* d_red_prob = nullptr;
  int64_t* d_red_first = nullptr;
  int nred = 0;
  int64_t red_total = 0;
  double bytes = 0.0;
  ~SplitPlan() {
    dev_free(d_red_prob);
    dev_free(d_red_first);
    dev_free(d_persist);
    dev_free(d_own_arena);
    dev_free(lng.d);
    dev_free(mid.d);
    dev_free(shrt.d);
    dev_free(d_all);
    for (auto& l : launches) {
      dev_free(l.d_probs);
      dev_free(l.d_tile_first);
      dev_free(l.d_maps);
    }
    dev_free(d_err);
  }
};

template <int BN>
int set_smem_attr() {
  const size_t smem = sizeof(Smem<BN>) + 1024;
  GBX_CUDA(cudaFuncSetAttribute(split_gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  return GBX_OK;
}

template <int... I>
int set_ks_attr(std::integer_sequence<int, I...>) {
  for (cudaError_t e : {cudaFuncSetAttribute(split_ks_kernel<kKsMinS + I>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(sizeof(KsSmem<kKsMinS + I>) + 1024))...})
    GBX_CUDA(e);
  return GBX_OK;
}

namespace {

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

// Where every buffer of a split plan lives.  Region 0 persists with the plan
// (slices and exponents of constant plan operands, split once); region 1 is
// rewritten by every run (the other operands' slices and exponents, split-K
// partial sums) and may be an arena shared with other plans.  Offsets are in
// elements of each region's slice, exponent and partial-sum sub-buffers.
struct SplitLayout {
  struct Prob {
    int bn = 0;
    bool thin = false, ks_kernel = false;
    int kb = BK;  // k-block: 64; 32 from five slices on in the k-stationary kernel and for thin problems with K <= 32
    int64_t Mp = 0, Np = 0, Kp = 0;
    int ra = 0, rb = 0;      // region of the GEMM's A and B slices
    int64_t sa = 0, sb = 0;  // slice offsets
    int64_t ea = 0, eb = 0;  // exponent offsets
    int ks = 1, per = 0;     // K split and k-blocks per range
    int64_t part = -1;       // partial-sum offset (region 1), -1 = none
  };
  std::vector<Prob> p;
  int64_t slices[2] = {0, 0}, exps[2] = {0, 0}, part = 0;
  size_t exps_at(int r) const { return align256(2 * (size_t)slices[r]); }
  size_t part_at() const { return exps_at(1) + align256(4 * (size_t)exps[1]); }
  size_t bytes(int r) const {
    size_t b = exps_at(r) + align256(4 * (size_t)exps[r]);
    if (r == 1) b += align256(8 * (size_t)part);
    return (r == 0 && slices[0] == 0 && exps[0] == 0) || (r == 1 && slices[1] == 0 && exps[1] == 0 && part == 0)
               ? 0
               : b;
  }
};

int split_layout(const std::vector<SplitProblem>& probs, int S, bool static_a, bool static_b, SplitLayout& L) {
  L = SplitLayout();
  int64_t out_tiles = 0;
  for (auto& q : probs) {
    if (q.M <= 0 || q.N <= 0 || q.K <= 0) return fail(GBX_EINVAL, "empty split problem");
    if (q.M >= (1ll << 30) || q.N >= (1ll << 30) || q.K >= (1ll << 30)) return fail(GBX_EUNSUPPORTED, "split problem too large");
    SplitLayout::Prob o;
    // thin-K problems (one k-block, at most 32 columns) take the thin kernel
    o.thin = q.K <= BK && q.N <= kThinBN && S <= 7;
    o.bn = o.thin ? kThinBN : (q.width ? q.width : choose_width());
    if (!o.thin && o.bn == kKsBN && q.K >= ks_max_k(S) / 2) o.bn = 128;
    o.ks_kernel = !o.thin && o.bn == kKsBN;
    if (!o.thin && o.bn != 32 && o.bn != 64 && o.bn != 128 && o.bn != 256)
      return fail(GBX_EINVAL, "split tile width %d", o.bn);
    o.Mp = (q.M + BM - 1) / BM * BM;
    o.Np = (q.N + o.bn - 1) / o.bn * o.bn;
    o.kb = o.ks_kernel ? ks_bk(S) : o.thin && q.K <= 32 ? 32 : BK;
    o.Kp = (q.K + o.kb - 1) / o.kb * o.kb;
    // the GEMM's A rows come from plan operand B when swapped
    const bool a_const = q.a_is_plan_b ? static_b : static_a;
    const bool b_const = q.a_is_plan_b ? static_a : static_b;
    o.ra = a_const ? 0 : 1;
    o.rb = b_const ? 0 : 1;
    o.sa = L.slices[o.ra];
    L.slices[o.ra] += S * q.M * o.Kp;
    o.sb = L.slices[o.rb];
    L.slices[o.rb] += S * q.N * o.Kp;
    o.ea = L.exps[o.ra];
    L.exps[o.ra] += o.Mp;
    o.eb = L.exps[o.rb];
    L.exps[o.rb] += o.Np;
    out_tiles += (o.Mp / BM) * (o.Np / o.bn);
    L.p.push_back(o);
  }
  for (size_t i = 0; i < probs.size(); ++i) {
    SplitLayout::Prob& o = L.p[i];
    const int nkb = (int)(o.Kp / o.kb);
    if (nkb < 1) return fail(GBX_EINVAL, "split problem without a k-block");
    // split K when the output tiles of all problems leave SMs idle; ranges are
    // whole exact-accumulation chunks: 16 k-blocks for the pair-by-pair
    // kernel, 256 elements for the k-stationary one (so few-tile problems --
    // matrix-vector shapes, small outputs with long K -- spread over many more
    // CTAs instead of walking K serially).  Only K that fills the accumulators
    // more than twice is worth the partial sums (two slices: 1024 elements; 3052
    // x 718 x 518 at 2 and 3 slices 53 and 60 us in ranges, 28 and 33 whole)
    const int chunk = o.ks_kernel ? 256 / o.kb : kChunkKb;
    const int least = o.ks_kernel ? std::max(chunk, 16 / S * BK / o.kb) : chunk;
    int ks = 1;
    if (!o.thin && out_tiles < kSplitFill && nkb > 2 * least) {
      int want = (int)((kSplitFill + out_tiles - 1) / out_tiles);
      ks = std::max(1, std::min(want, nkb / chunk));
    }
    if (o.ks_kernel && S == 5) ks = std::max(ks, (int)((probs[i].K + kFiveRange - 1) / kFiveRange));
    int per = (nkb + ks - 1) / ks;
    per = (per + chunk - 1) / chunk * chunk;
    ks = (nkb + per - 1) / per;
    o.ks = ks;
    o.per = per;
    if (ks > 1) {
      o.part = L.part;
      L.part += (int64_t)ks * probs[i].M * probs[i].N;
    }
  }
  return GBX_OK;
}

}  // namespace

int split_plan_sizes(const std::vector<SplitProblem>& probs, int slices, bool static_a, bool static_b,
                     size_t* persist_bytes, size_t* arena_bytes) {
  SplitLayout L;
  GBX_TRY(split_layout(probs, slices > 0 ? slices : 6, static_a, static_b, L));
  if (persist_bytes) *persist_bytes = L.bytes(0);
  if (arena_bytes) *arena_bytes = L.bytes(1);
  return GBX_OK;
}

int create_split_plan(const std::vector<SplitProblem>& probs, int slices, SplitPlan** out, const SplitMem* mem) {
  *out = nullptr;
  auto sp = std::make_unique<SplitPlan>();
  sp->S = slices > 0 ? slices : 6;
  if (sp->S < 2 || sp->S > 7) return fail(GBX_EINVAL, "split slices must be in [2, 7]");
  sp->L = sp->S - 1;
  sp->host = probs;
  const int S = sp->S;
  const bool static_a = mem && mem->static_a, static_b = mem && mem->static_b;
  SplitLayout lay;
  GBX_TRY(split_layout(probs, S, static_a, static_b, lay));
  for (auto& o : lay.p) {
    sp->width.push_back(o.bn);
    sp->thin.push_back(o.thin ? (o.kb == 32 ? 2 : 1) : 0);
    sp->kb.push_back(o.kb);
  }
  unsigned char* base[2] = {nullptr, nullptr};
  const size_t b0 = lay.bytes(0), b1 = lay.bytes(1);
  if (b0) {
    // constant operands are split once: their padding must read as zero
    GBX_TRY(dev_alloc((void**)&sp->d_persist, b0));
    GBX_CUDA(cudaMemset(sp->d_persist, 0, b0));
    base[0] = sp->d_persist;
  }
  if (b1) {
    if (mem && mem->arena) {
      base[1] = mem->arena;
    } else {
      GBX_TRY(dev_alloc((void**)&sp->d_own_arena, b1));
      GBX_CUDA(cudaMemset(sp->d_own_arena, 0, b1));
      base[1] = sp->d_own_arena;
    }
  }
  auto slice_ptr = [&](int r, int64_t off) { return (__nv_bfloat16*)base[r] + off; };
  auto exp_ptr = [&](int r, int64_t off) { return (int*)(base[r] + lay.exps_at(r)) + off; };
  double* part_base = b1 ? (double*)(base[1] + lay.part_at()) : nullptr;
  sp->bytes = (double)b0 + (double)b1;
  std::vector<SplitRowSet> sets[3][2];  // long, medium, short rows of plan A and B
  SplitPlan::Rows* const rows_of[3] = {&sp->lng, &sp->mid, &sp->shrt};
  int64_t all_rows = 0;
  for (const SplitProblem& p : probs) all_rows += p.M + p.N;
  const int64_t short_row = all_rows <= kFewRows ? kFewShortRow : kShortRow;
  struct ExpRange {
    int region, side;
    int64_t at, n;
  };
  std::vector<ExpRange> ranges;
  std::vector<DevProblem> dp;
  std::vector<CUtensorMap> maps;
  std::vector<int> red;
  std::vector<int64_t> red_first;
  int64_t red_total = 0;
  for (size_t i = 0; i < probs.size(); ++i) {
    const SplitProblem& p = probs[i];
    const SplitLayout::Prob& o = lay.p[i];
    const int bn = o.bn;
    // row sets are grouped by the plan operand they come from, so constant
    // plan operands can be split once
    SplitRowSet a{p.A, p.M, p.K, slice_ptr(o.ra, o.sa), p.M * o.Kp, o.Kp, exp_ptr(o.ra, o.ea), 0,
                  p.lda ? p.lda : p.K, p.K};
    SplitRowSet b{p.B, p.N, p.K, slice_ptr(o.rb, o.sb), p.N * o.Kp, o.Kp, exp_ptr(o.rb, o.eb), 0,
                  p.ldb ? p.ldb : p.K, p.K};
    SplitRowSet& to_a = p.a_is_plan_b ? b : a;  // rows that come from plan A
    SplitRowSet& to_b = p.a_is_plan_b ? a : b;
    if (p.dbl_from >= 0) (p.dbl_plan_b ? to_b : to_a).dbl = p.dbl_from;
    for (int side = 0; side < 2; ++side) {
      SplitRowSet& rs = side == 0 ? to_a : to_b;
      const int cls = p.K <= short_row ? 2 : p.K <= kMidRow ? 1 : 0;
      int64_t& items = rows_of[cls]->items[side];
      rs.first_row = items;
      items += cls == 0 ? rs.rows * ((p.K + kSplitChunk - 1) / kSplitChunk) : rs.rows;
      sets[cls][side].push_back(rs);
      const bool gemm_a = (side == 0) != p.a_is_plan_b;
      if (cls == 0) ranges.push_back({gemm_a ? o.ra : o.rb, side, gemm_a ? o.ea : o.eb, rs.rows});
    }
    while (p.K <= short_row && sp->short_lg < 5 && p.K > (2ll << sp->short_lg)) ++sp->short_lg;
    sp->mid_four = sp->mid_four || (p.K > 2048 && p.K <= 4096);
    DevProblem d;
    d.M = (int)p.M;
    d.N = (int)p.N;
    d.K = (int)p.K;
    d.nkb = (int)(o.Kp / o.kb);
    d.tiles_m = (int)(o.Mp / BM);
    d.tiles_n = (int)(o.Np / bn);
    d.ksplit = o.ks;
    d.kb_per_split = o.per;
    d.eA = exp_ptr(o.ra, o.ea);
    d.eB = exp_ptr(o.rb, o.eb);
    d.C = p.C;
    d.partial = nullptr;
    if (o.ks > 1) {
      d.partial = part_base + o.part;
      red.push_back((int)i);
      red_first.push_back(red_total);
      red_total += p.M * p.N;
    }
    d.ldc = p.ldc ? p.ldc : p.N;
    d.dbl = p.dbl_from >= 0 ? 1 : 0;
    dp.push_back(d);
    CUtensorMap ma, mb;
    // slices hold only the real rows: a tile's rows past M (or N) lie outside
    // the tensor and TMA fills them with zeros without reading memory
    GBX_TRY(encode_slices(&ma, slice_ptr(o.ra, o.sa), S, p.M, o.Kp, BM, o.kb));
    GBX_TRY(encode_slices(&mb, slice_ptr(o.rb, o.sb), S, p.N, o.Kp, bn, o.kb));
    maps.push_back(ma);
    maps.push_back(mb);
  }
  if (!red.empty()) {
    GBX_TRY(dev_alloc((void**)&sp->d_red_prob, sizeof(int) * red.size()));
    GBX_TRY(dev_alloc((void**)&sp->d_red_first, sizeof(int64_t) * red.size()));
    GBX_CUDA(cudaMemcpy(sp->d_red_prob, red.data(), sizeof(int) * red.size(), cudaMemcpyHostToDevice));
    GBX_CUDA(cudaMemcpy(sp->d_red_first, red_first.data(), sizeof(int64_t) * red.size(), cudaMemcpyHostToDevice));
    sp->nred = (int)red.size();
    sp->red_total = red_total;
  }
  sp->nsets = (int)probs.size();
  auto up = [&](const void* h, size_t bytes, void** d) -> int {
    if (bytes == 0) return GBX_OK;
    GBX_TRY(dev_alloc(d, bytes));
    GBX_CUDA(cudaMemcpy(*d, h, bytes, cudaMemcpyHostToDevice));
    return GBX_OK;
  };
  for (int cls = 0; cls < 3; ++cls) {
    SplitPlan::Rows& R = *rows_of[cls];
    std::vector<SplitRowSet> v = sets[cls][0];
    for (SplitRowSet rs : sets[cls][1]) {
      rs.first_row += R.items[0];
      v.push_back(rs);
    }
    for (int side = 0; side < 2; ++side) R.n[side] = (int)sets[cls][side].size();
    GBX_TRY(up(v.data(), sizeof(SplitRowSet) * v.size(), (void**)&R.d));
  }
  // the exponent words of a region lie one after another: a split that
  // writes all of them (every row's exponent, once the reset is done) resets
  // them as one range, another one each problem's
  int in_region[2] = {0, 0};
  for (const SplitLayout::Prob& o : lay.p) {
    const SplitProblem& p = probs[&o - lay.p.data()];
    in_region[o.ra] |= p.a_is_plan_b ? 2 : 1;
    in_region[o.rb] |= p.a_is_plan_b ? 1 : 2;
  }
  for (int sides = 1; sides < 4; ++sides)
    for (int r = 0; r < 2; ++r) {
      int64_t lo = -1, hi = 0;
      for (const ExpRange& x : ranges) {
        if (x.region != r || !(sides & (1 << x.side))) continue;
        if ((in_region[r] & ~sides) != 0) {
          sp->exp_ranges[sides].push_back({(void*)exp_ptr(r, x.at), sizeof(int) * (size_t)x.n});
          continue;
        }
        lo = lo < 0 ? x.at : std::min(lo, x.at);
        hi = std::max(hi, x.at + x.n);
      }
      if (lo >= 0) sp->exp_ranges[sides].push_back({(void*)exp_ptr(r, lo), sizeof(int) * (size_t)(hi - lo)});
    }
  GBX_TRY(up(dp.data(), sizeof(DevProblem) * dp.size(), (void**)&sp->d_all));
  // one launch per output tile width, plus one for the thin-K problems of
  // each k-block (bn 0: 64, bn 1: 32)
  for (int bn : {0, 1, 32, 64, 128, 256}) {
    std::vector<DevProblem> lp;
    std::vector<CUtensorMap> lm;
    std::vector<int> first;
    int tiles = 0;
    for (size_t i = 0; i < probs.size(); ++i) {
      if (bn <= 1 ? sp->thin[i] != bn + 1 : (sp->thin[i] || sp->width[i] != bn)) continue;
      lp.push_back(dp[i]);
      lm.push_back(maps[2 * i]);
      lm.push_back(maps[2 * i + 1]);
      first.push_back(tiles);
      tiles += dp[i].tiles_m * dp[i].tiles_n * dp[i].ksplit;
    }
    if (lp.empty()) continue;
    SplitLaunch L;
    L.bn = bn;
    L.nprob = (int)lp.size();
    L.total_tiles = tiles;
    GBX_TRY(up(lp.data(), sizeof(DevProblem) * lp.size(), (void**)&L.d_probs));
    GBX_TRY(up(first.data(), sizeof(int) * first.size(), (void**)&L.d_tile_first));
    GBX_TRY(up(lm.data(), sizeof(CUtensorMap) * lm.size(), (void**)&L.d_maps));
    L.hp = lp;
    L.hm = lm;
    L.hfirst = first;
    sp->launches.push_back(std::move(L));
  }
  GBX_TRY(dev_alloc((void**)&sp->d_err, sizeof(int)));
  GBX_CUDA(cudaMemset(sp->d_err, 0, sizeof(int)));
  GBX_TRY(set_smem_attr<32>());
  GBX_TRY(set_smem_attr<128>());
  GBX_TRY(set_smem_attr<256>());
  GBX_TRY(set_ks_attr(std::make_integer_sequence<int, kKsMaxS - kKsMinS + 1>()));
  GBX_CUDA(cudaFuncSetAttribute(split_thin_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(sizeof(ThinSmem<64>) + 1024)));
  GBX_CUDA(cudaFuncSetAttribute(split_thin_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(sizeof(ThinSmem<32>) + 1024)));
  *out = sp.release();
  return GBX_OK;
}

int split_operands(SplitPlan* sp, bool plan_a, bool plan_b, cudaStream_t st) {
  if (!sp || sp->nsets == 0) return GBX_OK;
  const int sides = (plan_a ? 1 : 0) | (plan_b ? 2 : 0);
  if (sides == 0) return GBX_OK;
  ProgRecorder* rec = prog_recording();
  const int S = sp->S;
  // the launch's part of a class: its first set, set count and work items
  const auto part = [&](const SplitPlan::Rows& R, int lg) {
    PaSplitSets a;
    a.sets = R.d + (plan_a ? 0 : R.n[0]);
    a.first = plan_a ? 0 : R.items[0];
    a.end = R.items[0] + (plan_b ? R.items[1] : 0);
    a.nsets = (plan_a ? R.n[0] : 0) + (plan_b ? R.n[1] : 0);
    a.S = S;
    a.lg = lg;
    return a;
  };
  const auto record = [&](int kind, int64_t grid, const PaSplitSets& a) {
    ProgArgs pa;
    pa.sets = a;
    return prog_mem(rec, kind, (uint32_t)grid, pa, {});
  };
  const PaSplitSets l = part(sp->lng, 0), m = part(sp->mid, 0), s = part(sp->shrt, sp->short_lg);
  if (l.end > l.first) {
    for (auto& z : sp->exp_ranges[sides]) GBX_TRY(zero_async(z.first, z.second, st));
    const int64_t grid = std::min<int64_t>(l.end - l.first, 152 * 16);
    if (rec) {
      GBX_TRY(record(PK_ROWEXP, grid, l));
      GBX_TRY(record(PK_DIGITS, grid, l));
    } else {
      GBX_TRY(launch(row_exponent_kernel, (unsigned)grid, 256, st, l.sets, l.nsets, l.first, l.end));
      GBX_TRY(launch(digits_kernel, (unsigned)grid, 256, st, l.sets, l.nsets, l.first, l.end, S));
    }
  }
  if (m.end > m.first) {
    const int64_t grid = std::min<int64_t>(m.end - m.first, 152 * 8);
    if (rec) GBX_TRY(record(PK_SPLITROWS, grid, m));
    else
      GBX_TRY(launch(sp->mid_four ? split_rows_kernel<true> : split_rows_kernel<false>, (unsigned)grid, 256, st, m.sets,
                     m.nsets, m.first, m.end, S));
  }
  if (s.end > s.first) {
    const int64_t per = 256 >> s.lg, grid = std::min<int64_t>((s.end - s.first + per - 1) / per, 152 * 32);
    if (rec) GBX_TRY(record(PK_SHORTROWS, grid, s));
    else
      GBX_TRY(launch(split_short_rows_kernel, (unsigned)grid, 256, st, s.sets, s.nsets, s.first, s.end, S, s.lg));
  }
  return GBX_OK;
}

namespace {

template <int BN>
int launch_width(const GemmParams& P, int nsm, cudaStream_t st) {
  const int grid = std::min(P.total_tiles, nsm * SplitCfg<BN>::kCtasPerSm);
  return launch_dependent(split_gemm_kernel<BN>, (unsigned)grid, SplitCfg<BN>::kThreads, st, 1u, sizeof(Smem<BN>) + 1024, P);
}

template <int S>
int launch_ks(const GemmParams& P, int nsm, cudaStream_t st) {
  return launch_dependent(split_ks_kernel<S>, (unsigned)std::min(P.total_tiles, nsm), kKsThreads, st, 1u,
                          sizeof(KsSmem<S>) + 1024, P);
}

// The GEMM kernel of one launch class -- bn 0 / 1: thin-K with a 64 / 32
// element k-block; 64: k-stationary; else the pair-by-pair kernel of that
// output tile width -- over the problems of P.
int launch_split_gemm(int bn, const GemmParams& P, cudaStream_t st) {
  if (P.total_tiles <= 0) return GBX_OK;
  int dev = 0, nsm = 152;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (bn <= 1) {
    const unsigned grid = (unsigned)std::min(P.total_tiles, nsm);
    const size_t smem = (bn == 0 ? sizeof(ThinSmem<64>) : sizeof(ThinSmem<32>)) + 1024;
    const cudaError_t le = try_launch_dependent(bn == 0 ? split_thin_kernel<64> : split_thin_kernel<32>, grid,
                                                kThinThreads, st, 1u, smem, P);
    if (le != cudaSuccess) {
      cudaFuncAttributes fa;
      std::memset(&fa, 0, sizeof(fa));
      cudaFuncGetAttributes(&fa, bn == 0 ? (const void*)split_thin_kernel<64> : (const void*)split_thin_kernel<32>);
      return fail(GBX_ECUDA, "thin-K launch (k-block %d): %s; dynamic smem %zu (max %d), static %zu, regs %d, max threads %d",
                  bn == 0 ? 64 : 32, cudaGetErrorString(le), smem,
                  fa.maxDynamicSharedSizeBytes, fa.sharedSizeBytes, fa.numRegs, fa.maxThreadsPerBlock);
    }
    return GBX_OK;
  }
  switch (bn) {
    case 32: return launch_width<32>(P, nsm, st);
    case 64:
      switch (P.S) {
        case 2: return launch_ks<2>(P, nsm, st);
        case 3: return launch_ks<3>(P, nsm, st);
        case 4: return launch_ks<4>(P, nsm, st);
        case 5: return launch_ks<5>(P, nsm, st);
        case 6: return launch_ks<6>(P, nsm, st);
        default: return launch_ks<7>(P, nsm, st);
      }
    case 128: return launch_width<128>(P, nsm, st);
    default: return launch_width<256>(P, nsm, st);
  }
}

GemmParams params_of(const SplitPlan* sp, const SplitLaunch& L) {
  GemmParams P;
  P.probs = L.d_probs;
  P.tile_first = L.d_tile_first;
  P.maps = L.d_maps;
  P.nprob = L.nprob;
  P.total_tiles = L.total_tiles;
  P.S = sp->S;
  P.L = sp->L;
  P.err = sp->d_err;
  return P;
}

}  // namespace

int run_split_plan(SplitPlan* sp, bool plan_a, bool plan_b, cudaStream_t st) {
  if (!sp || sp->nsets == 0) return GBX_OK;
  GBX_TRY(split_operands(sp, plan_a, plan_b, st));
  ProgRecorder* rec = prog_recording();
  for (size_t i = 0; i < sp->launches.size(); ++i) {
    const SplitLaunch& L = sp->launches[i];
    if (L.total_tiles <= 0) continue;
    if (rec) GBX_TRY(prog_split(rec, sp, (int)i));
    else GBX_TRY(launch_split_gemm(L.bn, params_of(sp, L), st));
  }
  if (sp->nred > 0) {
    int rg = (int)std::min<int64_t>((sp->red_total + 255) / 256, 152 * 8);
    if (rec) {
      ProgArgs a;
      a.splitred = {sp->d_all, sp->d_red_prob, sp->d_red_first, sp->red_total, sp->nred};
      return prog_mem(rec, PK_SPLITRED, (uint32_t)rg, a, {});
    }
    GBX_TRY(launch(split_reduce_kernel, (unsigned)rg, 256, st, sp->d_all, sp->d_red_prob, sp->d_red_first, sp->nred,
                   sp->red_total));
  }
  return GBX_OK;
}

// ---- merged launches of the persistent iteration program -------------------

int split_launch_class(const SplitPlan* sp, int launch) {
  if (!sp || launch < 0 || launch >= (int)sp->launches.size()) return -1;
  const int bn = sp->launches[launch].bn;
  return bn * 16 + sp->S;  // kernel and slice count
}

struct SplitMerged {
  int bn = 0;
  GemmParams P;
  DevProblem* d_probs = nullptr;
  int* d_first = nullptr;
  CUtensorMap* d_maps = nullptr;
  ~SplitMerged() {
    dev_free(d_probs);
    dev_free(d_first);
    dev_free(d_maps);
  }
};

int split_merge(const std::vector<std::pair<SplitPlan*, int>>& parts, int* err, SplitMerged** out) {
  *out = nullptr;
  if (parts.empty()) return fail(GBX_EINVAL, "split merge: no launches");
  auto m = std::make_unique<SplitMerged>();
  const int cls = split_launch_class(parts[0].first, parts[0].second);
  std::vector<DevProblem> hp;
  std::vector<CUtensorMap> hm;
  std::vector<int> first;
  int64_t tiles = 0;
  for (auto& pr : parts) {
    if (split_launch_class(pr.first, pr.second) != cls) return fail(GBX_EINVAL, "split merge: mixed launch classes");
    const SplitLaunch& L = pr.first->launches[pr.second];
    for (size_t i = 0; i < L.hp.size(); ++i) {
      hp.push_back(L.hp[i]);
      hm.push_back(L.hm[2 * i]);
      hm.push_back(L.hm[2 * i + 1]);
      first.push_back((int)(tiles + L.hfirst[i]));
    }
    tiles += L.total_tiles;
  }
  if (tiles >= (1ll << 31)) return fail(GBX_EUNSUPPORTED, "split merge: too many tiles");
  GBX_TRY(dev_alloc((void**)&m->d_probs, sizeof(DevProblem) * hp.size()));
  GBX_TRY(dev_alloc((void**)&m->d_first, sizeof(int) * first.size()));
  GBX_TRY(dev_alloc((void**)&m->d_maps, sizeof(CUtensorMap) * hm.size()));
  GBX_CUDA(cudaMemcpy(m->d_probs, hp.data(), sizeof(DevProblem) * hp.size(), cudaMemcpyHostToDevice));
  GBX_CUDA(cudaMemcpy(m->d_first, first.data(), sizeof(int) * first.size(), cudaMemcpyHostToDevice));
  GBX_CUDA(cudaMemcpy(m->d_maps, hm.data(), sizeof(CUtensorMap) * hm.size(), cudaMemcpyHostToDevice));
  const SplitPlan* sp0 = parts[0].first;
  m->bn = sp0->launches[parts[0].second].bn;
  m->P.probs = m->d_probs;
  m->P.tile_first = m->d_first;
  m->P.maps = m->d_maps;
  m->P.nprob = (int)hp.size();
  m->P.total_tiles = (int)tiles;
  m->P.S = sp0->S;
  m->P.L = sp0->L;
  m->P.err = err;
  *out = m.release();
  return GBX_OK;
}

int split_merged_run(const SplitMerged* m, cudaStream_t st) { return launch_split_gemm(m->bn, m->P, st); }

void split_merged_destroy(SplitMerged* m) { delete m; }

int split_plan_error(SplitPlan* sp) {
  if (!sp) return 0;
  int e = 0;
  if (cudaMemcpy(&e, sp->d_err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
  return e;
}

double split_plan_tensor_flops(const SplitPlan* sp) {
  if (!sp) return 0.0;
  double f = 0.0;
  const double pairs = sp->S * (sp->S + 1) / 2.0;
  for (size_t i = 0; i < sp->host.size(); ++i) {
    const SplitProblem& p = sp->host[i];
    const int bn = sp->width[i];  // thin-K problems: 32
    double Mp = (double)((p.M + BM - 1) / BM * BM), Np = (double)((p.N + bn - 1) / bn * bn);
    const int kb = sp->kb[i];
    double Kp = (double)((p.K + kb - 1) / kb * kb);
    f += 2.0 * pairs * Mp * Np * Kp;
  }
  return f;
}

void destroy_split_plan(SplitPlan* sp) { delete sp; }

int split_set_width(int bn) {
  if (bn != 0 && bn != 32 && bn != 64 && bn != 128 && bn != 256) return fail(GBX_EINVAL, "width must be 0, 32, 64, 128 or 256");
  g_width_override = bn;
  return GBX_OK;
}

double split_plan_bytes(const SplitPlan* sp) { return sp ? sp->bytes : 0.0; }

// ---- self-test of the bounded waits ---------------------------------------
// One CTA waits on an mbarrier that nothing arrives on, through the same
// bounded wait as the split kernels' pipeline waits; it gives up after the
// limit, records its stage in the error word and returns.
namespace {
constexpr int kSelftestStage = 31;
__device__ int g_wait_selftest_err;

__global__ void wait_selftest_reset_kernel() { g_wait_selftest_err = 0; }

__global__ void wait_selftest_kernel(long long limit) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (threadIdx.x == 0) mbar_wait(&bar, 0, &g_wait_selftest_err, kSelftestStage, limit);
  __syncthreads();
}
}  // namespace

}  // namespace gbx

extern "C" int gbx_wait_selftest(long long limit_cycles, void* stream) {
  using namespace gbx;
  if (limit_cycles < 0 || limit_cycles > kWaitCycles)
    return fail(GBX_EINVAL, "limit_cycles %lld outside [0, %lld]", limit_cycles, (long long)kWaitCycles);
  cudaStream_t st = (cudaStream_t)stream;
  wait_selftest_reset_kernel<<<1, 1, 0, st>>>();
  GBX_CUDA(cudaGetLastError());
  wait_selftest_kernel<<<1, 32, 0, st>>>(limit_cycles);
  GBX_CUDA(cudaGetLastError());
  GBX_CUDA(cudaStreamSynchronize(st));
  int e = 0;
  GBX_CUDA(cudaMemcpyFromSymbol(&e, g_wait_selftest_err, sizeof(int)));
  if (e != 0) return fail(GBX_ETIMEOUT, "a bounded device wait ran out (stage %d)", e);
  return GBX_OK;
}
