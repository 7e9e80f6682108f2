// Strided tile moves from descriptors in device memory: the packs, unpacks and
// permuted accumulates of contraction plans and programs, which keep their
// descriptors (one-call permutes and packs: permute.cu).
//
// A launch covers a whole set of moves (e.g. every tile of one operand of one
// contraction).  Each CTA takes one chunk of one move; threads walk the chunk
// in destination order, so stores are coalesced along the destination's
// fastest dimension and loads go through the read-only cache.
// Pure copies (op 0, scale 1) move bits unchanged, so permutes are bit-exact.
#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstring>

#include "bodies.cuh"
#include "common.h"
#include "launch.h"
#include "program.h"

namespace gbx {

namespace {
using dev::kMove4Chunk;
using dev::kMoveChunk;
using dev::kMoveThreads;
}  // namespace

MoveDesc make_move(int rank, const int64_t* ext, const int64_t* sstr, const int64_t* dstr, int64_t src,
                   int64_t dst, int op, double scale) {
  // drop unit extents, then order by destination stride (largest first)
  int idx[kMaxDims];
  int r = 0;
  for (int d = 0; d < rank; ++d)
    if (ext[d] != 1) idx[r++] = d;
  std::stable_sort(idx, idx + r, [&](int a, int b) { return dstr[a] > dstr[b]; });
  int64_t e[kMaxDims], s[kMaxDims], t[kMaxDims];
  int m = 0;
  for (int i = 0; i < r; ++i) {
    int d = idx[i];
    // merge with the previous (outer) dim when contiguous in both buffers
    if (m > 0 && s[m - 1] == sstr[d] * ext[d] && t[m - 1] == dstr[d] * ext[d]) {
      e[m - 1] *= ext[d];
      s[m - 1] = sstr[d];
      t[m - 1] = dstr[d];
    } else {
      e[m] = ext[d];
      s[m] = sstr[d];
      t[m] = dstr[d];
      ++m;
    }
  }
  MoveDesc md;
  std::memset(&md, 0, sizeof(md));
  if (m == 0) {  // a single element
    e[0] = 1;
    s[0] = 0;
    t[0] = 0;
    m = 1;
  }
  md.rank = m;
  int64_t n = 1;
  for (int i = 0; i < m; ++i) {
    md.ext[i] = (uint32_t)e[i];
    md.sstr[i] = s[i];
    md.dstr[i] = t[i];
    md.div[i] = FastDiv::make((uint32_t)e[i]);
    n *= e[i];
  }
  for (int i = 0; i < rank; ++i)
    if (ext[i] == 0) n = 0;
  md.n = (uint32_t)n;
  md.src = src;
  md.dst = dst;
  md.op = op;
  md.scale = scale;
  return md;
}

int MoveSet::upload() {
  release();
  ndesc = (int)host.size();
  if (ndesc == 0) return GBX_OK;
  bool small = true;
  for (const MoveDesc& m : host) {
    uint64_t prod = 1;
    for (int d = 0; d < m.rank; ++d) prod *= m.ext[d];
    if (prod >= (1ull << 31) || (prod != m.n && m.n != 0))
      return fail(GBX_EUNSUPPORTED, "tile move of %llu elements (at most 2^31 - 1)", (unsigned long long)prod);
    small = small && m.rank <= 4;
  }
  if (small) {
    chunk = chunk4();
    std::vector<MoveDesc4> h4(ndesc);
    std::vector<uint32_t> cd;
    uint64_t c = 0;
    for (int i = 0; i < ndesc; ++i) {
      const MoveDesc& m = host[i];
      MoveDesc4& q = h4[i];
      std::memset(&q, 0, sizeof(q));
      const int pad = 4 - m.rank;
      for (int d = 0; d < 4; ++d) {
        const bool real = d >= pad;
        q.ext[d] = real ? m.ext[d - pad] : 1u;
        q.sstr[d] = real ? m.sstr[d - pad] : 0;
        q.dstr[d] = real ? m.dstr[d - pad] : 0;
        q.div[d] = FastDiv::make(q.ext[d]);
      }
      q.src = m.src;
      q.dst = m.dst;
      q.n = m.n;
      q.op = m.op;
      q.scale = m.scale;
      // moves whose innermost run is contiguous on both sides, of even
      // length, starting at even offsets with even outer strides go two
      // elements at a time (16-byte loads and stores)
      bool pair = q.ext[3] % 2 == 0 && q.sstr[3] == 1 && q.dstr[3] == 1 && m.src % 2 == 0 && m.dst % 2 == 0;
      for (int d = 0; d < 3 && pair; ++d) pair = q.sstr[d] % 2 == 0 && q.dstr[d] % 2 == 0;
      q.pad = pair ? 1 : 0;
      q.first = (uint32_t)c;
      const uint64_t nc = (m.n + chunk - 1) / chunk;
      c += nc;
      if (c >= (1ull << 31)) return fail(GBX_EUNSUPPORTED, "move set too large (%llu chunks)", (unsigned long long)c);
      for (uint64_t k = 0; k < nc; ++k) cd.push_back((uint32_t)i);
    }
    nchunks = (uint32_t)c;
    GBX_TRY(dev_alloc((void**)&d_desc4, sizeof(MoveDesc4) * ndesc));
    GBX_CUDA(cudaMemcpy(d_desc4, h4.data(), sizeof(MoveDesc4) * ndesc, cudaMemcpyHostToDevice));
    if (nchunks) {
      GBX_TRY(dev_alloc((void**)&d_chunk_desc, sizeof(uint32_t) * nchunks));
      GBX_CUDA(cudaMemcpy(d_chunk_desc, cd.data(), sizeof(uint32_t) * nchunks, cudaMemcpyHostToDevice));
    }
    return GBX_OK;
  }
  std::vector<uint32_t> first(ndesc + 1);
  uint64_t c = 0;
  for (int i = 0; i < ndesc; ++i) {
    first[i] = (uint32_t)c;
    c += (host[i].n + kMoveChunk - 1) / kMoveChunk;
  }
  first[ndesc] = (uint32_t)c;
  if (c >= (1ull << 31)) return fail(GBX_EUNSUPPORTED, "move set too large (%llu chunks)", (unsigned long long)c);
  nchunks = (uint32_t)c;
  GBX_TRY(dev_alloc((void**)&d_desc, sizeof(MoveDesc) * ndesc));
  GBX_TRY(dev_alloc((void**)&d_first, sizeof(uint32_t) * (ndesc + 1)));
  GBX_CUDA(cudaMemcpy(d_desc, host.data(), sizeof(MoveDesc) * ndesc, cudaMemcpyHostToDevice));
  GBX_CUDA(cudaMemcpy(d_first, first.data(), sizeof(uint32_t) * (ndesc + 1), cudaMemcpyHostToDevice));
  return GBX_OK;
}

// Elements of a chunk: smaller ones where the larger would leave SMs without
// work (a pack of 187k elements: 6.6 us in 46 chunks of 4096, 5.5 in 183).
uint32_t MoveSet::chunk4() const {
  uint64_t c = 0;
  for (const MoveDesc& m : host) c += (m.n + kMove4Chunk - 1) / kMove4Chunk;
  return c < 152 * 2 ? (uint32_t)dev::kMove4Small : (uint32_t)kMove4Chunk;
}

size_t MoveSet::device_bytes() const {
  if (host.empty()) return 0;
  bool small = true;
  uint64_t c = 0;
  const uint32_t per = chunk4();
  for (const MoveDesc& m : host) {
    small = small && m.rank <= 4;
    c += (m.n + per - 1) / per;
  }
  if (small) return host.size() * sizeof(MoveDesc4) + c * sizeof(uint32_t);
  return host.size() * sizeof(MoveDesc) + (host.size() + 1) * sizeof(uint32_t);
}

void MoveSet::release() {
  dev_free(d_desc);
  dev_free(d_first);
  dev_free(d_desc4);
  dev_free(d_chunk_desc);
  d_desc = nullptr;
  d_first = nullptr;
  d_desc4 = nullptr;
  d_chunk_desc = nullptr;
  nchunks = 0;
}

__global__ void __launch_bounds__(kMoveThreads) tile_move_kernel(const MoveDesc* __restrict__ descs,
                                                                 const uint32_t* __restrict__ first, int ndesc,
                                                                 uint32_t nchunks, const double* __restrict__ src,
                                                                 double* __restrict__ dst, double alpha) {
  begin_dependent();
  dev::move_body<false>(descs, first, ndesc, nchunks, src, dst, alpha, blockIdx.x, gridDim.x);
}

// Moves of at most four dimensions (dev::move4_body).
template <int kPer, int kChunk>
__global__ void __launch_bounds__(kMoveThreads) tile_move4_kernel(const MoveDesc4* __restrict__ descs,
                                                                  const uint32_t* __restrict__ chunk_desc,
                                                                  uint32_t nchunks, const double* __restrict__ src,
                                                                  double* __restrict__ dst, double alpha,
                                                                  int allow_pairs) {
  begin_dependent();
  dev::move4_body<false, kPer, kChunk>(descs, chunk_desc, nchunks, src, dst, alpha, allow_pairs, blockIdx.x,
                                       gridDim.x);
}

struct Moves4 {
  const MoveDesc4* descs;
  const uint32_t* chunk_desc;
  const double* src;
  double* dst;
  uint32_t nchunks, blocks;
  int pairs, small;
};

// Two sets of moves, a's on the first a.blocks CTAs and b's on the others: a
// contraction's two packs wait for nothing of each other's, and small ones
// are bound by their launches (a split plan of M = N = K = 400 at 4 slices:
// 35.2 us with two launches, 33.5 so; of 3600 x 400 x 3600: 201 and 197).
__global__ void __launch_bounds__(kMoveThreads) tile_move4_two_kernel(const Moves4 a, const Moves4 b) {
  begin_dependent();
  const bool first = blockIdx.x < a.blocks;
  const Moves4& m = first ? a : b;
  const uint32_t bid = first ? blockIdx.x : blockIdx.x - a.blocks;
  if (m.small)
    dev::move4_body<false, 2, dev::kMove4Small>(m.descs, m.chunk_desc, m.nchunks, m.src, m.dst, 1.0, m.pairs, bid,
                                                m.blocks);
  else
    dev::move4_body<false, 8, kMove4Chunk>(m.descs, m.chunk_desc, m.nchunks, m.src, m.dst, 1.0, m.pairs, bid,
                                           m.blocks);
}

int run_moves_two(const MoveSet& ma, const double* srcA, double* dstA, const MoveSet& mb, const double* srcB,
                  double* dstB, cudaStream_t st) {
  const auto fits = [](const MoveSet& ms) { return ms.ndesc > 0 && ms.nchunks > 0 && ms.d_desc4; };
  if (!fits(ma) || !fits(mb) || prog_recording()) {
    GBX_TRY(run_moves(ma, srcA, dstA, st));
    return run_moves(mb, srcB, dstB, st);
  }
  const auto moves = [](const MoveSet& ms, const double* src, double* dst) {
    Moves4 m;
    m.descs = ms.d_desc4;
    m.chunk_desc = ms.d_chunk_desc;
    m.src = src;
    m.dst = dst;
    m.nchunks = ms.nchunks;
    m.blocks = std::min<uint32_t>(ms.nchunks, 152u * 8u);
    m.pairs = (((uintptr_t)src | (uintptr_t)dst) & 15) == 0 ? 1 : 0;
    m.small = ms.chunk == (uint32_t)kMove4Chunk ? 0 : 1;
    return m;
  };
  const Moves4 a = moves(ma, srcA, dstA), b = moves(mb, srcB, dstB);
  return launch(tile_move4_two_kernel, a.blocks + b.blocks, kMoveThreads, st, a, b);
}

int run_moves_scaled(const MoveSet& ms, const double* src, double* dst, double alpha, cudaStream_t st) {
  if (ms.ndesc == 0 || ms.nchunks == 0) return GBX_OK;
  ProgRecorder* rec = prog_recording();
  if (ms.d_desc4) {
    const int grid = (int)std::min<uint32_t>(ms.nchunks, 152u * 8u);
    // pairs need 16-byte aligned buffer bases (descriptor offsets are even)
    const int pairs = (((uintptr_t)src | (uintptr_t)dst) & 15) == 0 ? 1 : 0;
    if (rec) {
      ProgArgs a;
      a.move4 = {ms.d_desc4, ms.d_chunk_desc, ms.nchunks, pairs, src, dst, alpha};
      return prog_mem(rec, ms.chunk == (uint32_t)kMove4Chunk ? PK_MOVE4 : PK_MOVE4S, (uint32_t)grid, a,
                      {{src, false}, {dst, true}});
    }
    if (ms.chunk == (uint32_t)kMove4Chunk)
      GBX_TRY(launch(tile_move4_kernel<8, kMove4Chunk>, (unsigned)grid, kMoveThreads, st, ms.d_desc4, ms.d_chunk_desc,
                     ms.nchunks, src, dst, alpha, pairs));
    else
      GBX_TRY(launch(tile_move4_kernel<2, dev::kMove4Small>, (unsigned)grid, kMoveThreads, st, ms.d_desc4,
                     ms.d_chunk_desc, ms.nchunks, src, dst, alpha, pairs));
    return GBX_OK;
  }
  int grid = (int)std::min<uint32_t>(ms.nchunks, 152u * 16u);
  if (rec) {
    ProgArgs a;
    a.move = {ms.d_desc, ms.d_first, ms.ndesc, ms.nchunks, src, dst, alpha};
    return prog_mem(rec, PK_MOVE, (uint32_t)grid, a, {{src, false}, {dst, true}});
  }
  GBX_TRY(launch(tile_move_kernel, (unsigned)grid, kMoveThreads, st, ms.d_desc, ms.d_first, ms.ndesc, ms.nchunks, src,
                 dst, alpha));
  return GBX_OK;
}

int run_moves(const MoveSet& ms, const double* src, double* dst, cudaStream_t st) {
  return run_moves_scaled(ms, src, dst, 1.0, st);
}

// One CTA per work item of the fused sum (dev::fused_sum_body).
__global__ void __launch_bounds__(dev::kFsThreads, 3)
    fused_sum_kernel(const FsItem* __restrict__ items, int nitems, const FsTerm* __restrict__ terms, FsSrc src,
                     const double* __restrict__ scale, double* __restrict__ out) {
  begin_dependent();
  __shared__ dev::FsSmem sm;
  dev::fused_sum_body<false>(items, nitems, terms, src, scale, out, blockIdx.x, gridDim.x, sm);
}

int run_fused_sum(const FsItem* items, int nitems, const FsTerm* terms, const FsSrc& src, const double* scale,
                  double* out, cudaStream_t st) {
  if (nitems == 0) return GBX_OK;
  const int grid = std::min(nitems, 152 * 6);
  if (ProgRecorder* rec = prog_recording()) {
    ProgArgs a;
    a.fused.items = items;
    a.fused.terms = terms;
    a.fused.scale = scale;
    a.fused.out = out;
    a.fused.nitems = nitems;
    a.fused.src = src;
    std::vector<ProgTouch> t = {{scale, false}, {out, true}};
    for (int k = 0; k < kFsMaxSlots; ++k) t.push_back({src.p[k], false});
    return prog_mem(rec, PK_FUSED, (uint32_t)grid, a, t);
  }
  GBX_TRY(launch(fused_sum_kernel, (unsigned)grid, dev::kFsThreads, st, items, nitems, terms, src, scale, out));
  return GBX_OK;
}

}  // namespace gbx
