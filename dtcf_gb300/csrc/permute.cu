// One-call permutes and packs: the block permutes of the leaf entry points,
// the big-matrix packs and the DLTC executor's moves.
//
// Nothing is allocated or uploaded: the descriptors (and the table that says
// which permutation a block takes, or which tile a matrix position holds)
// travel in the kernel's arguments, so a call is one launch.  (With
// descriptors in stream-ordered temporaries a call was two allocations, two
// copies and two frees: 22 us beside others, 230 us after a synchronisation,
// when the allocator's pool had been given back.)
//
// Permutes are cut into boxes of up to 4096 elements that hold runs of at
// least 16 elements in both the source's and the destination's order, as far
// as the extents allow.  A CTA reads its box in source order into shared
// memory and writes it in destination order, so both sides of HBM see whole
// lines; the shared-memory pitches are chosen so that walking the
// destination's order meets no bank conflicts.  Moves that keep their
// fastest dimension go straight through registers.  The instructions of the
// index decode bound the kernel before HBM does, so dimensions that stay
// adjacent in a walk are merged, even runs go two elements to a decode with
// 16-byte accesses, one thread finds the box's corner for the CTA, and the
// walk's constants sit in registers.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.h"
#include "launch.h"

namespace gbx {

namespace {

constexpr int kBoxThreads = 256;
constexpr int kBoxElems = 4096;   // elements of a box
constexpr int kBoxSmem = 5120;    // with its pitches made odd
constexpr int kBoxDims = 6;       // dimensions a box may extend in
constexpr int kBoxPer = 8;        // elements in flight per thread
constexpr int kSetDescs = 16;     // permutations of one launch
// Entries of a launch's tables: about what fits into 32 KB of kernel arguments
// beside the descriptors, and for calls of fewer blocks or tiles (kSmallSet,
// kSmallPack) a few KB, since the host fills all of the arguments it launches
// with (2000 4^4 blocks 14.3 us, 16.0 with the large table; 81 packed tiles
// 9.1 and 9.6).
constexpr int kSetBlocks = 16384, kSmallSet = 2048;
constexpr int kListBlocks = 4096;  // with the blocks' numbers beside their permutations
constexpr int kPackTiles = 14336, kSmallPack = 1536;  // (slots below 65536; kPackTiles / 2 beyond)

// One dimension of a walk over a box: extent, ceil(2^32 / extent) for the
// division (exact: index x extent < 2^32), the tensor stride and the
// shared-memory pitch (the source's stride in straight moves); dim and mul:
// where the box is cut off, its real extent here is that of dimension dim
// times mul.
struct BoxDim {
  uint32_t ext, magic, str, pitch;
  uint32_t dim, mul;
};

struct BoxOrder {
  BoxDim d[kBoxDims];  // fastest first
  int32_t nd, pairs;   // dimensions; two elements to a decode (extents, strides in pairs)
};

struct BoxMove {
  int64_t sstr[kMaxDims], dstr[kMaxDims];
  uint32_t ext[kMaxDims], box[kMaxDims];
  FastDiv grid[kMaxDims];  // boxes per dimension
  BoxOrder in, out;
  int64_t src, dst;
  uint32_t boxes, n;  // boxes of the move, elements of a box
  int32_t rank, staged, op, pad;
  double scale;
};

struct OneMove {
  BoxMove m;
  FastDiv per;       // boxes per block
  int64_t block;     // elements between blocks, both sides
};

template <int kBlocks>
struct MoveTable {
  BoxMove m[kSetDescs];
  FastDiv per;
  int64_t block;
  uint8_t which[kBlocks];
};

// The same for blocks that do not follow one another.
struct MoveList {
  BoxMove m[kSetDescs];
  FastDiv per;
  int64_t block;
  uint32_t id[kListBlocks];
  uint8_t which[kListBlocks];
};

// What one thread finds out about the CTA's box.
struct BoxPlace {
  int64_t src, dst;
  uint32_t lim[kMaxDims];  // real extents
  int cut;                 // some extent is below the box's
};

// A walk's constants in registers.
template <int ND, bool kCut>
struct BoxWalk {
  uint32_t ext[ND], magic[ND], str[ND], pitch[ND], lim[ND];
  __device__ __forceinline__ BoxWalk(const BoxOrder& o, const uint32_t* real) {
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      ext[j] = o.d[j].ext;
      magic[j] = o.d[j].magic;
      str[j] = o.d[j].str;
      pitch[j] = o.d[j].pitch;
      lim[j] = kCut ? real[o.d[j].dim] * o.d[j].mul : 0u;
      if (kCut && j == 0 && o.pairs) lim[j] >>= 1;
    }
  }
  // offset and shared-memory place of item e; false: past the box's cut edge
  __device__ __forceinline__ bool at(uint32_t e, uint32_t& off, uint32_t& place) const {
    uint32_t o = 0, a = 0;
    bool in = true;
#pragma unroll
    for (int j = 0; j < ND; ++j) {
      const bool last = j == ND - 1;
      const uint32_t q = last ? 0u : __umulhi(e, magic[j]), c = last ? e : e - q * ext[j];
      o += c * str[j];
      a += c * pitch[j];
      if (kCut) in = in && c < lim[j];
      e = q;
    }
    off = o;
    place = a;
    return in;
  }
};

// What happens to an element on its way out: the two forms are separate code,
// since a select between x and scale * x issues the multiply either way and
// FP64 instructions are scarce (2 per clock and SM: the multiplies alone made
// 2000 8^4 blocks 43 us instead of 24).
struct BoxCopy {  // +-x
  long long flip;
  __device__ __forceinline__ double sign(double x) const { return __longlong_as_double(__double_as_longlong(x) ^ flip); }
  __device__ __forceinline__ void put(double* p, double x) const { *p = sign(x); }
  __device__ __forceinline__ void put(double2* p, double2 x) const { *p = make_double2(sign(x.x), sign(x.y)); }
};
struct BoxScale {  // scale * x, or dst + scale * x
  double scale;
  int add;
  __device__ __forceinline__ void put(double* p, double x) const {
    if (add) *p = __fma_rn(scale, x, *p);
    else *p = __dmul_rn(scale, x);
  }
  __device__ __forceinline__ void put(double2* p, double2 x) const {
    if (add) {
      const double2 y = *p;
      *p = make_double2(__fma_rn(scale, x.x, y.x), __fma_rn(scale, x.y, y.y));
    } else {
      *p = make_double2(__dmul_rn(scale, x.x), __dmul_rn(scale, x.y));
    }
  }
};

__device__ __forceinline__ void stage_get(const double* p, uint32_t, double& x) { x = *p; }
// Lanes 8 apart are 16 banks apart: every second eight lanes read their pair
// the other way round, which keeps each half warp on 16 different banks.
__device__ __forceinline__ void stage_get(const double* p, uint32_t step, double2& x) {
  const bool turn = (threadIdx.x & 8) != 0;
  const double u = p[turn ? step : 0], v = p[turn ? 0 : step];
  x = make_double2(turn ? v : u, turn ? u : v);
}

// Straight: source to destination in destination order, T one element or two.
struct BoxStraight {
  template <int ND, bool kCut, typename T, class Out>
  static __device__ __forceinline__ void run(const BoxOrder& order, uint32_t n, const uint32_t* real,
                                             const double* __restrict__ s, double* __restrict__ t, const Out& o) {
    constexpr int kW = (int)(sizeof(T) / sizeof(double)), kPer = kBoxPer / kW;
    const BoxWalk<ND, kCut> w(order, real);
    for (uint32_t b = 0; b < n; b += kBoxThreads * kPer) {
      T x[kPer];
      uint32_t off[kPer], at[kPer];
      bool in[kPer];
  #pragma unroll
      for (int k = 0; k < kPer; ++k) {
        in[k] = false;
        if (b + k * kBoxThreads < n) {
          const uint32_t e = b + k * kBoxThreads + threadIdx.x;
          in[k] = w.at(e, off[k], at[k]) && e < n;
          if (in[k]) x[k] = __ldg(reinterpret_cast<const T*>(s + at[k]));
        }
      }
  #pragma unroll
      for (int k = 0; k < kPer; ++k)
        if (in[k]) o.put(reinterpret_cast<T*>(t + off[k]), x[k]);
    }
  }
};

// Source to shared memory in source order, asynchronously: the whole box in
// flight at once, no registers held.
struct BoxFill {
  template <int ND, bool kCut, typename T>
  static __device__ __forceinline__ void run(const BoxOrder& order, uint32_t n, const uint32_t* real,
                                             const double* __restrict__ s, uint32_t stage) {
    const BoxWalk<ND, kCut> w(order, real);
#pragma unroll 4
    for (uint32_t e = threadIdx.x; e < n; e += kBoxThreads) {
      uint32_t off, at;
      if (!w.at(e, off, at)) continue;
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(stage + 8 * at), "l"(s + off) : "memory");
    }
  }
};

// Shared memory to destination in destination order; step: the pitch of the
// destination's fastest dimension.
struct BoxEmpty {
  template <int ND, bool kCut, typename T, class Out>
  static __device__ __forceinline__ void run(const BoxOrder& order, uint32_t n, const uint32_t* real, const double* stage,
                                            uint32_t step, double* __restrict__ t, const Out& o) {
    const BoxWalk<ND, kCut> w(order, real);
  #pragma unroll 4
    for (uint32_t e = threadIdx.x; e < n; e += kBoxThreads) {
      uint32_t off, at;
      if (!w.at(e, off, at)) continue;
      T x;
      stage_get(stage + at, step, x);
      o.put(reinterpret_cast<T*>(t + off), x);
    }
  }
};

// F::run with the walk's number of dimensions, cut or not, one element or two.
template <class F, bool kCut, typename T, class... A>
__device__ __forceinline__ void box_dims(const BoxOrder& o, uint32_t n, A&&... a) {
  switch (o.nd) {
    case 1: F::template run<1, kCut, T>(o, n, a...); break;
    case 2: F::template run<2, kCut, T>(o, n, a...); break;
    case 3: F::template run<3, kCut, T>(o, n, a...); break;
    case 4: F::template run<4, kCut, T>(o, n, a...); break;
    default: F::template run<kBoxDims, kCut, T>(o, n, a...); break;
  }
}
template <class F, class... A>
__device__ __forceinline__ void box_walk(const BoxOrder& o, bool cut, uint32_t n, A&&... a) {
  if (o.pairs) {
    if (cut) box_dims<F, true, double2>(o, n / 2, a...);
    else box_dims<F, false, double2>(o, n / 2, a...);
  } else {
    if (cut) box_dims<F, true, double>(o, n, a...);
    else box_dims<F, false, double>(o, n, a...);
  }
}

__device__ __forceinline__ void box_move(const BoxMove& m, uint32_t box, const double* __restrict__ src,
                                         double* __restrict__ dst, double alpha, double* stage, BoxPlace& place) {
  if (box >= m.boxes) return;  // a permutation that needs fewer boxes than another of the launch
  if (threadIdx.x == 0) {
    int64_t so = m.src, to = m.dst;
    int cut = 0;
    for (int d = m.rank - 1; d >= 0; --d) {
      const uint32_t q = m.grid[d].div(box), c = (box - q * m.grid[d].d) * m.box[d];
      box = q;
      so += (int64_t)c * m.sstr[d];
      to += (int64_t)c * m.dstr[d];
      const uint32_t left = min(m.box[d], m.ext[d] - c);
      cut |= left < m.box[d];
      place.lim[d] = left;
    }
    place.src = so;
    place.dst = to;
    place.cut = cut;
  }
  __syncthreads();
  const double* __restrict__ s = src + place.src;
  double* __restrict__ t = dst + place.dst;
  const bool cut = place.cut != 0;
  // a store ignores the run-time factor; +-x is a bit copy with the sign set
  const double scale = m.op ? __dmul_rn(m.scale, alpha) : m.scale;
  const unsigned long long sb = (unsigned long long)__double_as_longlong(scale);
  const bool copy = !m.op && (sb & 0x7FFFFFFFFFFFFFFFull) == 0x3FF0000000000000ull;
  const BoxCopy as_is{(long long)(sb & 0x8000000000000000ull)};
  const BoxScale scaled{scale, m.op};
  const uint32_t* real = place.lim;
  if (!m.staged) {
    if (copy) box_walk<BoxStraight>(m.out, cut, m.n, real, s, t, as_is);
    else box_walk<BoxStraight>(m.out, cut, m.n, real, s, t, scaled);
    return;
  }
  box_walk<BoxFill>(m.in, cut, m.n, real, s, (uint32_t)__cvta_generic_to_shared(stage));
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const uint32_t step = m.out.pairs ? m.out.d[0].pitch / 2 : 0;
  if (copy) box_walk<BoxEmpty>(m.out, cut, m.n, real, stage, step, t, as_is);
  else box_walk<BoxEmpty>(m.out, cut, m.n, real, stage, step, t, scaled);
}

__global__ void __launch_bounds__(kBoxThreads) box_one_kernel(const __grid_constant__ OneMove a,
                                                              const double* __restrict__ src, double* __restrict__ dst,
                                                              double alpha) {
  begin_dependent();
  __shared__ double stage[kBoxSmem];
  __shared__ BoxPlace place;
  const uint32_t b = a.per.div(blockIdx.x);
  box_move(a.m, blockIdx.x - b * a.per.d, src + b * a.block, dst + b * a.block, alpha, stage, place);
}

template <int kBlocks>
__global__ void __launch_bounds__(kBoxThreads) box_set_kernel(const __grid_constant__ MoveTable<kBlocks> a,
                                                              const double* __restrict__ src,
                                                              double* __restrict__ dst) {
  begin_dependent();
  __shared__ double stage[kBoxSmem];
  __shared__ BoxPlace place;
  const uint32_t b = a.per.div(blockIdx.x);
  box_move(a.m[a.which[b]], blockIdx.x - b * a.per.d, src + b * a.block, dst + b * a.block, 1.0, stage, place);
}

__global__ void __launch_bounds__(kBoxThreads) box_list_kernel(const __grid_constant__ MoveList a,
                                                               const double* __restrict__ src,
                                                               double* __restrict__ dst) {
  begin_dependent();
  __shared__ double stage[kBoxSmem];
  __shared__ BoxPlace place;
  const uint32_t i = a.per.div(blockIdx.x);
  const int64_t at = (int64_t)a.id[i] * a.block;
  box_move(a.m[a.which[i]], blockIdx.x - i * a.per.d, src + at, dst + at, 1.0, stage, place);
}

uint32_t magic_of(uint32_t d) { return d <= 1 ? 0u : (uint32_t)(((1ull << 32) + d - 1) / d); }

// A walk over the box's dimensions, fastest first: str and pitch by
// dimension.  Dimensions that continue the one before on both sides are
// merged into it (never across a dimension that can be cut).
BoxOrder make_order(const BoxMove& b, const int* order, const int64_t* str, const uint32_t* pitch, bool pairs) {
  BoxOrder o;
  std::memset(&o, 0, sizeof(o));
  bool whole = false;  // the last dimension added is never cut
  for (int i = 0; i < b.rank; ++i) {
    const int d = order[i];
    if (b.box[d] == 1) continue;
    BoxDim* last = o.nd ? &o.d[o.nd - 1] : nullptr;
    const bool uncut = b.box[d] == b.ext[d];
    if (last && whole && (uint64_t)last->str * last->ext == (uint64_t)str[d] &&
        (uint64_t)last->pitch * last->ext == pitch[d]) {
      last->mul = last->ext;
      last->dim = (uint32_t)d;
      last->ext *= b.box[d];
    } else {
      o.d[o.nd++] = BoxDim{b.box[d], 0, (uint32_t)str[d], pitch[d], (uint32_t)d, 1};
    }
    whole = uncut;
  }
  if (o.nd == 0) {
    o.nd = 1;
    o.d[0] = BoxDim{1, 0, 0, 0, 0, 1};
  }
  // pairs: the fastest run is contiguous and everything that moves its start
  // is even, its cut-off length included
  pairs = pairs && o.d[0].str == 1 && o.d[0].ext % 2 == 0 && o.d[0].ext >= 4;
  for (int d = 0; d < b.rank && pairs; ++d)
    if (str[d] != 1) pairs = str[d] % 2 == 0 || b.ext[d] == 1;
    else pairs = b.ext[d] % 2 == 0 && b.box[d] % 2 == 0;
  o.pairs = pairs;
  if (pairs) {
    o.d[0].ext /= 2;
    o.d[0].str = 2;
    o.d[0].pitch *= 2;
  }
  for (int j = 0; j < o.nd; ++j) o.d[j].magic = magic_of(o.d[j].ext);
  // more than four: the fifth and sixth walk together, unit extents at the end
  if (o.nd > 4)
    for (int j = o.nd; j < kBoxDims; ++j) {
      o.d[j].ext = 1;
      o.d[j].mul = 1;
    }
  return o;
}

// Cuts a move into boxes of about `target` elements.  pairs: both buffers
// start on 16-byte boundaries.
BoxMove make_box(const MoveDesc& md, uint32_t target, bool pairs) {
  BoxMove b;
  std::memset(&b, 0, sizeof(b));
  const int r = md.rank;
  b.rank = r;
  b.src = md.src;
  b.dst = md.dst;
  b.op = md.op;
  b.scale = md.scale;
  int in[kMaxDims], out[kMaxDims];  // dimensions, fastest first
  for (int d = 0; d < r; ++d) {
    in[d] = out[d] = d;
    b.ext[d] = md.ext[d];
    b.sstr[d] = md.sstr[d];
    b.dstr[d] = md.dstr[d];
    b.box[d] = 1;
  }
  std::sort(in, in + r, [&](int x, int y) { return md.sstr[x] < md.sstr[y]; });
  std::sort(out, out + r, [&](int x, int y) { return md.dstr[x] < md.dstr[y]; });
  b.staged = in[0] != out[0] || md.ext[in[0]] < 4;
  uint64_t vol = 1;
  int used = 0;
  // widens dimension d towards `want` elements, in even pieces
  const auto widen = [&](int d, uint64_t want) {
    const uint64_t room = target / (vol / b.box[d]);
    want = std::min<uint64_t>(std::min<uint64_t>(want, room), md.ext[d]);
    if (want <= b.box[d]) return;
    if (b.box[d] == 1 && used == kBoxDims) return;
    const uint64_t pieces = (md.ext[d] + want - 1) / want, even = (md.ext[d] + pieces - 1) / pieces;
    if (even <= b.box[d]) return;
    if (b.box[d] == 1) ++used;
    vol = vol / b.box[d] * even;
    b.box[d] = (uint32_t)even;
  };
  // runs of 16, then of 32 elements on either side, then whatever fits
  for (const uint64_t run : {16ull, 32ull, 1ull << 31})
    for (const int* order : {in, out}) {
      uint64_t have = 1;
      for (int i = 0; i < r && have < run; ++i) {
        widen(order[i], (run + have - 1) / have);
        if (b.box[order[i]] < md.ext[order[i]]) break;
        have *= b.box[order[i]];
      }
    }
  b.n = (uint32_t)vol;
  b.boxes = 1;
  for (int d = 0; d < r; ++d) {
    const uint32_t nb = md.ext[d] ? (md.ext[d] + b.box[d] - 1) / b.box[d] : 0;
    b.grid[d] = FastDiv::make(std::max(1u, nb));
    b.boxes *= nb;
  }
  if (md.n == 0) b.boxes = 0;
  // shared-memory pitches: modulo the 16 banks of 8 bytes the destination's
  // fastest dimension walks by one and its second one continues it
  uint32_t pitch[kMaxDims], p = 1;
  const auto assign = [&](bool pad) {
    p = 1;
    int lead[2] = {-1, -1}, nl = 0;
    for (int i = 0; i < r && nl < 2; ++i)
      if (b.box[out[i]] > 1) lead[nl++] = out[i];
    for (int i = 0; i < r; ++i) pitch[i] = 0;
    for (int i = 0; i < r; ++i) {
      const int d = in[i];
      if (b.box[d] == 1) continue;
      if (pad && d == lead[0]) p += (1u - p) & 15u;
      if (pad && d == lead[1] && b.box[lead[0]] < 16) p += (b.box[lead[0]] - p) & 15u;
      pitch[d] = p;
      p *= b.box[d];
    }
  };
  assign(true);
  if (b.staged && p > (uint32_t)kBoxSmem) assign(false);  // (the box itself always fits)
  if (!b.staged)
    for (int d = 0; d < r; ++d) pitch[d] = (uint32_t)md.sstr[d];
  const bool src_even = pairs && md.src % 2 == 0, dst_even = pairs && md.dst % 2 == 0;
  if (b.staged) {
    b.in = make_order(b, in, md.sstr, pitch, false);
    b.out = make_order(b, out, md.dstr, pitch, dst_even);
  } else {
    // 16-byte loads too: the fastest dimension is contiguous in the source and its starts are even
    bool both = src_even && dst_even && md.sstr[out[0]] == 1;
    for (int d = 0; d < r && both; ++d) both = d == out[0] || md.sstr[d] % 2 == 0;
    b.out = make_order(b, out, md.dstr, pitch, both);
  }
  return b;
}

// Box size for a call that moves `total` elements: smaller boxes where whole
// ones would leave SMs idle.
uint32_t box_target(int64_t total) {
  return total >= (int64_t)kBoxElems * 152 * 2 ? kBoxElems : total >= 1024ll * 152 ? 1024u : 512u;
}

// Offsets inside a box are 32-bit.
bool box_fits(const MoveDesc& m) {
  int64_t s = 0, d = 0;
  for (int i = 0; i < m.rank; ++i) {
    if (m.sstr[i] < 0 || m.dstr[i] < 0) return false;
    s += (int64_t)(m.ext[i] - 1) * m.sstr[i];
    d += (int64_t)(m.ext[i] - 1) * m.dstr[i];
  }
  return m.n == 0 || (s < (1ll << 32) && d < (1ll << 32));
}

}  // namespace

int run_move_one(const MoveDesc& md, const double* src, double* dst, double alpha, cudaStream_t st) {
  if (md.n == 0) return GBX_OK;
  if (!box_fits(md)) return fail(GBX_EUNSUPPORTED, "move spans 2^32 elements or more");
  OneMove a;
  a.m = make_box(md, box_target(md.n), (((uintptr_t)src | (uintptr_t)dst) & 15) == 0);
  a.per = FastDiv::make(a.m.boxes);
  a.block = 0;
  GBX_TRY(launch(box_one_kernel, a.m.boxes, kBoxThreads, st, a, src, dst, alpha));
  return GBX_OK;
}

// Blocks of more permutations than a launch carries: sorted by permutation
// (their order does not matter), so that consecutive ones share a launch and
// each permutation is cut into boxes once.  (Launches of consecutive blocks,
// up to the one that brings a 17th permutation, were one to every 27 blocks of
// 24 permutations in random order: 5000 8^4 blocks 1340 us, 546 with one launch and uploaded descriptors; 65 so.)
static int run_block_list(const std::vector<BoxMove>& b, const std::vector<int>& which, int64_t block_elems,
                          const double* src, double* dst, cudaStream_t st) {
  std::vector<uint32_t> end(b.size() + 1, 0);
  for (int w : which) ++end[w + 1];
  for (size_t i = 1; i <= b.size(); ++i) end[i] += end[i - 1];
  std::vector<uint32_t> next(end.begin(), end.end() - 1), order(which.size());
  for (size_t k = 0; k < which.size(); ++k) order[next[which[k]]++] = (uint32_t)k;
  MoveList a;
  a.block = block_elems;
  for (size_t m0 = 0; m0 < b.size(); m0 += kSetDescs) {
    const size_t m1 = std::min(b.size(), m0 + kSetDescs);
    uint32_t per = 0;
    for (size_t i = m0; i < m1; ++i) per = std::max(per, b[i].boxes);
    std::copy(b.begin() + m0, b.begin() + m1, a.m);
    a.per = FastDiv::make(per);
    const uint32_t most = (uint32_t)std::min<int64_t>(kListBlocks, ((1ll << 31) - 1) / per);
    for (uint32_t k0 = end[m0]; k0 < end[m1]; k0 += most) {
      const uint32_t n = std::min(most, end[m1] - k0);
      std::copy(order.begin() + k0, order.begin() + k0 + n, a.id);
      for (uint32_t k = 0; k < n; ++k) a.which[k] = (uint8_t)(which[a.id[k]] - m0);
      GBX_TRY(launch(box_list_kernel, n * per, kBoxThreads, st, a, src, dst));
    }
  }
  return GBX_OK;
}

int run_block_moves(const std::vector<MoveDesc>& moves, const std::vector<int>& which, int64_t nblocks,
                    int64_t block_elems, const double* src, double* dst, cudaStream_t st) {
  if (nblocks == 0 || block_elems == 0) return GBX_OK;
  const uint32_t target = box_target(nblocks * block_elems);
  std::vector<BoxMove> b;
  uint32_t per = 0;
  const bool pairs = (((uintptr_t)src | (uintptr_t)dst) & 15) == 0 && block_elems % 2 == 0;
  for (const MoveDesc& m : moves) {
    if (!box_fits(m)) return fail(GBX_EUNSUPPORTED, "block spans 2^32 elements or more");
    b.push_back(make_box(m, target, pairs));
    per = std::max(per, b.back().boxes);
  }
  if (b.size() > (size_t)kSetDescs) return run_block_list(b, which, block_elems, src, dst, st);
  // blocks of a launch: the table's size, and a grid below 2^31
  const int64_t most = std::min<int64_t>(moves.size() == 1 ? (1ll << 31) : kSetBlocks, ((1ll << 31) - 1) / per);
  for (int64_t b0 = 0; b0 < nblocks; b0 += most) {
    const int64_t nb = std::min(most, nblocks - b0);
    const double* s = src + b0 * block_elems;
    double* d = dst + b0 * block_elems;
    const unsigned grid = (unsigned)(nb * per);
    const auto fill = [&](auto& a) {
      a.per = FastDiv::make(per);
      a.block = block_elems;
    };
    if (moves.size() == 1) {
      OneMove a;
      a.m = b[0];
      fill(a);
      GBX_TRY(launch(box_one_kernel, grid, kBoxThreads, st, a, s, d, 1.0));
    } else {
      const auto run = [&](auto& a, auto kernel) {
        std::copy(b.begin(), b.end(), a.m);
        fill(a);
        std::copy(which.begin() + b0, which.begin() + b0 + nb, a.which);
        return launch(kernel, grid, kBoxThreads, st, a, s, d);
      };
      if (nb <= kSmallSet) {
        MoveTable<kSmallSet> a;
        GBX_TRY(run(a, box_set_kernel<kSmallSet>));
      } else {
        MoveTable<kSetBlocks> a;
        GBX_TRY(run(a, box_set_kernel<kSetBlocks>));
      }
    }
  }
  return GBX_OK;
}

// ---- big-matrix packs ----------------------------------------------------------

namespace {

// Tiles [first, first + n) of the matrix, row-major over its block grid.
template <typename S, int kTiles>
struct PackTable {
  uint32_t rows, cols;   // of a tile
  FastDiv fcols;         // columns of a tile, or pairs of them
  FastDiv per;           // chunks per tile
  uint32_t chunk;        // elements (or pairs) per chunk
  uint32_t first, ncols; // first tile; tiles per matrix row
  S slot[kTiles];
};

constexpr int kPackChunk = 2048;  // elements of a work item

// One chunk of one tile: T = double, or double2 where every run is even and
// 16-byte aligned.
template <typename T, bool kToBig, class Table>
__global__ void __launch_bounds__(kBoxThreads) pack_kernel(const __grid_constant__ Table a,
                                                           const double* __restrict__ src, double* __restrict__ dst) {
  begin_dependent();
  constexpr int kPer = kPackChunk / kBoxThreads / (int)(sizeof(T) / sizeof(double));
  const uint32_t tile = a.per.div(blockIdx.x), e0 = (blockIdx.x - tile * a.per.d) * a.chunk;
  const uint32_t at = a.first + tile, r = at / a.ncols, c = at - r * a.ncols;
  const uint32_t w = a.fcols.d, n = a.rows * w;
  const int64_t pitch = (int64_t)a.ncols * w;
  const T* s = reinterpret_cast<const T*>(src);
  T* d = reinterpret_cast<T*>(dst);
  const int64_t big = (int64_t)r * a.rows * pitch + (int64_t)c * w, own = (int64_t)a.slot[tile] * n;
  T x[kPer];
  int64_t to[kPer];
#pragma unroll
  for (int k = 0; k < kPer; ++k) {
    const uint32_t e = e0 + k * kBoxThreads + threadIdx.x;
    const uint32_t row = a.fcols.div(e);
    const int64_t m = big + (int64_t)row * pitch + (e - row * w), t = own + e;
    to[k] = e < n ? (kToBig ? m : t) : -1;
    if (e < n) x[k] = __ldg(s + (kToBig ? t : m));
  }
#pragma unroll
  for (int k = 0; k < kPer; ++k)
    if (to[k] >= 0) d[to[k]] = x[k];
}

template <class Table>
int launch_pack(const Table& a, unsigned grid, bool pairs, bool to_big, const double* src, double* dst,
                cudaStream_t st) {
  if (pairs && to_big) GBX_TRY(launch(pack_kernel<double2, true, Table>, grid, kBoxThreads, st, a, src, dst));
  else if (pairs) GBX_TRY(launch(pack_kernel<double2, false, Table>, grid, kBoxThreads, st, a, src, dst));
  else if (to_big) GBX_TRY(launch(pack_kernel<double, true, Table>, grid, kBoxThreads, st, a, src, dst));
  else GBX_TRY(launch(pack_kernel<double, false, Table>, grid, kBoxThreads, st, a, src, dst));
  return GBX_OK;
}

}  // namespace

int run_pack(int64_t rows, int64_t cols, int64_t nrows, int64_t ncols, const std::vector<int>& slots, bool to_big,
             const double* src, double* dst, cudaStream_t st) {
  const int64_t n = rows * cols, tiles = nrows * ncols;
  if (n == 0 || tiles == 0) return GBX_OK;
  if (n >= (1ll << 31) || tiles >= (1ll << 31)) return fail(GBX_EUNSUPPORTED, "big matrix too large");
  const bool pairs = cols % 2 == 0 && (((uintptr_t)src | (uintptr_t)dst) & 15) == 0;
  const uint32_t width = (uint32_t)(pairs ? cols / 2 : cols);
  const uint32_t chunk = pairs ? kPackChunk / 2 : kPackChunk;
  const uint32_t per = (uint32_t)((rows * width + chunk - 1) / chunk);
  const auto go = [&](auto& a, int64_t t0, int64_t nt) {
    a.rows = (uint32_t)rows;
    a.cols = (uint32_t)cols;
    a.fcols = FastDiv::make(width);
    a.per = FastDiv::make(per);
    a.chunk = chunk;
    a.first = (uint32_t)t0;
    a.ncols = (uint32_t)ncols;
    std::copy(slots.begin() + t0, slots.begin() + t0 + nt, a.slot);
    return launch_pack(a, (unsigned)(nt * per), pairs, to_big, src, dst, st);
  };
  const bool wide = *std::max_element(slots.begin(), slots.end()) > 65535;
  const int64_t most = std::max<int64_t>(1, std::min<int64_t>(wide ? kPackTiles / 2 : kPackTiles, ((1ll << 31) - 1) / per));
  for (int64_t t0 = 0; t0 < tiles; t0 += most) {
    const int64_t nt = std::min(most, tiles - t0);
    if (wide) {
      PackTable<uint32_t, kPackTiles / 2> a;
      GBX_TRY(go(a, t0, nt));
    } else if (nt <= kSmallPack) {
      PackTable<uint16_t, kSmallPack> a;
      GBX_TRY(go(a, t0, nt));
    } else {
      PackTable<uint16_t, kPackTiles> a;
      GBX_TRY(go(a, t0, nt));
    }
  }
  return GBX_OK;
}

}  // namespace gbx
