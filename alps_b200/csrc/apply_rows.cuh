// apply_rows.cuh -- y = H x over bundles of hi blocks whose x lies interleaved
// in shared memory: the apply of the single-instance and of the batched engine.
//
// The tile apply (apply.cuh) spends 20 to 30 instructions on every term of a
// row: bounds and padding tests per term, a table entry and a coupling per term
// and block, the test for the diagonal's column.  Here
//   * x of the bundle's B blocks is staged row by row (row r of all B blocks
//     side by side, 16 or 8 bytes), so that one lo-table entry, one coupling
//     and one shared load serve the lo-part flip of all B blocks;
//   * the lo table comes in slices of 32 rows (launch_lo_slices), each as wide
//     as its longest row, the entries of smaller targets before those of
//     larger ones: a warp walks its slice with a uniform trip count, the
//     diagonal falls between the two parts, and a padding entry adds 0 * 0
//     from a row of zeros (a row's sum is never -0, so that changes no bit);
//   * an entry holds the byte offsets of its x row and of its coupling;
//   * the flips outside the lo part come from a program formed once per handle,
//     their loads out together for all blocks.
// Rows add their terms in the order of the tile apply (FP64: the explicit
// matrix's columns), and the <x, y> partials have their thread order and tree:
// they are formed from the finished rows, after the bundle.
//
// Bound by the latency of the x loads outside the lo part (L2 and, above its
// size, DRAM) behind 32 warps per SM; part costs on 6x5 FP32 (of 3.93 ms, a copy
// with one part left out): hi-part flips 1.15 ms, crossing 1.48, lo-part 0.83;
// L=28 FP64 (of 1.34 ms, before hi_terms had its short form): outside the lo
// part 0.83, lo-part 0.29.
// Measured (applies in a row, with partials, us; in brackets the apply before:
// one block of x in shared memory, 4 rows per thread, L2 flushed between its
// applies): J1-J2 chain L=28 FP64 1173 (1684), FP32 771 (1102); 6x5 FP32 3870
// (5570); L=24 FP64 84 (133), FP32 64 (88).
//
// Reference paths are relative to the ALPS source tree.
#pragma once

#include "apply.cuh"

namespace aed {
namespace rapply {

using apply::ApplyCtx;
using apply::kTileRows;
using apply::SPair;
using apply::TileOp;

constexpr int kMaxB = 4;
// Flips (of all blocks; FP32: hi-part / crossing ones) whose loads go out
// together.  They fill the 64 registers of 1024 threads per SM without a spill;
// eight, or four crossing ones, spill and were 5-25 % slower on L=28 and 6x5.
constexpr int kU = 4, kUC = 2;
constexpr uint32_t kNullNb = 0x80000001u;  // FP32: an op that no row takes (no byte offset of an element)
// FP64 ops, TileOp::mc: 0 a hi-part flip; a crossing flip has kCrossFlip, its
// column of the crossing table (lo bit << Nlo, 20 bits) and, where the lo bit
// must be set, kWantSet, the bits that the table's sign-extended entry then
// has; kNullFlip: no row takes it.  kNoCross on the first op of a group of kU
// ops: none of the group's ops, of any block, is a crossing flip.
constexpr uint32_t kWantSet = 0xa0000000u, kNullFlip = 0x20000000u, kCrossFlip = 1u << 20, kNoCross = 1u << 30;
constexpr int kMaxItems = 32;  // (block, tile) pairs of a bundle: 4 blocks of at most 7 tiles

template <typename T, int B>
struct alignas(sizeof(T) * B) RowVec {
  T v[B];
};

struct RowsSmem {
  double lolo_c[kMaxBonds + 1];  // the last: 0, of the padding entries
  double red[kMaxItems][kHvThreads / 32];
  uint32_t ticket[2];  // Taker::slot
};

// A bundle's program: a head, then the flips outside the lo part that apply to
// its blocks, op o of all B blocks side by side.
//   FP64 (rows in column order): ops[o * B + j], the flips to smaller states in
//   [0, n1), those to larger ones in [n1, n1 + n2);
//   FP32: c[o * B + j] and nb[o * B + j], the hi-part flips at o < n1, the
//   crossing ones in [n1, n1 + n2) with their lo bit and required values in bits[o].
// Lists are as long as the longest block's, rounded up to a multiple of two
// (FP32 crossing flips: of kUC), filled with null ops.  Programs depend on the couplings alone: a
// handle forms them once (launch_row_progs), `cap` ops each, and a CTA copies
// the next bundle's while it runs one.  (Listed in the apply, by a warp per
// block while the others staged x, they put a chain of dependent loads and a
// barrier before every bundle.)
struct RowHead {
  uint32_t first[kMaxB], tile[kMaxB];  // first row and tile of each block
  uint32_t lbase, nk;                  // lo class offset and rows per block
  int32_t k, nv;                       // lo popcount, blocks (0: none)
  int32_t n1, n2, full, pad;           // ops of the lists; FP32 hi-part ops that every block has
};
static_assert(sizeof(RowHead) == 64, "a multiple of 16 bytes");
struct Program {
  TileOp* ops;
  uint32_t* nb;
  double* c;
  uint32_t* bits;
};
template <int B>
__host__ __device__ inline Program program_at(unsigned char* p, int cap) {
  Program g;
  g.ops = reinterpret_cast<TileOp*>(p + sizeof(RowHead));
  g.c = reinterpret_cast<double*>(p + sizeof(RowHead));
  g.nb = reinterpret_cast<uint32_t*>(g.c + (size_t)cap * B);
  g.bits = g.nb + (size_t)cap * B;
  return g;
}
// Bytes of one program of `cap` ops (cap even).
__host__ __device__ inline int prog_stride(int B, int elem, int cap) {
  const int b = (int)sizeof(RowHead) + cap * (elem == 8 ? B * 16 : B * 12 + 4);
  return (b + 15) & ~15;
}

// Dynamic shared memory: x rows (and the row of zeros) and two programs.
__host__ __device__ inline size_t rows_smem_bytes(int row_bytes, int maxrows, int stride) {
  return (((size_t)(maxrows + 1) * row_bytes + 15) & ~(size_t)15) + 2 * (size_t)stride;
}

// The value at a 32-bit byte offset (an FP32 vector of at most 2^30 rows; the
// largest sector has 601 M): one add per address.
template <typename T>
__device__ __forceinline__ T at_byte(const T* p, uint32_t off) {
  return *reinterpret_cast<const T*>(reinterpret_cast<const char*>(p) + off);
}

// The lo-part flips of one part of the slice: np pairs of entries.
template <typename T, typename Acc, int B>
__device__ __forceinline__ void lo_terms(const uint2* __restrict__ tp, int np, const unsigned char* xs,
                                         const unsigned char* cs, Acc (&acc)[B]) {
  constexpr int kShift = sizeof(T) * B == 16 ? 0 : 1;
  auto term = [&](uint32_t e) {
    const double c = *reinterpret_cast<const double*>(cs + (e >> 20));
    const RowVec<T, B> x = *reinterpret_cast<const RowVec<T, B>*>(xs + ((e & 0xfffffu) >> kShift));
#pragma unroll
    for (int j = 0; j < B; ++j) acc[j].add(c, x.v[j]);
  };
  // two pairs of entries ahead of the terms
  uint2 a{}, b{};
  if (np > 0) a = __ldg(tp);
  if (np > 1) b = __ldg(tp + 32);
#pragma unroll 1
  for (int p = 0; p < np; p += 2) {
    const uint2 e = a, f = b;
    tp += 64;
    if (p + 2 < np) a = __ldg(tp);
    if (p + 3 < np) b = __ldg(tp + 32);
    term(e.x);
    term(e.y);
    if (p + 1 < np) {
      term(f.x);
      term(f.y);
    }
  }
}

// FP64: U ops of every block: their loads first, then the terms in order.  A
// crossing flip that the row does not take adds c * 0, as a null op adds
// 0 * 0: neither changes a sum that is never -0 (the couplings are finite).
template <typename T, typename Acc, int B, int U, bool CROSS>
__device__ __forceinline__ void hi_group(const TileOp* ops, uint32_t r, const int16_t* __restrict__ xt,
                                         const T* x, Acc (&acc)[B]) {
  T xv[U][B];
  double c[U][B];
#pragma unroll
  for (int v = 0; v < U; ++v)
#pragma unroll
    for (int j = 0; j < B; ++j) {
      const TileOp e = ops[v * B + j];
      c[v][j] = e.c;
      uint32_t at = r;
      if (CROSS && e.mc != 0u) at = (uint32_t)(int)__ldg(xt + (e.mc & 0xfffffu));
      xv[v][j] = T(0);
      if (((CROSS ? at ^ e.mc : e.mc) & (CROSS ? kWantSet : kNullFlip)) == 0u) xv[v][j] = x[e.nb + at];
    }
#pragma unroll
  for (int v = 0; v < U; ++v)
#pragma unroll
    for (int j = 0; j < B; ++j) acc[j].add(c[v][j], xv[v][j]);
}

// FP64: n ops of every block (n even), U at a time and a last two.  Groups
// without a crossing flip, marked when the program is formed, skip the table
// load, its address and the test of its entry: on the chain L=28 the apply issues
// in 73 % of its cycles and spends 60 % of its time here.  Together with the
// remainder of two (the lists were padded to four) chain L=28 1191 -> 1124 us,
// 5x5 with 11 up 138 -> 129.  The choice made per block of the bundle takes the short
// form more often, but waits for one block's table entries before the other's
// loads go out: 1218 and 140 us.
template <typename T, typename Acc, int B, int U>
__device__ __forceinline__ void hi_terms(const TileOp* ops, int n, uint32_t r, const int16_t* __restrict__ xt,
                                         const T* x, Acc (&acc)[B]) {
  static_assert(U == 4, "a remainder of two");
  int o = 0;
#pragma unroll 1
  for (; o + U <= n; o += U) {
    if (ops[o * B].mc & kNoCross)
      hi_group<T, Acc, B, U, false>(ops + o * B, r, xt, x, acc);
    else
      hi_group<T, Acc, B, U, true>(ops + o * B, r, xt, x, acc);
  }
  if (o < n) hi_group<T, Acc, B, 2, true>(ops + o * B, r, xt, x, acc);
}

// FP32: hi-part flips [0, n) of every block (n even), of which those below
// nfull are real for all of them.  rb: the row's rank in bytes.
template <typename T, typename Acc, int B, int U>
__device__ __forceinline__ void hihi_terms(const Program& pg, int nfull, int n, uint32_t rb,
                                           const T* x, Acc (&acc)[B]) {
  using NB = RowVec<uint32_t, B>;
  using CB = RowVec<double, B == 1 ? 1 : 2>;
  auto add = [&](int o, const T (&xv)[B]) {
    const CB* c = reinterpret_cast<const CB*>(pg.c + o * B);
#pragma unroll
    for (int j = 0; j < B; ++j) acc[j].add(c[j / 2].v[j % 2], xv[j]);
  };
  int o = 0;
#pragma unroll 1
  for (; o + U <= nfull; o += U) {
    T xv[U][B];
#pragma unroll
    for (int v = 0; v < U; ++v) {
      const NB nb = *reinterpret_cast<const NB*>(pg.nb + (o + v) * B);
#pragma unroll
      for (int j = 0; j < B; ++j) xv[v][j] = at_byte(x, nb.v[j] + rb);
    }
#pragma unroll
    for (int v = 0; v < U; ++v) add(o + v, xv[v]);
  }
  constexpr int UT = 2;
#pragma unroll 1
  for (; o < n; o += UT) {  // null ops among them: 0 * 0
    T xv[UT][B];
#pragma unroll
    for (int v = 0; v < UT; ++v) {
      const NB nb = *reinterpret_cast<const NB*>(pg.nb + (o + v) * B);
#pragma unroll
      for (int j = 0; j < B; ++j) xv[v][j] = nb.v[j] != kNullNb ? at_byte(x, nb.v[j] + rb) : T(0);
    }
#pragma unroll
    for (int v = 0; v < UT; ++v) add(o + v, xv[v]);
  }
}

// FP32: crossing flips [o0, o0 + n), n a multiple of U: op o of every block
// names the same lo bit, so one table load serves them all; the table entries
// of the next U ops are asked for ahead.  A flip that the row does not take
// adds c * 0.
template <typename T, typename Acc, int B, int U>
__device__ __forceinline__ void cross_terms(const Program& pg, int o0, int n, const uint16_t* __restrict__ xt, int Nlo,
                                            const T* x, Acc (&acc)[B]) {
  using NB = RowVec<uint32_t, B>;
  using CB = RowVec<double, B == 1 ? 1 : 2>;
  if (n == 0) return;
  uint32_t at[U], next[U];
#pragma unroll
  for (int v = 0; v < U; ++v) next[v] = __ldg(xt + ((pg.bits[o0 + v] >> 16) << Nlo));
#pragma unroll 1
  for (int o = o0; o < o0 + n; o += U) {
    T xv[U][B];
#pragma unroll
    for (int v = 0; v < U; ++v) {
      at[v] = next[v];
      const uint32_t bits = pg.bits[o + v];  // bit j: block j wants the lo bit set; bit 8 + j: clear
      const uint32_t m = at[v] & 0x8000u ? bits : bits >> 8;
      const uint32_t ab = (at[v] & 0x7fffu) * (uint32_t)sizeof(T);
      const NB nb = *reinterpret_cast<const NB*>(pg.nb + (o + v) * B);
#pragma unroll
      for (int j = 0; j < B; ++j) xv[v][j] = m & 1u << j ? at_byte(x, nb.v[j] + ab) : T(0);
    }
    if (o + U < o0 + n) {
#pragma unroll
      for (int v = 0; v < U; ++v) next[v] = __ldg(xt + ((pg.bits[o + U + v] >> 16) << Nlo));
    }
#pragma unroll
    for (int v = 0; v < U; ++v) {
      const CB* c = reinterpret_cast<const CB*>(pg.c + (o + v) * B);
#pragma unroll
      for (int j = 0; j < B; ++j) acc[j].add(c[j / 2].v[j % 2], xv[v][j]);
    }
  }
}

// One warp: emit(position, pair) for the flips of `list` outside the lo part
// that apply to some rows of block h, in list order from position n on:
// kind 0 those with the condition's bits (either kind of flip), 1 the hi-part
// flips in either direction, 2 the crossing flips in either direction.
// Returns the position after the last.
template <class Emit>
__device__ __forceinline__ int walk_list(const SPair* list, int np, uint32_t h, int Nlo, uint32_t lm, int kind, int n,
                                         Emit&& emit) {
  const int lane = threadIdx.x & 31;
  for (int q0 = 0; q0 < np; q0 += 32) {
    const int q = q0 + lane;
    bool on = false;
    SPair e{};
    if (q < np) {
      e = list[q];
      const uint32_t fhi = e.flip >> Nlo, flo = e.flip & lm;
      on = kind == 0   ? fhi != 0u && (h & fhi) == e.cond >> Nlo
           : kind == 1 ? flo == 0u && __popc(h & fhi) == 1
                       : flo != 0u && fhi != 0u;
    }
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (on) emit(n + __popc(m & ((1u << lane) - 1u)), e);
    n += __popc(m);
  }
  return n;
}

// One warp compiles block j's (hi part h) column of the program.  FP64: lists
// of l1 and l2 ops; FP32: l1 hi-part ops, then l2 crossing ones.
template <int B>
__device__ __forceinline__ void compile_f64(const ApplyCtx& c, const uint32_t* __restrict__ thi, const SPair* low,
                                            const SPair* rise, uint32_t h, int j, int l1, int l2, TileOp* ops) {
  auto emit = [&](int at, const SPair& e) {
    const uint32_t flo = e.flip & c.lm, nb = __ldg(thi + (h ^ (e.flip >> c.Nlo)));
    const uint32_t v = (e.cond & c.lm) != 0u ? 1u : 0u;
    // (a sign-extended table entry is the rank - v 2^15)
    ops[at * B + j] = flo == 0u ? TileOp{0u, nb, e.c}
                                : TileOp{kCrossFlip | (uint32_t)(__ffs(flo) - 1) << c.Nlo | (v ? kWantSet : 0u),
                                         nb + (v << 15), e.c};
  };
  const int lane = threadIdx.x & 31;
  int n = walk_list(low, c.np, h, c.Nlo, c.lm, 0, 0, emit);
  for (int q = n + lane; q < l1; q += 32) ops[q * B + j] = {kNullFlip, 0u, 0.0};
  n = walk_list(rise, c.np, h, c.Nlo, c.lm, 0, l1, emit);
  for (int q = n + lane; q < l1 + l2; q += 32) ops[q * B + j] = {kNullFlip, 0u, 0.0};
}

template <int B>
__device__ __forceinline__ void compile_f32(const ApplyCtx& c, const uint32_t* __restrict__ thi, const SPair* low,
                                            uint32_t h, int j, int l1, int l2, const Program& pg) {
  const int lane = threadIdx.x & 31;
  auto put = [&](int at, uint32_t nb, double cc) {  // nb: bytes (a multiple of 4), or kNullNb
    pg.nb[at * B + j] = nb;
    pg.c[at * B + j] = cc;
  };
  int n = walk_list(low, c.np, h, c.Nlo, c.lm, 1, 0, [&](int at, const SPair& e) {
    put(at, __ldg(thi + (h ^ (e.flip >> c.Nlo))) * 4u, e.c);
  });
  for (int q = n + lane; q < l1; q += 32) put(q, kNullNb, 0.0);
  n = walk_list(low, c.np, h, c.Nlo, c.lm, 2, l1, [&](int at, const SPair& e) {
    put(at, __ldg(thi + (h ^ (e.flip >> c.Nlo))) * 4u, e.c);
    const uint32_t b = (uint32_t)(__ffs(e.flip & c.lm) - 1);
    // the lo bit must differ from the hi bit: set where h's is clear
    const uint32_t want = b << 16 | 1u << (h & (e.flip >> c.Nlo) ? 8 + j : j);
    pg.bits[at] = j == 0 ? want : pg.bits[at] | want;
  });
  for (int q = n + lane; q < l1 + l2; q += 32) {
    put(q, 0u, 0.0);
    pg.bits[q] = 0u;
  }
}

// One warp: lengths of the lists of bundle ub (rounded up) and, FP32, the
// hi-part ops that every block has.
template <typename T, int B, int U, int UC>
__device__ __forceinline__ int list_lengths(const ApplyCtx& c, const DevTables& t, int64_t ub, const SPair* low,
                                            const SPair* rise, int* n1, int* n2, int* full) {
  constexpr bool kOrdered = sizeof(T) == 8;
  auto none = [](int, const SPair&) {};
  int nv = 0, l1 = 0, l2 = 0, f = 1 << 20;
  for (int j = 0; j < B; ++j) {
    const uint32_t h = __ldg(t.blk_h + ub * B + j);
    if (h == kNoBlockEntry) break;  // real blocks come first in a bundle
    ++nv;
    const int n = walk_list(low, c.np, h, c.Nlo, c.lm, kOrdered ? 0 : 1, 0, none);
    l1 = max(l1, n);
    f = min(f, n);
    if (kOrdered || j == 0)
      l2 = max(l2, walk_list(kOrdered ? rise : low, c.np, h, c.Nlo, c.lm, kOrdered ? 0 : 2, 0, none));
  }
  *n1 = (l1 + 1) / 2 * 2;
  *n2 = kOrdered ? (l2 + 1) / 2 * 2 : (l2 + UC - 1) / UC * UC;
  *full = nv == B ? f : 0;
  return nv;
}

// One warp forms the program of bundle ub at `out` (cap ops; cap 0: only the
// length it needs, which it returns).
template <typename T, int B, int U, int UC>
__device__ __forceinline__ int form_program(const ApplyCtx& c, const DevTables& t, int64_t ub, const SPair* low,
                                            const SPair* rise, unsigned char* out, int cap) {
  constexpr bool kOrdered = sizeof(T) == 8;
  int n1, n2, full;
  const int nv = list_lengths<T, B, U, UC>(c, t, ub, low, rise, &n1, &n2, &full);
  if (cap == 0) return n1 + n2;
  const int lane = threadIdx.x & 31;
  const Program pg = program_at<B>(out, cap);
  RowHead hd{};
  hd.nv = nv;
  hd.n1 = n1;
  hd.n2 = n2;
  hd.full = full;
  for (int j = 0; j < B; ++j) {
    if (j < nv) {
      const uint32_t h = __ldg(t.blk_h + ub * B + j);
      if (j == 0) {
        hd.k = c.n_up - __popc(h);
        hd.lbase = __ldg(t.looff + hd.k);
        hd.nk = __ldg(t.looff + hd.k + 1) - hd.lbase;
      }
      hd.first[j] = __ldg(t.thi + h);
      hd.tile[j] = __ldg(t.tfirst + h);
      if constexpr (kOrdered)
        compile_f64<B>(c, t.thi, low, rise, h, j, n1, n2, pg.ops);
      else
        compile_f32<B>(c, t.thi, low, h, j, n1, n2, pg);
      __syncwarp();
    } else {  // no such block in the bundle: null ops
      for (int q = lane; q < n1 + n2; q += 32) {
        if constexpr (kOrdered) {
          pg.ops[q * B + j] = {kNullFlip, 0u, 0.0};
        } else {
          pg.nb[q * B + j] = kNullNb;
          pg.c[q * B + j] = 0.0;
        }
      }
    }
  }
  if constexpr (kOrdered) {  // the groups without crossing flips
    __syncwarp();
    const int g1 = n1 / U, g2 = n2 / U;
    for (int g = lane; g < g1 + g2; g += 32) {
      TileOp* o = pg.ops + (g < g1 ? g * U : n1 + (g - g1) * U) * B;
      uint32_t any = 0u;
      for (int q = 0; q < U * B; ++q) any |= o[q].mc;
      if (!(any & kCrossFlip)) o->mc |= kNoCross;
    }
  }
  if (lane == 0) *reinterpret_cast<RowHead*>(out) = hd;
  return n1 + n2;
}

// Bundles handed out on demand: a CTA works on bundles blockIdx.x and
// blockIdx.x + gridDim.x, then on what it draws from a counter, so that a
// sector with a few bundles per CTA, the large ones first, ends evenly.  A draw
// is made a whole bundle before its answer is needed, as the next bundle's
// program is fetched a bundle ahead.  Every CTA stops at its first draw past
// the end, so an apply over nb > 2 gridDim.x bundles makes nb - gridDim.x
// draws, and the CTA that holds the last one zeroes the counter for the
// handle's next apply, which reads it only after this one.  Rows and partials
// do not depend on who forms them.
struct Taker {
  uint32_t* word;
  uint32_t* slot;  // two words of shared memory, taken in turn
  uint32_t nb, drawn;
  __device__ __forceinline__ Taker(uint32_t* w, uint32_t* s, uint32_t n)
      : word(w), slot(s), nb(n), drawn(blockIdx.x + gridDim.x) {}
  // thread 0, before the barrier that precedes take(w)
  __device__ __forceinline__ void publish(int w) {
    if (threadIdx.x == 0) {
      slot[w] = drawn;
      if (drawn == nb + gridDim.x - 1u) *word = 0u;
    }
  }
  // every thread, after that barrier; the next publish(w) is two barriers on
  __device__ __forceinline__ uint32_t take(int w) {
    const uint32_t b = slot[w];
    if (b < nb && threadIdx.x == 0) drawn = 2u * gridDim.x + atomicAdd(word, 1u);
    return b;
  }
};

// A program on its way from `src` into shared memory (every thread; waited for
// by the next rows_bundle).
template <int NT>
__device__ __forceinline__ void fetch_program(const unsigned char* src, unsigned char* dst, int bytes) {
  for (int i = (int)threadIdx.x * 16; i < bytes; i += NT * 16) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + i);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + i) : "memory");
  }
}

// The bundle whose program is in (or on its way into) prog.  fetch_next() is
// called by every thread once nobody reads the previous bundle's program any
// more: it starts the copy of the next one's.
template <typename T, typename Acc, int B, int NT, int U, int UC, class Next>
__device__ __forceinline__ void rows_bundle(const DevTables& t, const T* x, T* y, double* alpha_part,
                                            RowsSmem& sm, unsigned char* xs,
                                            unsigned char* prog, int cap, Next&& fetch_next) {
  constexpr bool kOrdered = sizeof(T) == 8;
  using Row = RowVec<T, B>;
  Row* rows = reinterpret_cast<Row*>(xs);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();  // this program is here; the previous bundle is done with x, red and its program
  if (!kOrdered) fetch_next();
  const RowHead& hd = *reinterpret_cast<const RowHead*>(prog);
  const Program pg = program_at<B>(prog, cap);
  const int nv = hd.nv;
  if (nv == 0) {  // padding of the block list
    if (kOrdered) fetch_next();
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t lbase = hd.lbase, nk = hd.nk;
  uint32_t bj[B];
#pragma unroll
  for (int j = 0; j < B; ++j) bj[j] = hd.first[j];
  // x of the blocks, row by row, two rows in flight per thread
  for (uint32_t i = threadIdx.x; i < nk; i += 2 * NT) {
    Row a, b;
    const bool two = i + NT < nk;
#pragma unroll
    for (int j = 0; j < B; ++j) {
      a.v[j] = j < nv ? x[bj[j] + i] : T(0);
      b.v[j] = j < nv && two ? x[bj[j] + i + NT] : T(0);
    }
    rows[i] = a;
    if (two) rows[i + NT] = b;
  }
  // FP64: behind the loads of x (chain L=26, 512 threads, 350 us a product when
  // it stood before them, now 332; FP32 6x5 3754 us here, 3575 before them)
  if (kOrdered) fetch_next();
  __syncthreads();
  const int n1 = hd.n1, n2 = hd.n2, full = hd.full, Nlo = t.Nlo;
  const unsigned char* cs = reinterpret_cast<const unsigned char*>(sm.lolo_c);
  const uint32_t s0 = (lbase >> 5) + (uint32_t)hd.k;
#pragma unroll 1
  for (uint32_t r = threadIdx.x; r < nk; r += NT) {
    const uint16_t* xt = t.xtab + lbase + r;
    const int16_t* xs16 = reinterpret_cast<const int16_t*>(xt);
    const uint32_t s = s0 + (r >> 5);
    const uint32_t w = __ldg(t.low_w + s);
    const uint2* tp = t.low_e + ((size_t)s * t.low_st * 32 + lane);
    const int wl = (int)(w & 0xffffu), wu = (int)(w >> 16);
    Acc acc[B];
    if (kOrdered) {
      double dg[B];
#pragma unroll
      for (int j = 0; j < B; ++j) dg[j] = j < nv ? __ldg(t.dg + bj[j] + r) : 0.0;
      hi_terms<T, Acc, B, U>(pg.ops, n1, r, xs16, x, acc);
      lo_terms<T, Acc, B>(tp, wl, xs, cs, acc);
      {
        const Row own = rows[r];
#pragma unroll
        for (int j = 0; j < B; ++j) acc[j].add(dg[j], own.v[j]);
      }
      lo_terms<T, Acc, B>(tp + wl * 32, wu, xs, cs, acc);
      hi_terms<T, Acc, B, U>(pg.ops + n1 * B, n2, r, xs16, x, acc);
    } else {
      const Row own = rows[r];
#pragma unroll
      for (int j = 0; j < B; ++j)
        if (j < nv) acc[j].add(apply::diag_fp32(t, bj[j] + r), own.v[j]);
      hihi_terms<T, Acc, B, U>(pg, full, n1, r * (uint32_t)sizeof(T), x, acc);
      cross_terms<T, Acc, B, UC>(pg, n1, n2, xt, Nlo, x, acc);
      lo_terms<T, Acc, B>(tp, wl + wu, xs, cs, acc);
    }
#pragma unroll
    for (int j = 0; j < B; ++j)
      if (j < nv) y[bj[j] + r] = acc[j].value();
  }
  if (!alpha_part) return;
  // <x, y> of every (block, tile): threads of a tile as in the tile apply,
  // row r0 + thread + 256 i in order of i; groups of 128 threads take the
  // halves of the tiles in turn
  __syncthreads();  // the bundle's rows of y are written
  const uint32_t nt = (nk + kTileRows - 1) / kTileRows;
  const int items = nv * (int)nt;
  constexpr int kHalf = kHvThreads / 2;
  for (int q = threadIdx.x / kHalf; q < 2 * items; q += NT / kHalf) {
    const int it = q >> 1;
    const uint32_t th = threadIdx.x % kHalf + (q & 1 ? kHalf : 0);
    const int j = it / (int)nt;
    const uint32_t r0 = (uint32_t)(it - j * (int)nt) * kTileRows;
    const uint32_t base = hd.first[j];
    double dot = 0.0;
#pragma unroll
    for (int i = 0; i < kTileRows / kHvThreads; ++i) {
      const uint32_t r = r0 + th + i * kHvThreads;
      if (r < nk) dot = fma((double)rows[r].v[j], (double)y[base + r], dot);
    }
    for (int o = 16; o > 0; o >>= 1) dot += __shfl_down_sync(0xffffffffu, dot, o);
    if (lane == 0) sm.red[it][th >> 5] = dot;
  }
  __syncthreads();
  for (int it = warp; it < items; it += NT / 32) {
    const int j = it / (int)nt;
    const uint32_t first = hd.tile[j];
    double r = lane < kHvThreads / 32 ? sm.red[it][lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
    if (lane == 0) alpha_part[first + (uint32_t)(it - j * (int)nt)] = r;
  }
}

}  // namespace rapply
}  // namespace aed
