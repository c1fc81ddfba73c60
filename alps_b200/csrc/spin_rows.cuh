// spin_rows.cuh -- the rows apply of a spin-S sector: y = H x over bundles of
// hi blocks whose x lies interleaved in shared memory (apply_rows.cuh is the
// spin-1/2 counterpart).
//
// A bundle is B blocks of the same lo digit sum: the same lo codes, so the same
// rows and the same lo-lo terms.  Of a row's terms
//   * the bonds inside the lo word come from a table in slices of 32 rows, each
//     as wide as its longest row: an entry holds the byte offsets of the target
//     row and of its element; one entry serves all B blocks, x from shared memory;
//   * the bonds inside the hi word are the same for all rows of a block: one
//     warp per block lists their target blocks and elements, and a row adds
//     x[nb + r] (consecutive rows at consecutive addresses);
//   * the bonds across the words: the block's digit fixes the transitions
//     (hd -> hd + q), the row's digit ld the element and whether it exists; a
//     table per lo site and q names the target's rank and ld;
//   * the diagonal is the block's sum over its hi word, the lo code's sum from a
//     table and the crossing bonds' elements of (hd, ld).
// The blocks' lists are formed once per handle and couplings: listing them in
// the apply, by a warp while the others stage x, cost a chain of dependent loads
// and a barrier per bundle (spin-1 chain L=18 876 us against 833, L=12 16 against
// 8.3), and no kernel has to carry the couplings' tables any more.
// Bound by the latency of the hi-hi and crossing loads of x (L2) behind 32 warps
// per SM.  Rows agree with the walking apply to rounding (the terms come in another
// order).  The <x, y> partials are formed from the finished rows in its thread
// order and tree.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "spin.cuh"

namespace aed {

template <int B>
struct alignas(8 * B) SpinRow {
  double v[B];
};

// A block's program, formed once per handle and couplings (spin_prog_kernel) and
// copied to shared memory while the bundle before it runs: a head, then
struct SpinBlockHead {
  uint32_t first, tile, lbase, nk;  // first row and tile; its lo codes
  int k, nhh, nx;                   // lo digit sum; terms
  uint32_t hx;                      // the crossing bonds' digits
  double dg;                        // diagonal sum over the hi word (without keys)
  double pad;
};
static_assert(sizeof(SpinBlockHead) == 48, "a multiple of 16 bytes");
struct SpinBlockProg {
  uint32_t* nb;    // hi-hi terms: first row of the target block
  double* c;       // and element
  uint2* xop;      // crossing terms: first row of the target block, offset into the crossing table
  double* xc;      // and their elements, D per term (by the row's digit)
  double* xd;      // diagonal: by the key of the lo code's crossing digits, the sum over the hi word
                   // included; without keys D elements per crossing bond
};

constexpr int kSpinKeys = 81;  // most keys of a lo code's crossing digits

constexpr int kSpinRedItems = 16;  // (block, tile) partials formed at a time

struct SpinRowsSmem {
  double val[kSpinRowVals + 1];  // elements of the lo-lo terms; the last: 0, of the padding entries
  double red[kSpinRedItems][8];
};

__host__ __device__ inline size_t spin_block_prog_bytes(int d, int n_hh, int n_x, int n_key) {
  const size_t hh = ((size_t)n_hh + 3) & ~(size_t)3, xo = (size_t)n_x * (d - 1);
  const size_t b = sizeof(SpinBlockHead) + hh * 12 + xo * 8 + (xo * d + (n_key ? (size_t)n_key : (size_t)n_x * d)) * 8;
  return (b + 15) & ~(size_t)15;
}
// x rows and the row of zeros, and the programs of two bundles
__host__ __device__ inline size_t spin_rows_smem_bytes(int B, int d, int maxrows, int n_hh, int n_x, int n_key) {
  return (((size_t)(maxrows + 1) * 8 * B + 15) & ~(size_t)15) +
         2 * (size_t)B * spin_block_prog_bytes(d, n_hh, n_x, n_key);
}

template <int D>
__device__ __forceinline__ SpinBlockProg spin_block_prog(unsigned char* p, const SpinDev& t) {
  const size_t hh = ((size_t)t.n_hh + 3) & ~(size_t)3, xo = (size_t)t.n_x * (D - 1);
  SpinBlockProg g;
  g.c = reinterpret_cast<double*>(p + sizeof(SpinBlockHead));
  g.xc = g.c + hh;
  g.xd = g.xc + xo * D;
  g.xop = reinterpret_cast<uint2*>(g.xd + (t.n_key ? (size_t)t.n_key : (size_t)t.n_x * D));
  g.nb = reinterpret_cast<uint32_t*>(g.xop + xo);
  return g;
}

// One warp forms the program of block-list entry `at` (an empty one for padding).
template <class Sh, int D, int MO>
__device__ __forceinline__ void spin_compile(const Sh& sh, const SpinParams& p, const SpinDev& t, bool has_site,
                                             int64_t at, unsigned char* out) {
  constexpr int BITS = D <= 2 ? 1 : D <= 4 ? 2 : 3;
  constexpr uint32_t dm = (1u << BITS) - 1u;
  const int lane = threadIdx.x & 31, Nh = t.N - t.Nl;
  const uint32_t blk = __ldg(t.rblk + at);
  const bool real = blk != kSpinNone;
  const uint32_t h = real ? __ldg(t.blk_hi + blk) : 0u;
  int sum = 0;
  for (int i = 0; i < Nh; ++i) sum += (int)((h >> (BITS * i)) & dm);
  const int k = t.T - sum;
  int n = 0, nx = 0;
  uint32_t hx = 0u;
  double dg = 0.0;
  if (real) {
    const SpinBlockProg g = spin_block_prog<D>(out, t);
    for (int q0 = 0; q0 < p.n_bonds; q0 += 32) {
      const int q = q0 + lane;
      uint32_t kp = 0u;
      int pr = 0;
      int4 b = make_int4(0, 0, 0, 0);
      if (q < p.n_bonds) {
        b = sh.bond[q];
        if (bond_side(b) == 3) {
          pr = b.x + (int)((h >> (b.y & 255)) & dm) * D + (int)((h >> ((b.y >> 8) & 255)) & dm);
          kp = sh.pk[pr];
          dg += sh.dg[pr];
        }
      }
#pragma unroll
      for (int s = 0; s < MO; ++s) {
        const int kk = (int)(int8_t)(uint8_t)(kp >> (8 * s));
        const unsigned m = __ballot_sync(0xffffffffu, kk != 0);
        if (kk != 0) {
          const int o = n + __popc(m & ((1u << lane) - 1u));
          g.nb[o] = __ldg(t.thi + (h + (uint32_t)(kk * b.z)));
          g.c[o] = sh.ov[pr * MO + s];
        }
        n += __popc(m);
      }
    }
    if (has_site)
      for (int i = lane; i < Nh; i += 32) dg += sh.sdg[i * D + (int)((h >> (BITS * (Nh - 1 - i))) & dm)];
    for (int o = 16; o > 0; o >>= 1) dg += __shfl_xor_sync(0xffffffffu, dg, o);
    for (int q0 = 0; q0 < t.n_x; q0 += 32) {
      const int q = q0 + lane;
      SpinCross c{};
      int hd = 0;
      if (q < t.n_x) {
        c = t.cross[q];
        hd = (int)((h >> c.hshift) & dm);
        if (t.n_key == 0)
          for (int ld = 0; ld < D; ++ld) g.xd[q * D + ld] = __ldg(t.xdiag + ((size_t)q * D + hd) * D + ld);
      }
      for (int dq = -(D - 1); dq <= D - 1; ++dq) {
        if (dq == 0) continue;
        const bool on = q < t.n_x && (c.mask >> (hd * (2 * D - 1) + dq + D - 1) & 1ull) != 0ull;
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) {
          const int o = nx + __popc(m & ((1u << lane) - 1u));
          g.xop[o] = make_uint2(__ldg(t.thi + (h + (uint32_t)(dq * (1 << c.hshift)))),
                                (uint32_t)((c.tab * (2 * D - 1) + dq + D - 1) * (int)t.n_lo));
          for (int ld = 0; ld < D; ++ld)
            g.xc[o * D + ld] = __ldg(t.xoff + (((size_t)q * D + hd) * (2 * D - 1) + dq + D - 1) * D + ld);
        }
        nx += __popc(m);
      }
    }
    // by key: the hi word's sum and the crossing bonds' diagonal elements
    for (int key = lane; key < t.n_key; key += 32) {
      double v = dg;
      for (int q = 0; q < t.n_x; ++q) {
        const SpinCross c = t.cross[q];
        int ld = key;
        for (int s = 0; s < c.tab; ++s) ld /= D;
        v += __ldg(t.xdiag + ((size_t)q * D + (int)((h >> c.hshift) & dm)) * D + ld % D);
      }
      g.xd[key] = v;
    }
    hx = h & t.hxmask;
  }
  if (lane == 0) {
    SpinBlockHead hd{};
    if (real) {
      hd.first = __ldg(t.blk_off + blk);
      hd.tile = __ldg(t.tfirst + blk);
      hd.lbase = __ldg(t.looff + k);
      hd.nk = __ldg(t.looff + k + 1) - hd.lbase;
      hd.k = k;
      hd.nhh = n;
      hd.nx = nx;
      hd.hx = hx;
      hd.dg = dg;
    }
    *reinterpret_cast<SpinBlockHead*>(out) = hd;
  }
}

// The programs of bundle ub on their way into dst (every thread; waited for by
// spin_rows_bundle).
template <int NT>
__device__ __forceinline__ void spin_fetch(const SpinDev& t, int64_t ub, unsigned char* dst, size_t bytes) {
  const unsigned char* src = t.rprog + ub * bytes;
  for (size_t i = threadIdx.x * (size_t)16; i < bytes; i += (size_t)NT * 16) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst + i);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src + i) : "memory");
  }
}

// Bundle ub, whose programs are in (or on their way into) prog; the next
// bundle's (next < 0: none) go to other while this one runs.
template <int D, int B, int NT>
__device__ __forceinline__ void spin_rows_bundle(const SpinDev& t, int64_t next, const double* x, double* y,
                                                 double* alpha_part, SpinRowsSmem& sm,
                                                 unsigned char* xs, unsigned char* prog, unsigned char* other,
                                                 size_t pb) {
  constexpr int BITS = D <= 2 ? 1 : D <= 4 ? 2 : 3;
  constexpr uint32_t dm = (1u << BITS) - 1u;
  using Row = SpinRow<B>;
  Row* rows = reinterpret_cast<Row*>(xs);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();  // this bundle's programs are here; the previous one is done with x and other
  if (next >= 0) spin_fetch<NT>(t, next, other, (size_t)B * pb);
  const SpinBlockHead* hd[B];
#pragma unroll
  for (int j = 0; j < B; ++j) hd[j] = reinterpret_cast<const SpinBlockHead*>(prog + j * pb);
  const uint32_t nk = hd[0]->nk, lbase = hd[0]->lbase;
  const int nv = nk == 0u ? 0 : B == 2 && hd[B - 1]->nk != 0u ? 2 : 1;
  uint32_t bj[B];
#pragma unroll
  for (int j = 0; j < B; ++j) bj[j] = hd[j]->first;
  for (uint32_t i = threadIdx.x; i < nk; i += 2 * NT) {  // x of the blocks, row by row
    Row a, b;
    const bool two = i + NT < nk;
#pragma unroll
    for (int j = 0; j < B; ++j) {
      a.v[j] = j < nv ? x[bj[j] + i] : 0.0;
      b.v[j] = j < nv && two ? x[bj[j] + i + NT] : 0.0;
    }
    rows[i] = a;
    if (two) rows[i + NT] = b;
  }
  int nhh[B], nx[B], common = 1 << 20, most = 0;
#pragma unroll
  for (int j = 0; j < B; ++j) {
    nhh[j] = hd[j]->nhh;
    nx[j] = hd[j]->nx;
    common = min(common, nhh[j]);
    most = max(most, nhh[j]);
  }
  common &= ~3;
  const bool same = B == 2 && nv == 2 && hd[0]->hx == hd[B - 1]->hx;
  SpinBlockProg g[B];
#pragma unroll
  for (int j = 0; j < B; ++j) g[j] = spin_block_prog<D>(prog + j * pb, t);
  __syncthreads();
  const uint32_t s0 = (lbase >> 5) + (uint32_t)hd[0]->k;
  const unsigned char* vs = reinterpret_cast<const unsigned char*>(sm.val);
#pragma unroll 1
  for (uint32_t r = threadIdx.x; r < nk; r += NT) {
    const uint32_t u = lbase + r;
    const uint32_t s = s0 + (r >> 5);
    const int np = (int)__ldg(t.low_w + s);
    const uint2* tp = t.low_e + ((size_t)s * t.low_st * 32 + lane);
    uint2 ea{}, eb{};
    if (np > 0) ea = __ldg(tp);
    if (np > 1) eb = __ldg(tp + 32);
    const double ldg = __ldg(t.lodiag + u);
    const Row own = rows[r];
    const double* xr = x + r;
    double acc[B], dg[B];
    if (t.n_key) {
      const uint32_t key = __ldg(t.lokey + u);
#pragma unroll
      for (int j = 0; j < B; ++j) dg[j] = ldg + (j < nv ? g[j].xd[key] : 0.0);
    } else {
      const uint32_t lo = t.n_x ? __ldg(t.lolist + u) : 0u;
#pragma unroll
      for (int j = 0; j < B; ++j) dg[j] = ldg + hd[j]->dg;
#pragma unroll 1
      for (int q = 0; q < t.n_x; ++q) {
        const int ld = (int)((lo >> t.cross[q].lshift) & dm);
#pragma unroll
        for (int j = 0; j < B; ++j) dg[j] += j < nv ? g[j].xd[q * D + ld] : 0.0;
      }
    }
#pragma unroll
    for (int j = 0; j < B; ++j) acc[j] = 0.0;
    // hi-hi terms: four of every block at a time, then two, whichever block has them
#pragma unroll 1
    for (int o = 0; o < common; o += 4) {
      double v[4][B];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int j = 0; j < B; ++j) v[q][j] = xr[g[j].nb[o + q]];
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int j = 0; j < B; ++j) acc[j] = fma(g[j].c[o + q], v[q][j], acc[j]);
    }
#pragma unroll 1
    for (int o = common; o < most; o += 2) {
      double v[2][B];
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int j = 0; j < B; ++j) v[q][j] = o + q < nhh[j] ? xr[g[j].nb[o + q]] : 0.0;
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int j = 0; j < B; ++j)
          if (o + q < nhh[j]) acc[j] = fma(g[j].c[o + q], v[q][j], acc[j]);
    }
    // crossing terms, two at a time; blocks with the same crossing digits share table and elements
    if (same) {
#pragma unroll 1
      for (int o = 0; o < nx[0]; o += 2) {
        const bool two = o + 1 < nx[0];
        const uint2 a = g[0].xop[o], b = two ? g[0].xop[o + 1] : a;
        const uint32_t e = __ldg(t.xtab + a.y + u);
        const uint32_t f = two ? __ldg(t.xtab + b.y + u) : kSpinNone;
        double v[B], w[B];
#pragma unroll
        for (int j = 0; j < B; ++j) {
          v[j] = w[j] = 0.0;
          if (e != kSpinNone) v[j] = x[g[j].xop[o].x + (e & 0xffffffu)];
          if (f != kSpinNone) w[j] = x[g[j].xop[o + 1].x + (f & 0xffffffu)];
        }
        if (e != kSpinNone) {
          const double c = g[0].xc[o * D + (e >> 24)];
#pragma unroll
          for (int j = 0; j < B; ++j) acc[j] = fma(c, v[j], acc[j]);
        }
        if (f != kSpinNone) {
          const double c = g[0].xc[(o + 1) * D + (f >> 24)];
#pragma unroll
          for (int j = 0; j < B; ++j) acc[j] = fma(c, w[j], acc[j]);
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < B; ++j) {
#pragma unroll 1
        for (int o = 0; o < nx[j]; o += 2) {
          const bool two = o + 1 < nx[j];
          const uint2 a = g[j].xop[o];
          const uint2 b = two ? g[j].xop[o + 1] : a;
          const uint32_t e = __ldg(t.xtab + a.y + u);
          const uint32_t f = two ? __ldg(t.xtab + b.y + u) : kSpinNone;
          double v = 0.0, w = 0.0;
          if (e != kSpinNone) v = x[a.x + (e & 0xffffffu)];
          if (f != kSpinNone) w = x[b.x + (f & 0xffffffu)];
          if (e != kSpinNone) acc[j] = fma(g[j].xc[o * D + (e >> 24)], v, acc[j]);
          if (f != kSpinNone) acc[j] = fma(g[j].xc[(o + 1) * D + (f >> 24)], w, acc[j]);
        }
      }
    }
    // lo-lo terms, two pairs of entries ahead
    auto term = [&](uint32_t e) {
      const double c = *reinterpret_cast<const double*>(vs + (e >> 20));
      const Row v = *reinterpret_cast<const Row*>(xs + (B == 2 ? (e & 0xfffffu) : (e & 0xfffffu) >> 1));
#pragma unroll
      for (int j = 0; j < B; ++j) acc[j] = fma(c, v.v[j], acc[j]);
    };
#pragma unroll 1
    for (int q = 0; q < np; q += 2) {
      const uint2 e = ea, f = eb;
      tp += 64;
      if (q + 2 < np) ea = __ldg(tp);
      if (q + 3 < np) eb = __ldg(tp + 32);
      term(e.x);
      term(e.y);
      if (q + 1 < np) {
        term(f.x);
        term(f.y);
      }
    }
#pragma unroll
    for (int j = 0; j < B; ++j)
      if (j < nv) y[bj[j] + r] = fma(dg[j], own.v[j], acc[j]);
  }
  if (!alpha_part) return;
  __syncthreads();  // the bundle's rows of y are written
  constexpr int kTh = 256;  // threads of a tile's partial
  const uint32_t nt = (nk + kSpinTileRows - 1) / kSpinTileRows;
  const int items = nv * (int)nt;
  for (int i0 = 0; i0 < items; i0 += kSpinRedItems) {
    const int i1 = min(items, i0 + kSpinRedItems);
    for (int q = warp; q < (i1 - i0) * (kTh / 32); q += NT / 32) {  // a warp's share of a tile each
      const int it = i0 + q / (kTh / 32), th = q % (kTh / 32) * 32 + lane;
      const int j = it / (int)nt;
      const uint32_t r0 = (uint32_t)(it - j * (int)nt) * kSpinTileRows;
      const uint32_t base = hd[B == 2 ? j : 0]->first;
      double dot = 0.0;
#pragma unroll
      for (int i = 0; i < kSpinTileRows / kTh; ++i) {
        const uint32_t r = r0 + th + i * kTh;
        if (r < nk) dot = fma(rows[r].v[B == 2 ? j : 0], y[base + r], dot);
      }
      for (int o = 16; o > 0; o >>= 1) dot += __shfl_down_sync(0xffffffffu, dot, o);
      if (lane == 0) sm.red[it - i0][th >> 5] = dot;
    }
    __syncthreads();
    for (int it = i0 + warp; it < i1; it += NT / 32) {
      const int j = it / (int)nt;
      const uint32_t first = hd[B == 2 ? j : 0]->tile;
      double r = lane < kTh / 32 ? sm.red[it - i0][lane] : 0.0;
      for (int o = 16; o > 0; o >>= 1) r += __shfl_down_sync(0xffffffffu, r, o);
      if (lane == 0) alpha_part[first + (uint32_t)(it - j * (int)nt)] = r;
    }
    __syncthreads();
  }
}

}  // namespace aed
