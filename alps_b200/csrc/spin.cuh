// spin.cuh -- Sz sectors of spin-S models with S >= 1/2: tables and launch wrappers.
//
// Site i holds digit v_i = m_i + S in [0, 2S] (the index of its state in the
// spin site basis, Sz ascending; lib/xml/models.xml.in:24-36), stored in
// `bits` bits with site 0 most significant, so that integer order of the
// packed states is the basis order of basis_states::build (odometer, last
// site fastest; src/alps/model/basisstates.h:175-278).  The sector is the set
// of states with digit sum T = Sz_total + N S.  Ranks use two tables: the
// packed state splits into a hi part (the first Nh sites) and a lo part (the
// last Nl); rank = thi[hi] + tlo[lo], tlo[lo] the rank of lo among lo codes
// of the same digit sum, thi[hi] the number of sector states with a smaller
// hi code.  The sector's states come in blocks of one hi code each.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "kernels.cuh"

namespace aed {

constexpr int kSpinMaxSites = 32;
constexpr int kSpinMaxDim = 5;                     // 2S + 1 <= 5 (S <= 2)
constexpr int kSpinMaxPairs = kSpinMaxDim * kSpinMaxDim;
constexpr int kSpinMaxTrans = kSpinMaxPairs * kSpinMaxDim;
constexpr int kSpinTileRows = 1024;                // rows per <x, y> partial of the apply

constexpr int kSpinRowVals = 126;  // distinct elements of the rows apply's lo-lo terms

// A bond across the hi and lo words: bit offsets of its digits, its lo site's
// index among those with a crossing table, and per hi digit and its change q
// (bit hd (2 d - 1) + q + d - 1) whether any lo digit has an element.
struct SpinCross {
  int hshift, lshift, tab;
  unsigned long long mask;
};

// Host tables of one sector.
struct SpinTables {
  int N = 0, twoS = 0, d = 0, bits = 0, Nh = 0, Nl = 0, T = 0;
  int64_t D = 0;
  std::vector<uint32_t> thi;      // 2^(bits Nh): states before hi code h (kSpinNone: not a digit string)
  std::vector<uint32_t> tlo;      // 2^(bits Nl): rank of lo among lo codes of its digit sum
  std::vector<uint32_t> lolist;   // valid lo codes grouped by digit sum, ascending
  std::vector<uint32_t> looff;    // offsets into lolist per digit sum (max sum + 2 entries)
  std::vector<uint32_t> blk_hi;   // hi code of every block (ascending = basis order)
  std::vector<uint32_t> blk_off;  // first row of every block
  std::vector<uint32_t> tile_blk, tile_r;  // work tiles: (block, first row within it)
  std::vector<uint32_t> rblk, tfirst;      // the rows apply's block list; first tile of every block
  int maxrows = 0;                         // rows of the largest block
};
constexpr uint32_t kSpinNone = 0xffffffffu;
constexpr int kSpinRowsNone = 1;  // launch_spin_rows: the blocks do not fit, nothing launched
int build_spin_tables(int N, int twoS, int T, SpinTables& t);

struct SpinDev {
  const uint32_t *thi, *tlo, *lolist, *looff, *blk_hi, *blk_off, *tile_blk, *tile_r;
  int64_t D, n_blk, n_tiles;
  int N, bits, Nl, d, T;
  // the lo table of the tabulated form (nullptr: none): per bond with both
  // sites in lo (the j-th such bond, in bond order) and per lo code u (its
  // index in lolist), entry [j n_lo + u] = (r0 | pr << 26, r1): the digit
  // pair pr = a d + c and the ranks within the block (tlo of the target lo
  // code) of the pair's off-diagonal slots 0 and 1, kSpinLoNone where empty
  const uint2* lol;
  int64_t n_lo;
  int n_ll;
  // the rows apply (spin_rows.cuh; rblk == nullptr: none): blocks grouped by lo
  // digit sum, each group padded with kSpinNone to an even number; the first
  // tile of every block; the lo-lo terms in slices of 32 rows (slice
  // (looff[k] >> 5) + k + (r >> 5) of row r of digit sum k; low_w pairs of
  // entries, pair q of lane l at (slice * low_st + q) * 32 + l, an entry 16 x
  // target rank | 8 x element index << 20); the diagonal of every lo code over
  // the lo word; the crossing bonds with their tables: xtab[(tab (2 d - 1) + q +
  // d - 1) n_lo + u] = rank of lo code u with the site's digit lowered by q |
  // digit << 24, xoff / xdiag the elements by bond, hd, (q,) ld
  const uint32_t* rblk = nullptr;
  const uint32_t* tfirst = nullptr;
  const uint2* low_e = nullptr;
  const uint32_t* low_w = nullptr;
  const double* lodiag = nullptr;
  const SpinCross* cross = nullptr;
  const uint32_t* xtab = nullptr;
  const double *xoff = nullptr, *xdiag = nullptr;
  int64_t n_rblk = 0;
  int low_st = 0, maxrows = 0, n_hh = 0, n_x = 0, n_xtab = 0;
  // n_key > 0: key of every lo code over its digits at the sites with a
  // crossing table (d^n_xtab keys); hxmask the hi word's bits of crossing bonds
  const uint8_t* lokey = nullptr;
  const unsigned char* rprog = nullptr;  // the blocks' programs, in list order
  int n_key = 0;
  uint32_t hxmask = 0;
};
constexpr uint32_t kSpinLoNone = (1u << 26) - 1u;

// One transition of a bond's pair of digits (a, c) -> (a2, c2) with the
// element Jz * A + Jxy * B + K * C (A: Sz Sz, B: exchange_xy, C: biquadratic).
struct SpinTrans {
  uint8_t a2, c2;
  double A, B, C;
};

constexpr int kSpinMaxCls = 8;  // coupling classes whose elements are tabulated
constexpr int kSpinMaxOff = kSpinMaxDim - 1;  // off-diagonal transitions of one digit pair (they keep a + c)

struct SpinParams {
  int N, n_bonds, twoS;
  double site_h[kSpinMaxSites], site_d[kSpinMaxSites];
  int s1[kMaxBonds], s2[kMaxBonds];
  double jz[kMaxBonds], jxy[kMaxBonds], kq[kMaxBonds];
  int tstart[kSpinMaxPairs + 1];  // transitions of pair (a, c) = a d + c: [tstart[p], tstart[p+1])
  SpinTrans trans[kSpinMaxTrans];
  // bonds with the same (Jz, Jxy, K) share a class; with at most kSpinMaxCls
  // classes the elements Jz A + Jxy B + K C are tabulated per class and digit
  // pair (a, c) = a d + c (n_cls = 0: formed per bond in the kernel): pdg the
  // diagonal element, pov the off-diagonal elements that are nonzero (zero
  // elements are skipped, hamiltonian_matrix.hpp:316) in target order (a2, c2),
  // each with k = a2 - a = c - c2 in one signed byte of pk (byte s for pov[s],
  // 0 past the last); pmo the most off-diagonal elements of any class and pair
  int n_cls;
  int cls[kMaxBonds];
  int pmo;
  double pdg[kSpinMaxCls][kSpinMaxPairs];
  double pov[kSpinMaxCls][kSpinMaxPairs][kSpinMaxOff];
  uint32_t pk[kSpinMaxCls][kSpinMaxPairs];
  double sdiag[kSpinMaxSites][kSpinMaxDim];  // -h m + D m^2 of every site and digit
};
struct SpinRowVals {
  int n;
  double v[kSpinRowVals];
};
// The local operators of the spin model (models.xml.in:24-36, 282-300): the
// transitions of Sz Sz, exchange_xy and biquadratic for spin S = twoS / 2.
void spin_transitions(int twoS, SpinParams& p);
// Bonds, site terms, coupling classes and their tabulated elements (after
// spin_transitions).
void spin_set_couplings(const std::vector<int>& s1, const std::vector<int>& s2, const std::vector<double>& jz,
                        const std::vector<double>& jxy, const std::vector<double>& kq,
                        const std::vector<double>& site_h, const std::vector<double>& site_d, int N, SpinParams& p);

int launch_spin_basis(const SpinDev& t, uint64_t* out, int64_t offset, int64_t count, cudaStream_t st);
int launch_spin_hv(const SpinParams& p, const SpinDev& t, const double* x, double* y, double* alpha_part,
                   cudaStream_t st);
// Bytes of the lo table for p and t (0: the apply's form uses none), and its
// fill (the table at dst, t.n_lo set); t.n_ll is set by the first call.
size_t spin_lo_table_bytes(const SpinParams& p, SpinDev& t);
int launch_spin_lo_table(const SpinParams& p, const SpinDev& t, uint2* dst, cudaStream_t st);
// The rows apply's block list, ordered for p's bonds: largest blocks first,
// within a digit sum by the digits of the crossing bonds, so that the blocks of
// a bundle share their crossing terms, then by their number of hi-hi terms.
void spin_block_list(const SpinParams& p, SpinTables& t);
// Host plan of the rows apply for p's couplings: false when the form has none
// (untabulated couplings, too many elements, or blocks too large for shared
// memory).  Fills the counts of t and the arrays to upload.
struct SpinRowsPlan {
  std::vector<SpinCross> cross;
  std::vector<double> xoff, xdiag;
  std::vector<int> xsite;  // lo sites with a crossing table
  SpinRowVals vals;
};
bool spin_rows_plan(const SpinParams& p, SpinDev& t, SpinRowsPlan& r);
inline size_t spin_low_slices(const SpinDev& t) { return (size_t)t.n_lo / 32 + (size_t)(t.d - 1) * t.Nl + 2; }
// Fill low_e / low_w / lodiag and the crossing table (device arrays).
int launch_spin_rows_tables(const SpinParams& p, const SpinDev& t, const SpinRowsPlan& r, uint2* low_e,
                            uint32_t* low_w, double* lodiag, uint8_t* lokey, uint32_t* xtab, cudaStream_t st);
size_t spin_prog_bytes(const SpinDev& t);  // of all blocks' programs
int launch_spin_progs(const SpinParams& p, const SpinDev& t, unsigned char* out, cudaStream_t st);
int launch_spin_rows(const SpinParams& p, const SpinDev& t, const SpinRowVals& vals, const double* x, double* y,
                     double* alpha_part, cudaStream_t st);
__host__ __device__ inline int64_t spin_tiles_of(const SpinDev& t) { return t.n_tiles; }

}  // namespace aed
