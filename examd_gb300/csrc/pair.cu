// pair.cu -- the midpoint pair kernel: one CTA per tile of home cells.
//
// Replaces exaMD_forces_midpoint_all / _bdry / _overlap, exaMD_particle_
// interaction and lennardjones_12 (SRC/exaMD_forces.f90:41-551,
// user_func.f90:40-75).  A tile owns every cell pair whose home block -- given
// by the reference's 63-entry table (SRC/exaMD_module.f90:276-346) -- lies in
// the tile; the tile plus a one-cell halo is staged in shared memory with the
// periodic images folded into the staged coordinates (the SMEM counterpart of
// the MPI halo exchange, SRC/exaMD_comms.f90:44-244).
//
// Work order.  The 62 non-self table entries are, per cell A, 12 full x-rows
// of 5 cells (dy, dz fixed, dx = -2..2) plus the half row dx = +1, +2; with
// the pairs inside A that makes 13 "rows" r.  A warp turns (staged atom,
// row) pairs into items: the contiguous j-ranges of the cells of row r that
// the table assigns to this tile (ownership masks per position class),
// trimmed to the cells whose box comes within rc of the atom (the accepted
// pairs are unchanged).  Only rows with a nonzero mask for the atom's class
// are visited, 32 (atom, row) pairs per step whatever the atom; the items
// of one step (at most 32) have their candidate pairs laid end to end and
// tested 32 at a time, one per lane.  Accepted pairs are queued and their
// forces computed in batches of 32, both atoms' sums updated (Newton's third
// law).  The FP64 form's first pass (k_pair_fix) walks the same items, tested
// with an FP32 prefilter on a widened cutoff, and computes the queued pairs in
// fixed point (force_batch_fix).  Its FP64 body (the tiles that the fixed-point
// pass cannot take, and systems it cannot hold) builds items per (ext cell, row): the
// block of the cell's atoms against the row's owned j-cells, untrimmed; its
// batches then hold pairs of many different i atoms, so their FP64
// shared-memory atomics (compare-and-swap loops) rarely hit one address.
//
// What bounds the passes (1M liquid): the enumeration and the FP64 pass issue
// (71-81 % of the slots; ALU pipe 50 %); the list pass issue and shared memory
// (70 %; half of the wavefronts atomics); none of them DRAM (0.1-0.9 TB/s).
//
// Accumulation.  Mixed form: each per-atom force component is an exact 32-bit
// fixed-point sum in shared memory (scale 2^17, native integer atomics), so
// the result does not depend on the order of the terms and is reproducible
// bit for bit.  A term of magnitude >= 2048 (r < 0.74 sigma at eps = 1) is
// left out and flags the tile, so every fixed-point term is below 2^28 and a
// component's sum could leave the int32 range only through more than 8
// near-maximal terms of one sign on one atom, i.e. 8 neighbours within about
// 0.75 sigma on one side, which no physical configuration has (the repulsive
// cores of 8 such neighbours do not fit in one hemisphere).  A second
// launch (k_pair_redo) recomputes the flagged tiles, sums their large terms
// in FP32 and adds them to the outputs; thermal configurations flag no tile
// and the launch returns at once (only the rare FP32 sums' order can vary
// between runs).  FP64 form: integer sums that no number of terms overflows in
// the first pass (common.cuh, FixUnit), FP64 shared-memory atomics in the FP64
// body.
//
// Output: forces of the tile's home atoms go to Fown, those of halo copies to
// the partial slot P[s] (s = bitmask of the axes on which the copy is a halo
// copy); the integrator sums an atom's 1..8 partials in a fixed order.
#include <algorithm>
#include <type_traits>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

// The list build returns before the write-back that the other passes of the
// same tile body run (its instantiation has that code unreachable, by design).
#pragma nv_diag_suppress 128

#include "common.cuh"
#include "kernels.cuh"
#include "pairfn.cuh"

namespace examd {

// In global memory: a CTA's threads read different words of it, which the
// constant bank would serve one after the other.
__device__ OwnLut g_own;

cudaError_t upload_own_lut(const OwnLut& lut) { return cudaMemcpyToSymbol(g_own, &lut, sizeof(OwnLut)); }

constexpr int kDT = 6;        // origin differences for d = -2..3
constexpr int kQueue = 64;    // per-warp queue of accepted pairs
// Work units per 32 staged atoms.  Finer units end a CTA more evenly and set up
// more: 2 in a grid of many waves (1, 3 and 4 measured slower), 4 where the CTAs'
// own time shows (few waves: pair pass of 104k atoms in FP64 129 -> 124 us, 32k
// 46 -> 44, 2,048 18.6 -> 15.1; but 1M 867 -> 873).
constexpr int kUnitParts = 2, kFineParts = 4;
// Warps per CTA of the list build, whatever the other passes use: the build
// needs one count word per atom where they keep three force sums, and in the
// room 12 warps fit 3 CTAs on an SM at the tiles of a dense liquid (36 warps
// against 24 with 8), to hide its shared-memory latency.
constexpr int kBuildWarps = 12;
constexpr int kWideWarps = 12;
// Fixed-point scale 2^17: each term is rounded to 2^-18 in absolute value.
// With the pairs at the cutoff decided in FP64, the mixed form's error on an
// equilibrated 1M-atom liquid was 2.38e-6 RMS of F_rms at 2^16, about 1.6e-6
// of it the sums' rounding (55 terms an atom at F_rms ~ 35) and the rest the
// FP32 separations; 2^17 halves the rounding share.  Every kept term is below
// kFixMaxForce, so below 2^28 in fixed point: a component's int32 sum (exact
// modulo 2^32 whatever the order) leaves the range only through more than 8
// near-maximal terms of one sign on one atom, which no physical
// configuration has.
constexpr float kFix = 131072.f;
constexpr float kFixInv = 1.f / 131072.f;
constexpr int kRedoBlocks = 152;       // grid of the redo pass (1 per SM)
// Passes of the mixed form's tile body: the first pass; the redo pass's two
// kinds of tile, one whose large terms were left out (only those are summed
// and added) and one that overflowed the first pass's capacity (computed in
// full at the redo capacity, large terms in an FP32 side array).  Pair-list
// mode: the list build (the first pass's enumeration at the list cutoff,
// writing the tile's pairs instead of their forces), the forces from the
// list, and the redo of a listed tile's large terms.
// kFixed: the FP64 form's first pass in fixed point (enumerated as the mixed
// form's first pass; tiles with terms too large are computed by the FP64 form's
// own body in the same CTA, tiles over its capacity by the redo pass).
constexpr int kMain = 0, kRedoBig = 1, kRedoFull = 2, kListBuild = 3, kList = 4, kListBig = 5, kFixed = 6;
constexpr int kFullBit = 1 << 30;      // redo-list entry: tile | kFullBit for an overflowed tile
constexpr int kSeg = 4;                // lanes per segment of the i-side force sums
constexpr int kSegFix = 2;             // the same, kFixed (a shuffle of nine words per doubling)
constexpr int kMaxListK = 1024;        // pair-list mode: most list entries of one atom
// Mixed form: a pair whose FP32 r^2 lies within this fraction of rc^2 (a few
// times the FP32 separation's rounding) is accepted or not on its FP64 r^2,
// as the FP64 form decides it, so that no pair straddling the cutoff enters
// one form's sums and not the other's (about 1e-4 of an atom's pairs)
constexpr float kBorder = 4e-6f;
constexpr float kWiden = 1.f + 2.f * kBorder;  // of rc^2: the pairs that the batch of forces looks at

// Shared-memory carve-up, identical on host and device.
struct Layout {
  int lstart, gfirst, ox, oy, oz, dyt, dzt, img, cw, r2l, lut, ljt, queue;
  int pf, fa, px, code, fr;
  int perm, hist;  // pair-list passes: the staged atoms by entry count, and the counts' histogram
  int bytes;
};

// Per-warp tables after the accepted-pair queues.  Mixed form and kFixed: one
// step's items by rank (pt, float4) and the work unit's atoms by rank (bt, two
// float4; kFixed: one, the positions are read again from the staged atoms, which
// makes room for the coarse words of 340 atoms).  FP64 form: one step's items by
// lane (float4).
constexpr int kWarpTab = 32 * 16 + 32 * 32;
constexpr int kWarpTabFix = 32 * 16 + 32 * 16;
constexpr int kWarpTabFp64 = 32 * 16;

__host__ __device__ inline int align16(int x) { return (x + 15) & ~15; }

// mode: kMain, kRedoBig (fr: the large terms' FP32 sums, over the
// accepted-pair queues, which that pass does not use, when they fit there)
// or kRedoFull (fr after everything else); kListBuild (the per-warp tables
// without queues, the count order and its histogram); kList, kListBig (no
// queues, no ownership table: the queue region holds only the scan and
// reduction scratch; kListBig's fr after everything).
// ne_max, ext_max: the largest tile's ext cells and ext extent on one axis.
// own: with a copy of the ownership table (see pair_own_global).
__host__ __device__ inline Layout make_layout(bool fp64, int cap, int ne_max, int ext_max, int nw, int mode,
                                              bool multi, bool own = true) {
  const bool from_list = mode == kList || mode == kListBig;
  Layout L;
  int o = 0;
  L.lstart = o; o = align16(o + 2 * (ne_max + 1));  // < 2^16: at most the capacity
  L.gfirst = o; o = align16(o + 4 * ne_max);
  L.ox = o;     o = align16(o + 4 * (ext_max + 1));
  L.oy = o;     o = align16(o + 4 * (ext_max + 1));
  L.oz = o;     o = align16(o + 4 * (ext_max + 1));
  L.dyt = o;    o = align16(o + 8 * ext_max * kDT);  // float2 (row origin offset, near face, both from row l) per (l, d)
  L.dzt = o;    o = align16(o + 8 * ext_max * kDT);
  const bool fix = mode == kFixed;
  L.img = o;    o = align16(o + (fp64 || fix ? 3 * 32 : 0));  // periodic image per ext coordinate (FP64 form)
  L.cw = o;     o = align16(o + 16);  // unit counter, large-term flag, staged-atom total
  L.r2l = o;    o = align16(o + (fp64 ? 64 * nw : 0));  // rank -> lane tables (FP64 form)
  L.lut = o;    o = align16(o + (from_list || !own ? 0 : (int)sizeof(OwnLut)));
  // the LJ table per ordered type pair (several types): per-lane type indices
  // would serialise on the kernel-parameter bank, shared memory serves them at once
  L.ljt = o;    o = align16(o + (multi ? (fix ? (int)sizeof(FixPair) : (int)sizeof(LJ64)) * EXAMD_MAX_TYPES * EXAMD_MAX_TYPES : 0));
  const int qbytes = (fp64 ? 4 * kQueue + kWarpTabFp64
                           : (from_list ? 64 : fix ? 4 * kQueue + kWarpTabFix : (mode == kListBuild ? 0 : 16) * kQueue + kWarpTab)) *
                     nw;
  L.queue = o;  o = align16(o + qbytes);
  L.pf = o;     o = align16(o + 16 * (from_list ? cap + 1 : cap));  // list passes: + the padding atom
  if (fp64 || fix) {
    L.fa = o;   o = align16(o + 3 * (fix ? 12 : 8) * cap);  // FP64 force sums (kFixed: low, high and coarse words)
    L.px = o;   o = align16(o + 3 * 8 * cap);  // FP64 (kFixed: fixed-point) positions
  } else {
    L.fa = o;   o = align16(o + (mode == kListBuild ? 1 : 3) * 4 * cap);  // fixed-point force sums, x y z per atom (build: counts)
    L.px = o;
  }
  L.code = o;   o = align16(o + 2 * cap);
  L.perm = L.hist = o;
  if (mode == kListBuild) {  // the build orders the atoms by entry count, at its end:
    // in the per-warp tables' region, which the enumeration no longer uses then, if it fits
    if (align16(2 * cap) + 4 * (kMaxListK + 1) <= qbytes) {
      L.perm = L.queue;
      L.hist = L.queue + align16(2 * cap);
    } else {
      L.perm = o; o = align16(o + 2 * cap);
      L.hist = o; o = align16(o + 4 * (kMaxListK + 1));
    }
  }
  L.fr = L.queue;
  if (!fp64 && (mode == kRedoFull || mode == kListBig || (mode == kRedoBig && 3 * 4 * cap > 16 * kQueue * nw))) {
    L.fr = o;   o = align16(o + 3 * 4 * cap);
  }
  L.bytes = o;
  return L;
}

static int redo_smem_bytes(const PairConfig& cfg, int cap_redo, int ne_max, int ext_max) {
  if (cfg.fix) return make_layout(true, cap_redo, ne_max, ext_max, cfg.warps, kRedoFull, cfg.multi).bytes;
  const int b = std::max(make_layout(false, cap_redo, ne_max, ext_max, cfg.warps, kRedoBig, cfg.multi).bytes,
                         make_layout(false, cap_redo, ne_max, ext_max, cfg.warps, kRedoFull, cfg.multi).bytes);
  return cfg.list ? std::max(b, make_layout(false, cap_redo, ne_max, ext_max, cfg.warps, kListBig, cfg.multi).bytes)
                  : b;
}

static bool uses_wide(const PairConfig& c) { return c.wide && !c.fp64 && !c.list && !c.count; }

// The first pass's layout: the enumeration's, or in pair-list mode (without
// counters, which the enumeration gives) the list pass's.
static int main_smem_bytes(const PairConfig& cfg, int cap, int ne_max, int ext_max) {
  const int mode = (cfg.list && !cfg.count && !cfg.fp64) ? kList : kMain;
  if (cfg.fix)  // (and the FP64 body in the same CTA)
    return std::max(make_layout(true, cap, ne_max, ext_max, cfg.warps, kMain, cfg.multi).bytes,
                    make_layout(false, cap, ne_max, ext_max, cfg.warps, kFixed, cfg.multi, !cfg.own_global).bytes);
  if (uses_wide(cfg)) return make_layout(false, cap, ne_max, ext_max, kWideWarps, kMain, cfg.multi).bytes;
  return make_layout(cfg.fp64, cap, ne_max, ext_max, cfg.warps, mode, cfg.multi).bytes;
}

static int build_smem_bytes(const PairConfig& cfg, int cap, int ne_max, int ext_max) {
  return make_layout(false, cap, ne_max, ext_max, kBuildWarps, kListBuild, cfg.multi).bytes;
}

int pair_smem_bytes(const PairConfig& cfg, int cap, int cap_redo, int ne_max, int ext_max) {
  if (cfg.fix) return std::max(main_smem_bytes(cfg, cap, ne_max, ext_max), redo_smem_bytes(cfg, cap_redo, ne_max, ext_max));
  int b = make_layout(cfg.fp64, cap, ne_max, ext_max, cfg.wide ? kWideWarps : cfg.warps, kMain, cfg.multi).bytes;
  if (cfg.fp64) return b;
  b = std::max(b, redo_smem_bytes(cfg, cap_redo, ne_max, ext_max));
  if (cfg.list) b = std::max(b, std::max(main_smem_bytes(cfg, cap, ne_max, ext_max),
                                         build_smem_bytes(cfg, cap, ne_max, ext_max)));
  return b;
}

int pair_ctas(const PairConfig& cfg, int cap, int ne_max, int ext_max, int sm_smem) {
  constexpr int kReserved = 1024;  // of every CTA, by the system
  const int regs = 32 * cfg.warps * (cfg.multi ? 80 : 64);
  return std::min(sm_smem / (main_smem_bytes(cfg, cap, ne_max, ext_max) + kReserved), 65536 / regs);
}

// The FP64 form's first pass with one type reads the ownership table from global
// memory (its lines stay in L1) where a copy of 3.4 KB in each CTA would cost one
// of the SM's CTAs: at 78 bytes an atom an SM holds four of 528 atoms with the
// copy and of 572 without (8 warps, 4^3 cells; 1M liquid, 568: 951 -> 846 us a
// pass; 87,808 atoms, 536: 100 -> 92).  Elsewhere the copy is nearer (1,000 atoms 9.5
// against 10 us, a 512-box ensemble 1 %); with several types the registers allow
// three either way.
bool pair_own_global(PairConfig cfg, int cap, int ne_max, int ext_max, int sm_smem) {
  if (!cfg.fix || cfg.multi) return false;
  cfg.own_global = false;
  const int n = pair_ctas(cfg, cap, ne_max, ext_max, sm_smem);
  cfg.own_global = true;
  return pair_ctas(cfg, cap, ne_max, ext_max, sm_smem) > n;
}

// Exact sum of FP32 terms in 64-bit fixed point (2^-32 resolution): the total
// does not depend on the order of the terms.  A term of magnitude >= 30000
// (a pair closer than ~0.46 sigma) goes to an FP32 side sum.
// Below 8192 the term is split at 2^-9 and rounded at 2^-32 by adding constants
// whose ulp is that bit and taking the difference of the sums' bits (the same
// value as the conversions', which run at an eighth of the FP32 rate and were
// six of a pair's nine).
struct FixSum {
  long long v = 0;
  float side = 0.f;
  __device__ __forceinline__ void add(float x) {
    if (fabsf(x) < 8192.f) {
      constexpr float kHi = 24576.f, kLo = 1.5f / 512.f;  // 1.5 2^14 (ulp 2^-9), 1.5 2^-9 (ulp 2^-32)
      const float hi = __fadd_rn(x, kHi);
      const float lo = __fadd_rn(__fsub_rn(x, __fsub_rn(hi, kHi)), kLo);  // (inner differences exact, at most 2^-10)
      v += (long long)(__float_as_int(hi) - 0x46c00000) * (1 << 23) + (__float_as_int(lo) - 0x3b400000);
    } else if (fabsf(x) < 30000.f) {
      const float hs = x * 65536.f;  // exact power-of-two scaling
      const int h = __float2int_rz(hs);
      const int l = __float2int_rn((hs - (float)h) * 65536.f);  // hs - h is exact
      v += ((long long)h << 16) + l;
    } else {
      side += x;
    }
  }
};

// The force of one accepted pair per lane (act), from registers: d = x_j -
// x_i with d.w = r^2, P the type pair's parameters; i = -1 on a lane outside
// the batch, which also ends any run of equal i.  Lanes that hold a pair
// that was not accepted keep their i, add nothing, and do not break the run.
template <bool ENERGY, bool COUNT, bool SIDE, class FA, class FR>
__device__ __forceinline__ void pair_force32(bool act, int i, int m, float4 d, const LJ32& P, FA& fa, FR& fr,
                                             int cap, const PairArgs& A, FixSum& ek, FixSum& wk, int& nacc,
                                             int* big_flag) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  float fx = 0.f, fy = 0.f, fz = 0.f;
  bool big = false;
  if (act) {
    big = d.w < P.r2big;  // left to the redo pass
    float dg = 0.f, e = 0.f;
    const int rv = pair_fn32<ENERGY>(A.lj.pot, d.w, P, dg, e);
    if (rv == 0) {
      const float dgs = kFix * dg;
      fx = dgs * d.x;
      fy = dgs * d.y;
      fz = dgs * d.z;
      if (ENERGY) {
        ek.add(e);
        wk.add(-dg * d.w);
      }
      if (COUNT) ++nacc;
    } else if (rv < 0) {
      atomicOr(A.status, ST_PAIRFN);
    }
  }
  int ix = 0, iy = 0, iz = 0;
  if (act && !big) {
    ix = __float2int_rn(fx);
    iy = __float2int_rn(fy);
    iz = __float2int_rn(fz);
    atomicAdd(&fa[3 * m], -ix);
    atomicAdd(&fa[3 * m + 1], -iy);
    atomicAdd(&fa[3 * m + 2], -iz);
  }
  if (big) {
    if (SIDE) {
      atomicAdd(&fr[i], fx * kFixInv);
      atomicAdd(&fr[cap + i], fy * kFixInv);
      atomicAdd(&fr[2 * cap + i], fz * kFixInv);
      atomicAdd(&fr[m], -fx * kFixInv);
      atomicAdd(&fr[cap + m], -fy * kFixInv);
      atomicAdd(&fr[2 * cap + m], -fz * kFixInv);
    } else {
      *big_flag = 1;
    }
  }
  // i side: sum over runs of equal i (lanes outside the batch form one run
  // with i = -1), in segments of kSeg lanes from the run's first one: each
  // segment's last lane adds the segment's total (4: measured against 2, 8
  // and 16)
  const int ip = __shfl_up_sync(FULL, i, 1);
  const unsigned hb = __ballot_sync(FULL, lane == 0 || ip != i);
  const int dist = (lane - (31 - __clz(hb & (FULL >> (31 - lane))))) & (kSeg - 1);
#pragma unroll
  for (int o = 1; o < kSeg; o <<= 1) {
    const int yx = __shfl_up_sync(FULL, ix, o), yy = __shfl_up_sync(FULL, iy, o), yz = __shfl_up_sync(FULL, iz, o);
    if (o <= dist) {
      ix += yx;
      iy += yy;
      iz += yz;
    }
  }
  const bool tail = lane == 31 || dist == kSeg - 1 || ((hb >> (lane + 1)) & 1u);
  if (i >= 0 && tail && (ix | iy | iz) != 0) {
    atomicAdd(&fa[3 * i], ix);
    atomicAdd(&fa[3 * i + 1], iy);
    atomicAdd(&fa[3 * i + 2], iz);
  }
}

// Forces of cnt queued accepted pairs, one per lane: entry = (d = x_j - x_i,
// key) with key = i | type_i << 14 | j << 16 | type_j << 30; r^2 is recomputed
// with the distance test's expression, so it has the same bits.  user_func.f90:58-69
// in FP32: dg = -24 eps (2 s^12 - s^6) / r^2, f_i += dg d, f_j -= dg d.
// The queue keeps an atom's accepted pairs next to each other, so the i-side
// fixed-point terms are first summed over segments of each run of lanes with
// the same i (a segmented shuffle scan; integer sums, so the result is exact)
// and each segment's last lane adds its total: one shared atomic per segment
// instead of one per pair on the same address.
// A pair-force term too large for the fixed-point sums (|F| >= kFixMaxForce,
// decided on r^2 < r2big of the type pair: r < ~0.74 sigma at eps = 1, which
// thermal configurations do not reach) is left out here and raises the
// tile's flag (*big_flag); the redo pass adds it.  SIDE (the full redo pass):
// such terms go to the FP32 side sums fr instead.
template <bool MULTI, bool ENERGY, bool COUNT, bool SIDE, class QD, class FA, class FR, class IN64>
__device__ __forceinline__ void force_batch(int cnt, int q0, const QD& qd, FA& fa, FR& fr, int cap, const PairArgs& A,
                                            const LJ32* ljs, FixSum& ek, FixSum& wk, int& nacc, int* big_flag,
                                            const IN64& in64) {
  const int lane = threadIdx.x & 31;
  bool act = lane < cnt;
  int i = -1, m = 0;
  float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
  LJ32 P = A.lj.p32[0];
  if (act) {
    d = qd[q0 + lane];
    const unsigned key = __float_as_uint(d.w);
    d.w = fmaf(d.x, d.x, fmaf(d.y, d.y, d.z * d.z));  // r^2 exactly as the distance test computed it
    i = key & 0x3fff;
    m = (key >> 16) & 0x3fff;
    const int ti = MULTI ? (key >> 14) & 3 : 0, tj = MULTI ? key >> 30 : 0;
    if (MULTI) P = ljs[ti * A.lj.nt + tj];
    // the queue also holds the pairs just beyond the cutoff: at the border (kBorder) the FP64 test decides
    act = d.w <= P.rc2;
    if (fabsf(d.w - P.rc2) <= kBorder * P.rc2) act = in64(i, m, ti, tj);
  }
  pair_force32<ENERGY, COUNT, SIDE>(act, i, m, d, P, fa, fr, cap, A, ek, wk, nacc, big_flag);
}

// FP64 form: the reference's arithmetic for cnt queued pairs that passed the
// FP32 prefilter, one per lane (key as in force_batch).  The separation is
// x_j - x_i plus the difference of the two staged copies' periodic images,
// (n_j - n_i) L, which is exact (Sterbenz) and equals the reference's
// dx - Nint(dx/L) L (SRC/exaMD_forces.f90:509-523); then user_func.f90:52-69.
template <bool MULTI, bool ENERGY, bool COUNT, class QK, class PD, class CODE, class IMG, class FD>
__device__ __forceinline__ void force_batch64(int cnt, const QK& qk, const PD& pd, const CODE& code, const IMG& img,
                                              const double* Lbox, FD& fd, int cap, const LJTable& lj,
                                              const LJ64* ljs, double& esum, double& wsum, int* status, int& nacc,
                                              int q0) {
  const int lane = threadIdx.x & 31;
  if (lane >= cnt) return;
  const unsigned key = (unsigned)qk[q0 + lane];
  const int i = key & 0x3fff, m = (key >> 16) & 0x3fff;
  const int ci = code[i], cm = code[m];
  // difference of the copies' periodic images per axis: -1, 0 or +1 box
  const int nx = img[cm & 31] - img[ci & 31];
  const int ny = img[32 + ((cm >> 5) & 31)] - img[32 + ((ci >> 5) & 31)];
  const int nz = img[64 + (cm >> 10)] - img[64 + (ci >> 10)];
  double dx = __dsub_rn(pd[m], pd[i]);
  double dy = __dsub_rn(pd[cap + m], pd[cap + i]);
  double dz = __dsub_rn(pd[2 * cap + m], pd[2 * cap + i]);
  if (nx) dx = __dadd_rn(dx, nx > 0 ? Lbox[0] : -Lbox[0]);
  if (ny) dy = __dadd_rn(dy, ny > 0 ? Lbox[1] : -Lbox[1]);
  if (nz) dz = __dadd_rn(dz, nz > 0 ? Lbox[2] : -Lbox[2]);
  const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
  LJ64 P = lj.p64[0];
  if (MULTI) P = ljs[((key >> 14) & 3) * lj.nt + (key >> 30)];
  double dg = 0.0, e = 0.0;
  const int rv = pair_fn64<ENERGY>(lj.pot, d2, P, dg, e);
  if (rv == 0) {
    const double fx = __dmul_rn(dg, dx), fy = __dmul_rn(dg, dy), fz = __dmul_rn(dg, dz);
    atomicAdd(&fd[i], fx);
    atomicAdd(&fd[cap + i], fy);
    atomicAdd(&fd[2 * cap + i], fz);
    atomicAdd(&fd[m], -fx);
    atomicAdd(&fd[cap + m], -fy);
    atomicAdd(&fd[2 * cap + m], -fz);
    if (ENERGY) {
      esum += e;
      wsum += -__dmul_rn(dg, d2);
    }
    if (COUNT) ++nacc;
  } else if (rv < 0) {
    atomicOr(status, ST_PAIRFN);
  }
}

// FP64 form, fixed-point first pass: the forces of cnt queued pairs that
// passed the FP32 prefilter, one per lane (key as in force_batch).
//
// GB300 runs FP64 arithmetic at 1/64 of the FP32 rate (1.6-2.0 per clock per
// SM), a correctly rounded FP64 reciprocal at the price of about six
// operations, and FP64 shared-memory atomics as compare-and-swap loops that
// add on the same pipe.  With the reference's operations and six such atomics
// a pair cost 35 FP64 operations and more, and the pass was bound by that
// pipe (79 % busy, issue 17 %).  Here the pair keeps eight:
// - positions are integers in units of 2^ue (modulo 2^64, rc < 2^62), so the
//   separation is exact, and D = r^2 / 2^64 to less than one unit by 32-bit
//   multiplies (of the lowest product, below one unit, only the mean is taken):
//   2^55 units or more at r > 0.74 sigma and rc = 2.5 sigma, 3 2^51 at least
//   (build_fix);
// - D becomes a double (one rounding), y = 1/D from an FP32 estimate (relative
//   error e of 2^-22) by one step of Householder's third-order iteration,
//   y (1 + e + e^2), error e^3: three operations;
// - the LJ force per unit distance is y^4 (c6 - c12 y^3), five operations; its
//   53 bits, as an integer, multiply the separation in 32-bit pieces, and the
//   product is taken at the bit that the factor's exponent gives, rounded at the
//   sums' unit 2^-sf (common.cuh, FixUnit);
// - the sums are integers in shared memory with native 32-bit atomics: two words
//   modulo 2^64 (the low one with carry into the high one) and a coarse one:
//   exact, in any order, whatever the number of terms.
// An isolated pair's force is then off by less than the FP64 body's, RMS (1e-16:
// r 0.9-1.1 sigma 9.0 against 11.5; 2.0-2.5 2.9 / 3.6; at rc 4.6 3.4 / 3.7; a pair of
// a sixteenth of the strongest eps 3.1 / 3.6), and the forces do not depend on
// the order.  Where the reference itself rounds coarsely, its rounding is kept: a
// pair across the periodic face is first subtracted at box scale (x_j - x_i,
// rounded to 53 bits of about L, then L added exactly), which moves its
// separation by up to ulp(L) / 2; `face` gives that rounded separation.
// A pair within a unit of D's high word (a few 1e-9) of its range is decided on
// the FP64 body's own r^2 (in64), so that both accept the same pairs; a pair
// whose force is too large for the sums' range flags the tile, and the FP64
// body computes it.
template <bool MULTI, bool ENERGY, bool COUNT, class QK, class PX, class FA, class FACE, class IN64>
__device__ __forceinline__ void force_batch_fix(int cnt, int q0, const QK& qk, const PX& px, FA& fa, int cap,
                                                const PairArgs& A, const FixPair* ljx, double& esum, double& wsum,
                                                int& nacc, int* big_flag, bool edge, const FACE& face,
                                                const IN64& in64) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int i = -1, m = 0;
  long long fx = 0, fy = 0, fz = 0;  // the force on i, in units of 2^-sf modulo 2^64,
  int cx = 0, cy = 0, cz = 0;        // and in coarse steps
  bool app = false;
  if (lane < cnt) {
    const unsigned key = (unsigned)qk[q0 + lane];
    i = key & 0x3fff;
    m = (key >> 16) & 0x3fff;
    const int ti = MULTI ? (key >> 14) & 3 : 0, tj = MULTI ? key >> 30 : 0;
    const FixPair P = MULTI ? ljx[ti * A.lj.nt + tj] : A.fx.p[0];
    long long dx = (long long)(px[m] - px[i]);
    long long dy = (long long)(px[cap + m] - px[cap + i]);
    long long dz = (long long)(px[2 * cap + m] - px[2 * cap + i]);
    if (edge) face(i, m, dx, dy, dz);  // the tile holds periodic copies
    // d = h 2^32 + l with signed l: r^2 / 2^64 = sum h^2 + 2^-31 sum h l + sum l^2 / 2^64, the third term (below one)
    // at its mean, a quarter.  The shift rounds down, by half a unit on average, which the conversion to a double,
    // halves up, makes good
    const int hx = (int)((dx + 0x80000000ll) >> 32), lx = (int)dx;
    const int hy = (int)((dy + 0x80000000ll) >> 32), ly = (int)dy;
    const int hz = (int)((dz + 0x80000000ll) >> 32), lz = (int)dz;
    const long long D = (long long)hx * hx + (long long)hy * hy + (long long)hz * hz +
                        ((0x20000000ll + (long long)hx * lx + (long long)hy * ly + (long long)hz * lz) >> 31);
    const int Dh = (int)(D >> 32);
    app = Dh < P.limh;
    if (abs(Dh - P.limh) <= 1) app = in64(i, m, ti, tj);
    if (app && Dh < P.bigh) {
      app = false;
      *big_flag = 1;
    }
    if (app) {
      // D as a double: normalised so that its first bit is bit 62, 53 bits kept
      const int s = __clz(Dh) - 1;
      const unsigned long long N = ((unsigned long long)D << s) + 512ull;  // (a carry moves into the exponent)
      const double Dd = __longlong_as_double((long long)((N >> 10) + ((unsigned long long)(1084 - s) << 52)));
      // 1/D: the reciprocal of the mantissa in FP32, its exponent put back
      const float mf = __uint_as_float(((unsigned)(N >> 32) >> 7) + 0x3f000000u);
      const unsigned rb = __float_as_uint(rcp_approx(mf));
      const double y0 = __hiloint2double((int)((rb >> 3) + ((unsigned)(834 + s) << 20)), (int)(rb << 29));
      double e = fma(-Dd, y0, 1.0);
      e = fma(e, e, e);
      const double y = fma(y0, e, y0);
      const double y2 = y * y;
      const double y3 = y2 * y;
      const double g = (y2 * y2) * fma(-P.c12, y3, P.c6);
      if (ENERGY) {
        // differences per pair, as the FP64 body forms them (sums of the terms apart cancel at the end), in four
        // operations: 4 eps (s^6 - 1) s^6, and -g r^2 in the tables' units
        const double q6 = P.s6 * y3;
        esum = fma(fma(P.e4, q6, -P.e4), q6, esum);
        if (A.lj.pot != EXAMD_POT_LJ) esum -= P.eshift;
        wsum = fma(-g, Dd, wsum);
      }
      if (COUNT) ++nacc;
      // g = G 2^(e - 1084) with its 53 bits at the top of 62 (|g| < 2^62), then G d / 2^K, rounded; where
      // K would pass 63, G gives up its last bits (the first nine are zeros)
      const int gb = __double2hiint(g);
      const unsigned long long gm =
          ((((unsigned long long)(unsigned)((gb & 0xfffff) | 0x100000)) << 32) | (unsigned)__double2loint(g)) << 9;
      const int Kg = A.fx.k0 + 1084 - ((gb >> 20) & 0x7ff), K = min(Kg, 63);
      long long G = (long long)(gm >> min(Kg - K, 63));
      if (gb < 0) G = -G;
      const int gh = (int)((G + 0x80000000ll) >> 32), gl = (int)G;
      const int ka = 64 - K, kb = K - 32;
      const int half = 1 << (kb - 1);
      // (the coarse part from the product's top 32 bits, a step of which is 2^kc, 16 or more)
      const int kc = K + A.fx.coarse - 96, halfc = 1 << (kc - 1);
      auto term = [&](int h, int l, int& c) {
        const long long hi = (long long)gh * h;
        c = ((int)(hi >> 32) + halfc) >> kc;
        const long long mid = (long long)gh * l + ((long long)gl * h + ((long long)__mulhi(gl, l) + half));
        const unsigned h0 = (unsigned)hi, h1 = (unsigned)((unsigned long long)hi >> 32);
        const unsigned m0 = (unsigned)mid, m1 = (unsigned)((unsigned long long)mid >> 32);
        const unsigned long long a = ((unsigned long long)__funnelshift_l(h0, h1, ka) << 32) | (h0 << ka);
        const unsigned long long b =
            ((unsigned long long)(unsigned)((int)m1 >> kb) << 32) | __funnelshift_r(m0, m1, kb);
        return (long long)(a + b);
      };
      fx = term(hx, lx, cx);
      fy = term(hy, ly, cy);
      fz = term(hz, lz, cz);
    }
  }
  // v and its coarse part vc to the sum of component c of atom t: low word, carry, high word; coarse word
  auto add = [&](int t, int c, long long v, int vc) {
    const unsigned lo = (unsigned)v;
    const unsigned old = atomicAdd((unsigned*)&fa[c * cap + t], lo);
    atomicAdd(&fa[(6 + c) * cap + t], vc);
    atomicAdd(&fa[(3 + c) * cap + t], (int)(v >> 32) + (old + lo < lo ? 1 : 0));
  };
  if (app) {
    add(m, 0, -fx, -cx);
    add(m, 1, -fy, -cy);
    add(m, 2, -fz, -cz);
  }
  // i side: runs of equal i in segments of kSegFix lanes, as in pair_force32
  const int ip = __shfl_up_sync(FULL, i, 1);
  const unsigned hb = __ballot_sync(FULL, lane == 0 || ip != i);
  const int dist = (lane - (31 - __clz(hb & (FULL >> (31 - lane))))) & (kSegFix - 1);
#pragma unroll
  for (int o = 1; o < kSegFix; o <<= 1) {
    const long long yx = __shfl_up_sync(FULL, fx, o), yy = __shfl_up_sync(FULL, fy, o),
                    yz = __shfl_up_sync(FULL, fz, o);
    const int zx = __shfl_up_sync(FULL, cx, o), zy = __shfl_up_sync(FULL, cy, o), zz = __shfl_up_sync(FULL, cz, o);
    if (o <= dist) {
      fx += yx;
      fy += yy;
      fz += yz;
      cx += zx;
      cy += zy;
      cz += zz;
    }
  }
  const bool tail = lane == 31 || dist == kSegFix - 1 || ((hb >> (lane + 1)) & 1u);
  if (i >= 0 && tail) {
    add(i, 0, fx, cx);
    add(i, 1, fy, cy);
    add(i, 2, fz, cz);
  }
}

// One tile.  MODE (mixed form; the FP64 form has only kMain):
// - kMain: the first pass, at capacity A.cap; a tile with more staged atoms
//   is listed for a full redo, one with a large term for a large-term redo;
// - kRedoBig (without energy or counters): recomputes the tile's pairs, sums
//   only the large terms (FP32 shared atomics) and adds them to the outputs
//   that the first pass wrote;
// - kRedoFull: the whole tile at capacity A.cap_redo, large terms in FP32
//   side sums, outputs, energy and counters written as the first pass would.
// Pair-list mode:
// - kListBuild: the first pass's enumeration at the list cutoff (rl2, with
//   prune2_list), which writes the tile's accepted pairs as staged-index
//   entries to its list instead of computing them; a tile over capacity or
//   with more pairs than its list holds goes to the fallback list;
// - kList: the tile's forces from its list, with the same per-pair FP32
//   expressions as the first pass (the same bits when the atoms are where
//   the list was built), outputs, energy and the large-term flag as there;
// - kListBig: kRedoBig from the list.
// kFixed: returns true, nothing written, for a tile with a term too large.
// CUT (list pass): the potential's own range rcut2 is tested (WCA; infinite otherwise).
// kOwnGlobal: the ownership table in global memory.
template <bool FP64, bool MULTI, bool ENERGY, bool COUNT, int MODE, bool CUT = true, int kParts = kUnitParts,
          bool kOwnGlobal = false>
__device__ __forceinline__ bool pair_tile(const PairArgs& A, const int tile) {
  extern __shared__ __align__(16) unsigned char smem[];
  const unsigned FULL = 0xffffffffu;
  // ownership table, type table and axis tables come first: they are fixed for the context
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  const int4 t0 = A.tiles[2 * tile], t1 = A.tiles[2 * tile + 1];
  const BoxDev& B = A.boxes[t0.x];
  const int X0 = t0.y, Y0 = t0.z, Z0 = t0.w;
  const int tx = t1.x, ty = t1.y, tz = t1.z;
  const int EX = tx + 2, EY = ty + 2, EZ = tz + 2;
  const int NE = EX * EY * EZ;
  constexpr bool kFromList = MODE == kList || MODE == kListBig;
  if (MODE == kMain || MODE == kFixed) grid_trigger();
  if (kFromList && MODE == kList && A.lcount[tile] < 0) return false;  // a fallback tile: the redo pass computes it
  constexpr bool FIX = MODE == kFixed;
  const int cap = (MODE == kMain || MODE == kListBuild || MODE == kList || FIX) ? A.cap : A.cap_redo;
  const Layout L = make_layout(FP64, cap, A.ne_max, A.ext_max, nw, MODE, MULTI, !kOwnGlobal);
  // shared-memory arrays (index-checked in the checked build)
  int* const st = A.status;  // the index checks' status word (checked build)
  (void)st;
  auto lstart = EXAMD_ARR(unsigned short, smem + L.lstart, A.ne_max + 1, st);
  auto gfirst = EXAMD_ARR(int, smem + L.gfirst, A.ne_max, st);
  auto ox = EXAMD_ARR(float, smem + L.ox, A.ext_max + 1, st);
  auto oy = EXAMD_ARR(float, smem + L.oy, A.ext_max + 1, st);
  auto oz = EXAMD_ARR(float, smem + L.oz, A.ext_max + 1, st);
  auto dyt = EXAMD_ARR(float2, smem + L.dyt, A.ext_max * kDT, st);
  auto dzt = EXAMD_ARR(float2, smem + L.dzt, A.ext_max * kDT, st);
  auto img = EXAMD_ARR(signed char, smem + L.img, FP64 || FIX ? 96 : 1, st);
  double* red = (double*)(smem + L.queue);  // scan and reduction scratch, before and after the queues' use
  int* cw = (int*)(smem + L.cw);
  OwnLut* sown = (OwnLut*)(smem + L.lut);
  auto own_nrow = [&](int c) -> int { return kOwnGlobal ? __ldg(&g_own.nrow[c]) : sown->nrow[c]; };
  auto own_ent = [&](int c, int k) -> unsigned { return kOwnGlobal ? __ldg(&g_own.ent[c][k]) : sown->ent[c][k]; };
  LJ32* ljs32 = (LJ32*)(smem + L.ljt);
  LJ64* ljs64 = (LJ64*)(smem + L.ljt);
  FixPair* ljx = (FixPair*)(smem + L.ljt);
  auto pf = EXAMD_ARR(float4, smem + L.pf, kFromList ? cap + 1 : cap, st);
  auto code = EXAMD_ARR(unsigned short, smem + L.code, cap, st);
  auto U = EXAMD_ARR(const float4, A.U, A.N, st);

  {
    const uint4* src = reinterpret_cast<const uint4*>(&g_own);
    uint4* dst = reinterpret_cast<uint4*>(sown);
    if (!kFromList && !kOwnGlobal)
      for (int k = tid; k < (int)(sizeof(OwnLut) / 16); k += blockDim.x) dst[k] = src[k];
    if (MULTI)
      for (int k = tid; k < A.lj.nt * A.lj.nt; k += blockDim.x) {
        if (FIX)
          ljx[k] = A.fx.p[k];
        else if (FP64)
          ljs64[k] = A.lj.p64[k];
        else
          ljs32[k] = A.lj.p32[k];
        if (MODE == kList) ljs32[k].m24eps *= kFix;  // (a power of two: the same bits)
      }
  }
  // Per-axis tables.  Ext coordinate l (cell X0 + l - 1, l = 0..E; l = E is
  // the far edge of the last ext cell) has origin (g0 + l - 1)*bl + n*r, with
  // n = -1, 0, +1 its periodic image and r = L - nb*bl the extra width of the
  // box's last cell.  o*[l]: origin relative to the tile centre, FP32 (the
  // multiple of bl is exact, so the value is rounded once).  d*t[l*6 + d + 2]
  // (y, z): the origin difference between ext rows l and l + d (d = -2..3),
  // rounded once, and the same for l + d + (d < 0), the near face of row l + d
  // seen from row l.  img[32a + l] (FP64 form): n.
  {
    const int a = tid >> 5, l = tid & 31;
    if (a < 3) {
      const int E = a == 0 ? EX : (a == 1 ? EY : EZ);
      const int g0 = a == 0 ? X0 : (a == 1 ? Y0 : Z0);
      const int t = a == 0 ? tx : (a == 1 ? ty : tz);
      const int nb = B.nb[a];
      const float blf = B.blf, rf = B.remf[a];
      auto nimg = [&](int ll) {
        const int g = g0 + ll - 1;
        return g < 0 ? -1 : (g >= nb ? 1 : 0);
      };
      if (l <= E) {
        const int n = nimg(l);
        (a == 0 ? ox : (a == 1 ? oy : oz))[l] = fmaf((float)(2 * (l - 1) - t), 0.5f * blf, (float)n * rf);
        if (l < E) {
          if (FP64 || FIX) img[32 * a + l] = (signed char)n;
          if (a > 0) {
            auto dt = a == 1 ? dyt : dzt;
#pragma unroll
            for (int d = -2; d <= 3; ++d) {
              const int l2 = l + d, ln = l + d + (d < 0);
              const float off = (l2 >= 0 && l2 <= E) ? fmaf((float)(nimg(l2) - n), rf, (float)d * blf) : 0.f;
              const float near = d == 0 ? -1e30f  // the atom's own row: no gap
                                 : (ln >= 0 && ln <= E) ? fmaf((float)(nimg(ln) - n), rf, (float)(d + (d < 0)) * blf)
                                                        : 0.f;
              dt[l * kDT + d + 2] = make_float2(off, near);
            }
          }
        }
      }
    }
  }
  // (1) ext cells: global cell, count, first atom
  grid_wait();  // what came before this line depends on no earlier kernel
  int cc0 = 0;  // the code of cell tid
  for (int e = tid; e < NE; e += blockDim.x) {
    int lx = e % EX, rr = e / EX, ly = rr % EY, lz = rr / EY;
    if (e == tid) cc0 = lx | (ly << 5) | (lz << 10);
    int gx = X0 + lx - 1, gy = Y0 + ly - 1, gz = Z0 + lz - 1;
    gx += (gx < 0) ? B.nb[0] : 0;
    gx -= (gx >= B.nb[0]) ? B.nb[0] : 0;
    gy += (gy < 0) ? B.nb[1] : 0;
    gy -= (gy >= B.nb[1]) ? B.nb[1] : 0;
    gz += (gz < 0) ? B.nb[2] : 0;
    gz -= (gz >= B.nb[2]) ? B.nb[2] : 0;
    int gc = B.cell0 + gx + B.nb[0] * (gy + B.nb[1] * gz);
    int s0 = A.cstart[gc];
    gfirst[e] = s0;
    lstart[e] = (unsigned short)min(A.cstart[gc + 1] - s0, 0xffff);  // a larger count overflows any capacity
  }
  __syncthreads();

  // (2) exclusive scan of the ext-cell counts
  {
    const int per = (NE + blockDim.x - 1) / blockDim.x;
    const int b = tid * per, e = min(b + per, NE);
    int s = 0;
    for (int k = b; k < e; ++k) s += lstart[k];
    int x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(FULL, x, o);
      if (lane >= o) x += y;
    }
    int* wsum = (int*)red;
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    int base = 0;
    for (int w = 0; w < warp; ++w) base += wsum[w];
    int run = base + x - s;
    for (int k = b; k < e; ++k) {
      int c = lstart[k];
      lstart[k] = run;
      // the cell of each staged atom, for the staging and the write-back
      int ck = cc0;
      if (k != tid) {
        const int lx = k % EX, rr = k / EX, ly = rr % EY, lz = rr / EY;
        ck = lx | (ly << 5) | (lz << 10);
      }
      const unsigned short cc = (unsigned short)ck;
      for (int t = run, t1 = min(run + c, cap); t < t1; ++t) code[t] = cc;
      run += c;
    }
    if (tid == blockDim.x - 1) {
      lstart[NE] = (unsigned short)run;
      cw[2] = run;
    }
    __syncthreads();
  }
  const int total = cw[2];
  if (kFromList && A.lcount[tile] != total) {  // the lists of another binning: not computed from
    if (tid == 0) atomicOr(A.status, ST_BOUNDS);
    return false;
  }
  if (kFromList && !(A.lj.pot == EXAMD_POT_LJ || A.lj.pot == EXAMD_POT_LJ_SHIFTED || A.lj.pot == EXAMD_POT_WCA)) {
    if (tid == 0) atomicOr(A.status, ST_PAIRFN);  // a potential the list passes do not evaluate
    return false;
  }
  if (MODE == kListBuild && (total > cap || total > A.lslots)) {  // no list: the redo pass enumerates it every step
    if (tid == 0) {
      A.lcount[tile] = -1;
      A.fb[atomicAdd(&A.lw[LW_FBN], 1)] = tile;
    }
    return false;
  }
  if ((FIX || (!FP64 && MODE == kMain)) && total > cap) {  // the redo pass computes it at its capacity
    if (tid == 0) A.redo[atomicAdd(A.redo_n, 1)] = tile | kFullBit;
    return false;
  }
  if (total > cap) {
    if (tid == 0) {
      atomicOr(A.status, ST_OVERFLOW);
      if (ENERGY) {
        A.tileE[tile] = 0.0;
        A.tileW[tile] = 0.0;
      }
      if (COUNT) {
        A.tileC[3 * tile] = 0;
        A.tileC[3 * tile + 1] = 0;
        A.tileC[3 * tile + 2] = 0;
      }
    }
    return false;
  }
  // (3) stage atoms, one thread per atom, kStage atoms' reads in flight at a
  // time.  (One thread per ext cell, the cell's atoms one after the other, waited
  // for a read per atom: a third of the lanes idle and 188 us of the FP64 form's
  // 950 us on a 1M-atom liquid went into staging and write-back.)
  auto fa = EXAMD_ARR(int, smem + L.fa, (MODE == kListBuild ? 1 : FIX ? 9 : 3) * cap, st);
  auto fr = EXAMD_ARR(float, smem + L.fr, 3 * cap, st);  // redo pass: FP32 sums of the large terms
  auto fd = EXAMD_ARR(double, smem + L.fa, 3 * cap, st);
  auto pd = EXAMD_ARR(double, smem + L.px, 3 * cap, st);
  auto px = EXAMD_ARR(unsigned long long, smem + L.px, 3 * cap, st);  // kFixed: fixed-point positions, images applied
  constexpr int kStage = FP64 || FIX ? 2 : 4;
  for (int t0 = tid; t0 < total; t0 += kStage * blockDim.x) {
    float4 uu[kStage];
    double xx[kStage][3];
#pragma unroll
    for (int k = 0; k < kStage; ++k) {
      const int t = t0 + k * blockDim.x;
      if (t < total) {
        const int cc = code[t];
        const int e = (cc & 31) + EX * (((cc >> 5) & 31) + EY * (cc >> 10));
        const int g = gfirst[e] + (t - (int)lstart[e]);
        uu[k] = U[g];
        if (FP64 || FIX) {
          const int64_t gg = EXAMD_IDX(g, A.N, st);
          xx[k][0] = A.X0[gg];
          xx[k][1] = A.X1[gg];
          xx[k][2] = A.X2[gg];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < kStage; ++k) {
      const int t = t0 + k * blockDim.x;
      if (t >= total) break;
      const int cc = code[t];
      const int lx = cc & 31, ly = (cc >> 5) & 31, lz = cc >> 10;
      const float4 u = uu[k];
      if (FP64) {
        pf[t] = make_float4(ox[lx] + u.x, oy[ly] + u.y, oz[lz] + u.z, u.w);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          pd[c * cap + t] = xx[k][c];
          fd[c * cap + t] = 0.0;
        }
      } else {
        // from a list: the atom's row (ly, lz) as two bf16 numbers in w (the list
        // pass subtracts both rows' at once; small integers, exact)
        pf[t] = make_float4(ox[lx] + u.x, u.y, u.z,
                            kFromList ? __uint_as_float((__float_as_uint((float)ly) >> 16) |
                                                        __float_as_uint((float)lz))
                                      : u.w);
        if (FIX) {
          px[t] = to_fixed(xx[k][0], A.fx.ue) + (unsigned long long)(img[lx] * B.Lq[0]);
          px[cap + t] = to_fixed(xx[k][1], A.fx.ue) + (unsigned long long)(img[32 + ly] * B.Lq[1]);
          px[2 * cap + t] = to_fixed(xx[k][2], A.fx.ue) + (unsigned long long)(img[64 + lz] * B.Lq[2]);
#pragma unroll
          for (int c = 0; c < 9; ++c) fa[c * cap + t] = 0;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (MODE == kRedoBig || MODE == kRedoFull || MODE == kListBig) fr[c * cap + t] = 0.f;
          // (list build: fa holds the atoms' entry counts, one word each)
          if (MODE == kMain || MODE == kRedoFull || MODE == kList || (MODE == kListBuild && c == 0))
            fa[MODE == kListBuild ? t : 3 * t + c] = 0;
        }
      }
    }
  }
  int* big_flag = cw + 1;  // mixed form: a term was too large for the fixed-point sums
  // list passes: the padding entries' atom, beyond every cutoff
  if (kFromList && tid == 0) pf[total] = make_float4(1e30f, 0.f, 0.f, 0.f);
  if (tid == 0) {
    cw[0] = 0;  // work-unit counter
    cw[3] = 0;  // list build: the tile's entries so far
    *big_flag = 0;
  }
  __syncthreads();

  const LJ32 q32 = A.lj.p32[0];
  const float rcpre = A.lj.rc2max * 1.0001f + 1e-4f;  // FP32 prefilter of the FP64 form
  double esum = 0.0, wsum = 0.0;  // FP64 form
  FixSum ek, wk;                  // mixed form: exact fixed-point sums of FP32 terms
  int ncand = 0, neval = 0, nacc = 0;
  // per-warp queue of accepted pairs (mixed form: the separation and the key
  // in one 16-byte entry, r^2 recomputed from it; FP64 form: the key only)
  // bytes per queue entry (the list build writes its pairs to the lists directly)
  constexpr int kQe = FP64 || FIX ? 4 : (MODE == kListBuild ? 0 : 16);
  auto qd = EXAMD_ARR(float4, (float4*)(smem + L.queue) + warp * kQueue, kQueue, st);
  auto qk = EXAMD_ARR(int, (int*)(smem + L.queue) + warp * kQueue, kQueue, st);
  // per-warp tables: one step's items (pt) and, but for the FP64 form, the
  // work unit's atoms (bt)
  unsigned char* wtab = smem + L.queue + kQe * kQueue * nw + warp * (FP64 ? kWarpTabFp64 : FIX ? kWarpTabFix : kWarpTab);
  auto pt = EXAMD_ARR(float4, wtab, 32, st);
  auto btA = EXAMD_ARR(float4, wtab + 32 * 16, 32, st);
  auto btB = EXAMD_ARR(float4, wtab + (FIX ? 32 * 16 : 32 * 32), 32, st);
  int qn = 0;  // queued pairs
  const unsigned lt = (1u << lane) - 1u;
  const unsigned le = FULL >> (31 - lane);
  auto r2l = EXAMD_ARR(unsigned char, smem + L.r2l + 64 * warp, FP64 ? 64 : 1, st);  // FP64 form: two rank -> lane tables of 32
  // ---- accepted pairs go to the warp's queue (a stack of kQueue entries);
  // their forces are computed in full batches of 32 ----
  // list build: an accepted pair (i, m) is entry k of atom i in the scratch
  // (i's entries side by side, lk per atom), k from the atom's counter (fa);
  // entries beyond lk are counted, not written (the tile then goes to the
  // fallback list)
  const size_t ltile = (size_t)tile * A.lslots;
  auto list_add = [&](bool acc, int key) {
    if (!acc) return;
    const int i = key & 0x3fff, m = (int)((unsigned)key >> 16);  // with several types: m and its type above 14 bits
    const int k = atomicAdd(&fa[i], 1);
    if (k < A.lk)
      A.lraw[EXAMD_IDX((ltile + i) * A.lk + k, (size_t)A.ntiles * A.lslots * A.lk, st)] = (unsigned short)m;
  };
  // ---- mixed form: the FP64 cutoff test of a pair of staged atoms (a, b)
  // at the border, r^2 from the FP64 positions as the FP64 form and the
  // reference form it: the difference, then the periodic image (the pair is
  // far nearer than half a box), SRC/exaMD_forces.f90:509-523 ----
  auto inside64 = [&](int a, int b, int ta, int tb) -> bool {
    auto gidx = [&](int t) {
      const int c = code[t];
      const int e = (c & 31) + EX * (((c >> 5) & 31) + EY * ((c >> 10) & 31));
      return (int64_t)gfirst[e] + (t - (int)lstart[e]);
    };
    const int64_t ga = EXAMD_IDX(gidx(a), A.N, st), gb = EXAMD_IDX(gidx(b), A.N, st);
    const double* Xs[3] = {A.X0, A.X1, A.X2};
    double d2 = 0.0;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      double d = __dsub_rn(Xs[ax][gb], Xs[ax][ga]);
      d = __dsub_rn(d, __dmul_rn(rint(__dmul_rn(d, B.Li[ax])), B.L[ax]));
      d2 = ax == 0 ? __dmul_rn(d, d) : __dadd_rn(d2, __dmul_rn(d, d));
    }
    const LJ64& Q = A.lj.p64[ta * A.lj.nt + tb];
    return d2 <= (FIX ? Q.rcut2 : Q.rc2);  // (kFixed: the potential's own range, as pair_fn64 decides it)
  };

  // kFixed: the separation of a pair whose copies lie in different periodic
  // images, d = t + n L with t = x_j - x_i: t rounded to 53 bits, ties to even,
  // as the FP64 subtraction rounds it (|t| = L - |d| has L's exponent, or the
  // next lower one where |d| is above qthr; L is a multiple of that bit)
  const bool edge = FIX && (X0 == 0 || Y0 == 0 || Z0 == 0 || X0 + tx >= B.nb[0] || Y0 + ty >= B.nb[1] ||
                            Z0 + tz >= B.nb[2]);
  auto face = [&](int i, int m, long long& dx, long long& dy, long long& dz) {
    const int ci = code[i], cm = code[m];
    auto round_axis = [&](int a, int li, int lm, long long& d) {
      const int n = img[32 * a + lm] - img[32 * a + li];
      if (n == 0) return;
      const long long nl = n > 0 ? B.Lq[a] : -B.Lq[a];
      const unsigned long long t = (unsigned long long)(d - nl);
      const int q = B.qbit[a] - ((d < 0 ? -d : d) > B.qthr[a] ? 1 : 0);
      const unsigned long long r = t + (1ull << (q - 1)) - 1ull + ((t >> q) & 1ull);
      d = (long long)((r >> q) << q) + nl;
    };
    round_axis(0, ci & 31, cm & 31, dx);
    round_axis(1, (ci >> 5) & 31, (cm >> 5) & 31, dy);
    round_axis(2, (ci >> 10) & 31, (cm >> 10) & 31, dz);
  };
  auto enqueue = [&](bool acc, const float4& dq, int key) {
    const unsigned bal = __ballot_sync(FULL, acc);
    if (acc) {
      const int p = qn + __popc(bal & lt);
      if (FP64 || FIX)
        qk[p] = key;
      else
        qd[p] = make_float4(dq.x, dq.y, dq.z, __int_as_float(key));
    }
    qn += __popc(bal);
    if (qn >= 32) {  // a batch: the last 32, so that what is left stays where it is
      qn -= 32;
      __syncwarp();
      if (FP64)
        force_batch64<MULTI, ENERGY, COUNT>(32, qk, pd, code, img, B.L, fd, cap, A.lj, ljs64, esum, wsum, A.status,
                                            nacc, qn);
      else if (FIX)
        force_batch_fix<MULTI, ENERGY, COUNT>(32, qn, qk, px, fa, cap, A, ljx, esum, wsum, nacc, big_flag,
                                              edge, face, inside64);
      else
        force_batch<MULTI, ENERGY, COUNT, MODE == kRedoFull>(32, qn, qd, fa, fr, cap, A, ljs32, ek, wk, nacc,
                                                             big_flag, inside64);
      __syncwarp();
    }
  };

  // ---- redo pass: the force of each accepted pair at once; only the large
  // terms, decided exactly as force_batch decides them, are summed (both atoms)
  auto redo_pair = [&](bool acc, const float4& dq, int key) {
    if (!acc) return;
    const int i = key & 0x3fff, m = (key >> 16) & 0x3fff;
    LJ32 P = A.lj.p32[0];
    if (MULTI) P = ljs32[((key >> 14) & 3) * A.lj.nt + ((unsigned)key >> 30)];
    float dg = 0.f, e = 0.f;
    if (pair_fn32<false>(A.lj.pot, dq.w, P, dg, e) != 0) return;
    const float dgs = kFix * dg;
    const float fx = dgs * dq.x, fy = dgs * dq.y, fz = dgs * dq.z;
    if (!(dq.w < P.r2big)) return;
    atomicAdd(&fr[i], fx * kFixInv);
    atomicAdd(&fr[cap + i], fy * kFixInv);
    atomicAdd(&fr[2 * cap + i], fz * kFixInv);
    atomicAdd(&fr[m], -fx * kFixInv);
    atomicAdd(&fr[cap + m], -fy * kFixInv);
    atomicAdd(&fr[2 * cap + m], -fz * kFixInv);
  };

  // ---- consume one step's (atom, row) items, at most one per lane (n <= 0:
  // none): the atom at (x, y, z) (tile-frame x; y, z from its row's origin)
  // against the staged atoms [lo, lo + n), whose row's origin is offset by
  // (cy, cz).  The items' candidate pairs are laid end to end and the warp
  // walks them 32 at a time, one pair per lane, so no lane idles while another
  // finishes a long j-range.  A lane finds its item from the bitmask of the
  // items that start in the current 32 candidates, and reads it from the
  // per-warp table by its rank: one 16-byte word, the atom's position moved into
  // the j-cells' frame and id + ((lo - s0) << 16), to which candidate k adds
  // k << 16: the sum is the pair's key (the j-range's upper half wraps).
  // (Shared-memory wavefronts bound this walk: 83 % of the cycles on a mixture.
  // An item of two words, with room for the rare second run, cost 2 of 13 per
  // window; a second run is now an item of a second call.)
  auto consume = [&](int id, float x, float y, float z, float cy, float cz, int lo, int n) {
    const unsigned hb = __ballot_sync(FULL, n > 0);
    if (hb == 0u) return;
    const int nt = max(n, 0);
    // exclusive scan of the items' candidate counts
    int incl = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y2 = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y2;
    }
    const int s0 = incl - nt;
    const int T = __shfl_sync(FULL, incl, 31);
    if (nt > 0) pt[__popc(hb & lt)] = make_float4(-x, cy - y, cz - z, __int_as_float(id + ((lo - s0) << 16)));
    __syncwarp();
    // distance tests; accepted pairs go to the queue
    int qb = 0;  // items that start before K
    const int sw = nt > 0 ? s0 >> 5 : -1;  // the 32-candidate window in which the item starts
    const unsigned sbit = 1u << (s0 & 31);
    for (int K = 0, kw = 0; K < T; K += 32, ++kw) {
      const unsigned M = __reduce_or_sync(FULL, sw == kw ? sbit : 0u);
      const int qr = qb + __popc(M & le) - 1;  // >= 0: the first item starts at 0
      qb += __popc(M);
      const float4 a = pt[qr];
      const int k = K + lane;
      const bool valid = k < T;
      const unsigned kb = (unsigned)__float_as_int(a.w) + ((unsigned)k << 16);
      const int m = (int)(kb >> 16);
      const float4 pj = pf[valid ? m : 0];
      float4 dq;
      dq.x = pj.x + a.x;
      dq.y = pj.y + a.y;
      dq.z = pj.z + a.z;
      dq.w = fmaf(dq.x, dq.x, fmaf(dq.y, dq.y, dq.z * dq.z));
      const int tj = __float_as_int(pj.w), ti = MULTI ? (kb >> 14) & 3 : 0;
      if (COUNT && valid) ++neval;
      const float thr = FIX ? (MULTI ? ljx[ti * A.lj.nt + tj].pre : A.fx.p[0].pre)
                        : MODE == kListBuild ? (MULTI ? ljs32[ti * A.lj.nt + tj].rl2 : q32.rl2)
                        : MODE == kRedoBig   ? (MULTI ? ljs32[ti * A.lj.nt + tj].rc2 : q32.rc2)
                                             : (MULTI ? ljs32[ti * A.lj.nt + tj].rc2 * kWiden : q32.rc2 * kWiden);
      const int key = (int)(kb + (MULTI ? (unsigned)tj << 30 : 0u));
      const bool acc = valid && dq.w <= thr;
      if (MODE == kRedoBig)
        redo_pair(acc, dq, key);
      else if (MODE == kListBuild)
        list_add(acc, key);
      else
        enqueue(acc, dq, key);
    }
    __syncwarp();
  };

  // ---- FP64 form: consume one step's (ext cell, row) blocks ----
  // Item (at most one per lane): atoms [i0, i0 + ni) of one cell against the
  // j-range(s) [lo1, lo1 + n1) and [lo2, lo2 + n2) of one owned row; in the
  // row through the cell itself (self) only j > i.  The items' ni * nj
  // candidate pairs are laid end to end and tested 32 at a time, one per lane,
  // against the FP32 prefilter.  A lane finds its item from the bitmask of
  // item starts and splits its index into (i, j) by a float division
  // corrected to the exact quotient.  Consecutive queued pairs then share an
  // i only within one block (a few pairs), which keeps the FP64 batches'
  // shared-memory atomics on i from serialising; the atom-item order of the
  // mixed form would put one atom's whole row list (~30 pairs) in a batch.
  auto consume_cells = [&](int i0, int ni, int lo1, int n1, int lo2, int n2, bool self) {
    const int nj = n1 + n2;
    const int nt = ni * nj;
    const unsigned hb = __ballot_sync(FULL, nt > 0);
    if (hb == 0u) return;
    int incl = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, incl, o);
      if (lane >= o) incl += y;
    }
    const int s0 = incl - nt;
    const int T = __shfl_sync(FULL, incl, 31);
    const int pa = i0 | (ni << 16), p1 = lo1 | (n1 << 16), l2 = lo2 - n1, pn = nj | (self ? 1 << 16 : 0);
    if (nt > 0) {
      pt[lane] = make_float4(0.f, 0.f, 1.0f / (float)nj, __int_as_float(s0));
      r2l[32 + __popc(hb & lt)] = (unsigned char)lane;
    }
    __syncwarp();
    int qb = 0;  // items that start before K
    const int sw = nt > 0 ? s0 >> 5 : -1;  // the 32-candidate window in which the item starts
    const unsigned sbit = 1u << (s0 & 31);
    for (int K = 0, kw = 0; K < T; K += 32, ++kw) {
      const unsigned M = __reduce_or_sync(FULL, sw == kw ? sbit : 0u);
      const int qr = qb + __popc(M & le) - 1;  // >= 0: the first item starts at 0
      qb += __popc(M);
      const int ql = r2l[32 + qr];
      const int bpa = __shfl_sync(FULL, pa, ql), bp1 = __shfl_sync(FULL, p1, ql);
      const int bl2 = __shfl_sync(FULL, l2, ql), bpn = __shfl_sync(FULL, pn, ql);
      const float4 a = pt[ql];
      const int k = K + lane;
      const int kl = k - __float_as_int(a.w);
      const int bnj = bpn & 0xffff;
      int ia = __float2int_rz(((float)kl + 0.5f) * a.z);
      int jb = kl - ia * bnj;
      if (jb < 0) {
        --ia;
        jb += bnj;
      } else if (jb >= bnj) {
        ++ia;
        jb -= bnj;
      }
      const bool valid = k < T && (!(bpn >> 16) || jb > ia);
      const int i = (bpa & 0xffff) + ia;
      const int m = jb < (bp1 >> 16) ? (bp1 & 0xffff) + jb : bl2 + jb;
      const float4 pi = pf[valid ? i : 0], pj = pf[valid ? m : 0];
      float4 dq;  // positions are in the tile frame: no row offset
      dq.x = pj.x - pi.x;
      dq.y = pj.y - pi.y;
      dq.z = pj.z - pi.z;
      dq.w = fmaf(dq.x, dq.x, fmaf(dq.y, dq.y, dq.z * dq.z));
      const int ti = __float_as_int(pi.w), tj = __float_as_int(pj.w);
      if (COUNT && valid) {
        ++ncand;
        ++neval;
      }
      enqueue(valid && dq.w <= rcpre, dq, i | (ti << 14) | (m << 16) | (tj << 30));
    }
    __syncwarp();
  };

  int* ucnt = cw;  // work-unit counter
  if constexpr (kFromList) {
    // ---- forces from the tile's lists ----
    // The build ordered the staged atoms by entry count, most first; a warp
    // takes 32 consecutive atoms of that order, one per lane, so its lanes
    // have about as many entries each and few idle while the longest runs
    // out.  A lane reads four entries at a time, the warp's 32 lanes' four
    // side by side (one 256-byte load per warp), the next four loaded
    // ahead.  Entry m of atom i is the pair (i, m).  The separation is
    // formed as the first pass forms it: x in the tile frame, y and z from
    // the atoms' cell offsets and the origin offset between their rows (read
    // from the rows in the staged codes); the same bits when the atoms are
    // where the lists were built.  Atom i's terms add up in registers (exact
    // integer sums) and go to shared memory once; m's go at once.
    const int lk = A.lk;
    const unsigned short* lst = A.list + ltile * lk;
    const unsigned short* perm = A.lperm + ltile;
    const unsigned short* cnts = A.lcnt + ltile;
    const int ng = (total + 31) >> 5;
    constexpr int kBurst = MULTI ? 1 : 2;  // entries taken together (several types: no registers for two)
    bool bigl = false, perr = false;  // a large term left out; a pair-function error
    // The origin offset between rows l and l + d (d = -2..2 for a listed
    // pair) is fmaf(image difference, r, d bl) in the tables: d bl itself
    // (exact) unless the tile reaches the box's periodic face on that axis
    // and the box's last cell is wider by r != 0.  Such tiles read the
    // tables; the others form d bl in registers, the same bits.
    const bool taby = B.remf[1] != 0.f && (Y0 == 0 || Y0 + ty >= B.nb[1]);
    const bool tabz = B.remf[2] != 0.f && (Z0 == 0 || Z0 + tz >= B.nb[2]);
    const float blf = B.blf;
    const float band0 = kBorder * q32.rc2, m24k0 = kFix * q32.m24eps;
    while (true) {
      int g = 0;
      if (lane == 0) g = atomicAdd(ucnt, 1);
      g = __shfl_sync(FULL, g, 0);
      if (g >= ng) break;
      const int r = g * 32 + lane;
      const bool vi = r < total;
      const int ip = vi ? perm[r] : 0;
      const int i = MULTI ? ip & 0x3fff : ip, ti = MULTI ? ip >> 14 : 0;
      const int cnt = vi ? cnts[r] : 0;
      const int gm = __shfl_sync(FULL, cnt, 0);  // the order puts the group's longest first
      const float4 pi = pf[i];
      const unsigned wi = __float_as_uint(pi.w);
      const int ci = code[i];
      const int lrow = ti * A.lj.nt;
      // entries k..k+3 of this lane: 8 bytes at brick k / 4 of the group
      const uint2* col = reinterpret_cast<const uint2*>(lst + (size_t)g * 32 * lk) + lane;
      // (every lane's bricks hold entries up to the group's longest, the
      // padding entries naming the far atom `total`: no per-lane count test)
      auto four = [&](int k) { return k < gm ? __ldcs(col + (size_t)(k >> 2) * 32) : make_uint2(0u, 0u); };
      uint2 nxt = four(0);
      int sx = 0, sy = 0, sz = 0;  // atom i's fixed-point sums
      // the entries, in one of two versions: row offsets from the tables or
      // formed in registers (no table load)
      auto walk = [&](auto tables) {
      constexpr bool TAB = decltype(tables)::value;
      for (int k0 = 0; k0 < gm; k0 += 4) {
        const uint2 cur = nxt;
        nxt = four(k0 + 4);
        const unsigned wv[2] = {cur.x, cur.y};
#pragma unroll
        for (int q0 = 0; q0 < 4; q0 += kBurst) {
          unsigned en[kBurst];
          float4 dq[kBurst];
          LJ32 P[kBurst];
          bool rare = false;
#pragma unroll
          for (int b = 0; b < kBurst; ++b) {
            const int q = q0 + b;
            en[b] = (q & 1) ? wv[q >> 1] >> 16 : wv[q >> 1] & 0xffffu;
            const int m = MULTI ? en[b] & 0x3fff : en[b];  // the entry: the staged atom, and its type above 14 bits
            const float4 pj = pf[m];
            // y, z of atom i in the frame of atom j's row: (the row origins'
            // offset) - pi, rounded once
            float yi, zi;
            if constexpr (TAB) {  // (the table entry of rows l, l + d: l kDT + d + 2)
              const int cm = code[EXAMD_IDX(min(m, total - 1), cap, st)];
              yi = dyt[((ci >> 5) & 31) * (kDT - 1) + 2 + ((cm >> 5) & 31)].x - pi.y;
              zi = dzt[(ci >> 10) * (kDT - 1) + 2 + (cm >> 10)].x - pi.z;
            } else {  // d bl, exact: both rows' differences d in one bf16x2 subtraction
              const unsigned wj = __float_as_uint(pj.w);
              const __nv_bfloat162 dr = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&wj),
                                                *reinterpret_cast<const __nv_bfloat162*>(&wi));
              const unsigned du = *reinterpret_cast<const unsigned*>(&dr);
              yi = fmaf(__uint_as_float(du << 16), blf, -pi.y);
              zi = fmaf(__uint_as_float(du & 0xffff0000u), blf, -pi.z);
            }
            dq[b].x = pj.x - pi.x;
            dq[b].y = pj.y + yi;
            dq[b].z = pj.z + zi;
            dq[b].w = fmaf(dq[b].x, dq[b].x, fmaf(dq[b].y, dq[b].y, dq[b].z * dq[b].z));
            P[b] = MULTI ? ljs32[lrow + (en[b] >> 14)] : q32;
            rare |= fabsf(dq[b].w - P[b].rc2) <= (MULTI ? kBorder * P[b].rc2 : band0) || dq[b].w < P[b].r2big;
          }
          if (MODE == kListBig) {
#pragma unroll
            for (int b = 0; b < kBurst; ++b)
              redo_pair(dq[b].w <= P[b].rc2, dq[b], i | (ti << 14) | (int)(en[b] << 16));
            continue;
          }
          // The LJ family's expression of pair_fn32 (the potential was checked
          // per tile) for every entry, its result kept where the entry applies:
          // some lane of the warp takes nearly every entry.  The same expressions:
          // the same bits as pair_fn32 where it applies.  The scale kFix is in m24
          // (a power of two).  An entry applies within rc (and the potential's own
          // range).  What is rare -- an r^2 at the border (the FP64 test), a large
          // term (left to the redo pass), a pair-function error (r^2 < kR2Min32
          // <= r2big) -- is looked for in kBurst entries at once, and all of the
          // warp's then go through the careful version: with a branch in every
          // entry their arithmetic did not interleave.
          auto apply = [&](auto careful) {
#pragma unroll
            for (int b = 0; b < kBurst; ++b) {
              const int m = MULTI ? en[b] & 0x3fff : en[b];
              const float r2 = dq[b].w;
              const float m24 = MULTI ? P[b].m24eps : m24k0;
              const float ri = rcp_approx(r2);
              const float s2 = P[b].sig2 * ri;
              const float s6 = s2 * s2 * s2;
              const float dgs = m24 * s6 * fmaf(2.f, s6, -1.f) * ri;
              bool fix = r2 <= P[b].rc2 && !(CUT && r2 > P[b].rcut2);
              bool app = fix;
              if constexpr (decltype(careful)::value) {
                const bool edge64 = fabsf(r2 - P[b].rc2) <= (MULTI ? kBorder * P[b].rc2 : band0);
                const bool acc = edge64 ? inside64(i, m, ti, MULTI ? en[b] >> 14 : 0) : r2 <= P[b].rc2;
                perr |= acc && !(r2 >= kR2Min32);
                app = acc && r2 >= kR2Min32 && !(CUT && r2 > P[b].rcut2);
                bigl |= app && r2 < P[b].r2big;
                fix = app && !(r2 < P[b].r2big);
              }
              if (ENERGY && app) {
                ek.add(P[b].c4eps * s6 * (s6 - 1.f) - P[b].eshift);
                wk.add(-(dgs * kFixInv) * r2);
              }
              // atom m's terms; atom i's are the same with the other sign
              const int jx = __float2int_rn(-(dgs * dq[b].x)), jy = __float2int_rn(-(dgs * dq[b].y)),
                        jz = __float2int_rn(-(dgs * dq[b].z));
              if (fix) {
                atomicAdd(&fa[3 * m], jx);
                atomicAdd(&fa[3 * m + 1], jy);
                atomicAdd(&fa[3 * m + 2], jz);
                sx -= jx;
                sy -= jy;
                sz -= jz;
              }
            }
          };
          if (__any_sync(FULL, rare))
            apply(std::true_type{});
          else
            apply(std::false_type{});
        }
      }
      };
      if (taby || tabz)
        walk(std::true_type{});
      else
        walk(std::false_type{});
      if (MODE == kList && (sx | sy | sz) != 0) {
        atomicAdd(&fa[3 * i], sx);
        atomicAdd(&fa[3 * i + 1], sy);
        atomicAdd(&fa[3 * i + 2], sz);
      }
    }
    if (bigl) *big_flag = 1;
    if (perr) atomicOr(A.status, ST_PAIRFN);
  } else if constexpr (!FP64) {
    // ---- item building: (staged atom, owned row) pairs, laid end to end ----
    // A unit is 32 consecutive staged atoms and one of kParts shares of each
    // atom's list of owned rows (the rows whose ownership mask for the atom's
    // position class is nonzero; ordinals n = kParts m + part).  The warp lays
    // the unit's (atom, row) pairs end to end and builds one item per lane per
    // step, so lanes do not idle on atoms that own few rows (the halo).  Units are handed out by a
    // shared counter: their cost varies, and the force sums do not depend on the
    // order.  An item is the atom's j-range(s) in the row: the owned cells,
    // trimmed to those whose box comes within rc of the atom (the 1e-4 margin in
    // prune2 covers the FP32 rounding; the accepted pairs are unchanged).
    const int nunits = kParts * ((total + 31) >> 5);
    const float prune2 = MODE == kListBuild ? A.lj.prune2_list : A.lj.prune2;
    while (true) {
      int u = 0;
      // (kFixed: a tile with a term too large is the FP64 body's, and not finished here)
      if (lane == 0) u = FIX && *(volatile int*)big_flag ? nunits : atomicAdd(ucnt, 1);
      u = __shfl_sync(FULL, u, 0);
      if (u >= nunits) break;
      const int c = u / kParts, part = u - c * kParts;
      // per-atom quantities of lane l's atom c*32 + l
      const int ia = c * 32 + lane;
      const bool va = ia < total;
      const int cia = code[va ? ia : 0];
      const int ax = cia & 31, ay = (cia >> 5) & 31, az = cia >> 10;
      const int acls = pos_class(ax - 1, tx) * 25 + pos_class(ay - 1, ty) * 5 + pos_class(az - 1, tz);
      const int aw = va ? (own_nrow(acls) + kParts - 1 - part) / kParts : 0;
      const float4 pa = pf[va ? ia : 0];
      // squared x-gaps to the cells dx = -2, -1, +1, +2 (ox has EX + 1 entries)
      const float gm2 = fmaxf(pa.x - ox[max(ax - 1, 0)], 0.f), gm1 = fmaxf(pa.x - ox[ax], 0.f);
      const float gp1 = fmaxf(ox[min(ax + 1, EX)] - pa.x, 0.f), gp2 = fmaxf(ox[min(ax + 2, EX)] - pa.x, 0.f);
      const float am2 = gm2 * gm2, am1 = gm1 * gm1, ap1 = gp1 * gp1, ap2 = gp2 * gp2;
      int incl = aw;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
      }
      const int as0 = incl - aw, W = __shfl_sync(FULL, incl, 31);
      const unsigned wb = __ballot_sync(FULL, aw > 0);
      if (aw > 0) {  // the working atoms' data by rank (as0 < 512, ia < 2^14, acls < 128)
        const int rk = __popc(wb & lt);
        const int wa = as0 | (ia << 9), wc = cia | (acls << 15) | (MULTI ? __float_as_int(pa.w) << 22 : 0);
        // the gaps as FP16 rounded toward zero: they prune no more than they may
        const __half2 hm = __halves2half2(__float2half_rz(am2), __float2half_rz(am1));
        const __half2 hp = __halves2half2(__float2half_rz(ap1), __float2half_rz(ap2));
        if (!FIX) btA[rk] = make_float4(pa.x, pa.y, pa.z, 0.f);
        btB[rk] = make_float4(*reinterpret_cast<const float*>(&hp), __int_as_float(wa), __int_as_float(wc),
                              *reinterpret_cast<const float*>(&hm));
      }
      __syncwarp();
      int qb = 0;  // working atoms that start before K
      const int aww = aw > 0 ? as0 >> 5 : -1;  // the 32-item window in which the atom's items start
      const unsigned abit = 1u << (as0 & 31);
      for (int K = 0, kw = 0; K < W; K += 32, ++kw) {
        const unsigned M = __reduce_or_sync(FULL, aww == kw ? abit : 0u);
        const int qr = qb + __popc(M & (FULL >> (31 - lane))) - 1;  // >= 0: the first worker starts at 0
        qb += __popc(M);
        const int k = K + lane;
        const bool valid = k < W;
        const float4 b1v = btB[qr];
        const int sq = __float_as_int(b1v.y), cc = __float_as_int(b1v.z);
        const int s_q = sq & 511, i = sq >> 9;
        const float4 b0v = FIX ? pf[i] : btA[qr];
        const int cls = (cc >> 15) & 127;
        const int lx = cc & 31, ly = (cc >> 5) & 31, lz = (cc >> 10) & 31;
        const unsigned ent = valid ? own_ent(cls, kParts * (k - s_q) + part) : 0u;
        int mask = ent & 31;
        int lo1 = 0, n1 = 0, lo2 = 0, n2 = 0;
        float cy = 0.f, cz = 0.f;
        if (mask) {
          const int yc = (ent >> 5) & 7, zc = (ent >> 8) & 7;  // dy + 2, dz + 2
          const int dy = yc - 2, dz = zc - 2;
          const bool selfrow = ent >> 11;
          const int rowbase = ((ly + dy) + EY * (lz + dz)) * EX + lx - 2;  // + bit b -> ext cell of dx = b - 2
          const float2 ry = dyt[ly * kDT + yc], rz = dzt[lz * kDT + zc];
          cy = ry.x;
          cz = rz.x;
          if (COUNT) {  // every atom of the owned cells, as the reference visits them
            for (int b = 0; b < 5; ++b)
              if ((mask >> b) & 1) {
                const int e = rowbase + b;
                ncand += (selfrow && b == 2) ? lstart[e + 1] - i - 1 : lstart[e + 1] - lstart[e];
              }
          }
          // distance from the atom to the row's cell boxes
          // (the row's near face comes with its origin offset)
          const float ty = ry.y - b0v.y, tz = rz.y - b0v.z;
          const float gy = fmaxf(__int_as_float(__float_as_int(ty) ^ (dy & 0x80000000)), 0.f);
          const float gz = fmaxf(__int_as_float(__float_as_int(tz) ^ (dz & 0x80000000)), 0.f);
          const float tr = prune2 - (gy * gy + gz * gz);
          if (tr < 0.f) mask = 0;
          // the x-gaps beyond tr, compared as FP16 (tr rounded up, so that no cell is pruned wrongly)
          const __half2 tr2 = __half2half2(__float2half_ru(tr));
          const unsigned pm = (__hgt2_mask(*reinterpret_cast<const __half2*>(&b1v.w), tr2) & 0x00020001u) |
                              (__hgt2_mask(*reinterpret_cast<const __half2*>(&b1v.x), tr2) & 0x00100008u);
          mask &= ~(pm | (pm >> 16));
          if (mask) {
            const int b0 = __ffs(mask) - 1, b1 = 31 - __clz(mask);
            const int mm = mask >> b0;
            lo1 = lstart[rowbase + b0];
            int hi1 = lstart[rowbase + b1 + 1];
            if (mm & (mm + 1)) {  // two runs: [b0, e1) and [b2, b1]
              const int e1 = b0 + __ffs(~mm) - 1;
              const int b2 = __ffs(mask & ~((1 << e1) - 1)) - 1;
              lo2 = lstart[rowbase + b2];
              n2 = hi1 - lo2;
              hi1 = lstart[rowbase + e1];
            }
            n1 = hi1 - lo1;
            if (selfrow && b0 == 2) {  // pairs inside the cell: a2 > a1
              n1 -= i + 1 - lo1;
              lo1 = i + 1;
            }
          }
        }
        const int id = i | (MULTI ? (cc >> 22) << 14 : 0);
        while (true) {
          consume(id, b0v.x, b0v.y, b0v.z, cy, cz, lo1, n1);
          if (!__any_sync(FULL, n2 > 0)) break;  // a second run: 0.6 % of the items, most steps have none
          lo1 = lo2;
          n1 = n2;
          n2 = 0;
        }
      }
      __syncwarp();
    }
  } else {
    // ---- item building: (ext cell, owned row) pairs, laid end to end ----
    // A unit is 32 consecutive ext cells and one of kCellParts shares of each
    // cell's owned rows; empty cells have no work.  An item is the row's owned
    // j-cells as at most two contiguous runs (no per-atom trimming: the block
    // is tested in full).
    constexpr int kCellParts = 4;
    const int nunits = kCellParts * ((NE + 31) >> 5);
    while (true) {
      int u = 0;
      if (lane == 0) u = atomicAdd(ucnt, 1);
      u = __shfl_sync(FULL, u, 0);
      if (u >= nunits) break;
      const int c = u / kCellParts, part = u - c * kCellParts;
      const int e = c * 32 + lane;
      const bool ve = e < NE;
      const int ee = ve ? e : 0;
      const int ex = ee % EX, er = ee / EX, ey = er % EY, ez = er / EY;
      const int ai0 = lstart[ee], ana = ve ? lstart[ee + 1] - ai0 : 0;
      const int acls = pos_class(ex - 1, tx) * 25 + pos_class(ey - 1, ty) * 5 + pos_class(ez - 1, tz);
      const int aw = ana > 0 ? (own_nrow(acls) + kCellParts - 1 - part) / kCellParts : 0;
      int incl = aw;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += y;
      }
      const int as0 = incl - aw, W = __shfl_sync(FULL, incl, 31);
      const unsigned wb = __ballot_sync(FULL, aw > 0);
      if (aw > 0) r2l[__popc(wb & lt)] = (unsigned char)lane;
      __syncwarp();
      const int ageo = ex | (ey << 5) | (ez << 10) | (acls << 15);
      const int apa = ai0 | (ana << 16);
      int qb = 0;
      const int aww = aw > 0 ? as0 >> 5 : -1;  // the 32-item window in which the cell's items start
      const unsigned abit = 1u << (as0 & 31);
      for (int K = 0, kw = 0; K < W; K += 32, ++kw) {
        const unsigned M = __reduce_or_sync(FULL, aww == kw ? abit : 0u);
        const int qr = qb + __popc(M & le) - 1;
        qb += __popc(M);
        const int k = K + lane;
        const bool valid = k < W;
        const int ql = r2l[qr];
        const int s_q = __shfl_sync(FULL, as0, ql);
        const int geo = __shfl_sync(FULL, ageo, ql);
        const int qpa = __shfl_sync(FULL, apa, ql);
        const int lx = geo & 31, ly = (geo >> 5) & 31, lz = (geo >> 10) & 31, cls = geo >> 15;
        const unsigned ent = valid ? own_ent(cls, kCellParts * (k - s_q) + part) : 0u;
        const int mask = ent & 31;
        int lo1 = 0, n1 = 0, lo2 = 0, n2 = 0;
        bool self = false;
        if (mask) {
          const int dy = (int)((ent >> 5) & 7) - 2, dz = (int)((ent >> 8) & 7) - 2;
          const int rowbase = ((ly + dy) + EY * (lz + dz)) * EX + lx - 2;  // + bit b -> ext cell of dx = b - 2
          const int b0 = __ffs(mask) - 1, b1 = 31 - __clz(mask);
          const int mm = mask >> b0;
          lo1 = lstart[rowbase + b0];
          int hi1 = lstart[rowbase + b1 + 1];
          if (mm & (mm + 1)) {  // two runs: [b0, e1) and [b2, b1]
            const int e1 = b0 + __ffs(~mm) - 1;
            const int b2 = __ffs(mask & ~((1 << e1) - 1)) - 1;
            lo2 = lstart[rowbase + b2];
            n2 = hi1 - lo2;
            hi1 = lstart[rowbase + e1];
          }
          n1 = hi1 - lo1;
          self = (dy | dz) == 0 && b0 == 2;  // the first run starts at the cell itself
          if (n1 <= 0 && !self) {
            lo1 = lo2;
            n1 = n2;
            lo2 = 0;
            n2 = 0;
          }
        }
        consume_cells(qpa & 0xffff, qpa >> 16, lo1, n1, lo2, n2, self);
      }
      __syncwarp();
    }
  }
  if (qn > 0) {  // the last, partial batch
    __syncwarp();
    if (FP64)
      force_batch64<MULTI, ENERGY, COUNT>(qn, qk, pd, code, img, B.L, fd, cap, A.lj, ljs64, esum, wsum, A.status,
                                          nacc, 0);
    else if (FIX)
      force_batch_fix<MULTI, ENERGY, COUNT>(qn, 0, qk, px, fa, cap, A, ljx, esum, wsum, nacc, big_flag,
                                            edge, face, inside64);
    else
      force_batch<MULTI, ENERGY, COUNT, MODE == kRedoFull>(qn, 0, qd, fa, fr, cap, A, ljs32, ek, wk, nacc,
                                                           big_flag, inside64);
  }
  __syncthreads();
  // a large term was left out: list the tile for the redo pass
  // (kFixed: the same CTA computes it in full by the FP64 body)
  if (!FP64 && (MODE == kMain || MODE == kList) && tid == 0 && *big_flag) A.redo[atomicAdd(A.redo_n, 1)] = tile;
  if (FIX && *big_flag) return true;
  if (MODE == kListBuild) {
    // The atoms in the order of their entry counts, most first (a counting
    // sort), and the entries moved from the scratch into that order; a tile
    // with an atom over lk goes to the fallback list.
    const int lk = A.lk;
    auto perm = EXAMD_ARR(unsigned short, smem + L.perm, cap, st);
    auto hist = EXAMD_ARR(int, smem + L.hist, kMaxListK + 1, st);
    int mx = 0;
    for (int c = tid; c <= lk; c += blockDim.x) hist[c] = 0;
    __syncthreads();
    for (int t = tid; t < total; t += blockDim.x) {
      const int c = fa[t];
      mx = max(mx, c);
      atomicAdd(&hist[min(c, lk)], 1);
    }
    mx = warp_max(mx);
    if (lane == 0) atomicMax(&cw[3], mx);
    __syncthreads();
    if (warp == 0) {  // exclusive scan from the largest count down
      int run = 0;
      for (int c0 = lk; c0 >= 0; c0 -= 32) {
        const int c = c0 - lane;
        const int h = c >= 0 ? hist[c] : 0;
        int x = h;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(FULL, x, o);
          if (lane >= o) x += y;
        }
        if (c >= 0) hist[c] = run + x - h;
        run += __shfl_sync(FULL, x, 31);
      }
    }
    __syncthreads();
    for (int t = tid; t < total; t += blockDim.x)
      perm[atomicAdd(&hist[min((int)fa[t], lk)], 1)] = (unsigned short)(t | (MULTI ? __float_as_int(pf[t].w) << 14 : 0));
    __syncthreads();
    // A lane moves its atom's entries from the scratch row into the group's
    // bricks (4 entries of 32 lanes side by side); every lane fills the group's
    // bricks up to the group's longest count, the entries past its own count
    // naming the padding atom `total` (staged by the list passes beyond every
    // cutoff), so that the list pass tests no per-lane count.
    //
    // On the way every 32 entries are put in an order that spreads the list
    // pass's shared-memory reads: at step k its lane reads the 16-byte position
    // of entry k, eight lanes a wavefront, and adds to three words of the same
    // atom.  Entry k is therefore taken, where there is one, among those with
    // m = lane + k modulo 8: eight neighbouring lanes then read eight different
    // bank groups, and of the four lanes of one residue few meet in a bank.
    // (Unordered, bank conflicts were 55 % of the list pass's shared wavefronts
    // and those 68 % of its cycles.)  The entry of rank r in residue class c goes
    // to step (c - lane) % 8 + 8 r, or, if that is past the atom's entries or
    // taken, to the last free step.  The sums are exact integers, so the order
    // changes no bit.
    constexpr int kRowBytes = 72, kOrd = 32;  // a lane's row of kOrd entries; 18 words: 8-byte reads without conflicts
    const int row0 = align16(L.perm < L.pf ? L.hist + 4 * (kMaxListK + 1) : L.queue);  // up to the counts at L.fa: free now
    const int nrow = min(nw, (L.fa - row0) / (32 * kRowBytes));  // warps that have room for their rows
    const size_t nbrick = (size_t)A.ntiles * A.lslots * lk / 4;
    const unsigned short* raw = A.lraw + ltile * lk;
    (void)nbrick;
    for (int g = warp < nrow ? warp : total; g * 32 < total; g += nrow) {
      const int p = g * 32 + lane;
      const int pv = p < total ? perm[p] : 0;
      const int t = MULTI ? pv & 0x3fff : pv;
      const int c = p < total ? min((int)fa[t], lk) : 0;
      A.lperm[EXAMD_IDX(ltile + p, (size_t)A.lslots * A.ntiles, st)] = (unsigned short)pv;
      A.lcnt[EXAMD_IDX(ltile + p, (size_t)A.lslots * A.ntiles, st)] = (unsigned short)c;
      const int gm = __shfl_sync(FULL, c, 0);
      const unsigned short* own = raw + (size_t)t * lk;
      unsigned short* row = (unsigned short*)(smem + row0 + (32 * warp + lane) * kRowBytes);
      const size_t b0 = (ltile + (size_t)g * 32) * lk / 4 + lane;  // brick k / 4 of this lane: b0 + (k / 4) * 32
      uint2* dst = reinterpret_cast<uint2*>(A.list);
      const unsigned dd = (unsigned)total * 0x10001u;  // two padding entries
      // word w holds two entries, left of them the atom's
      auto pad = [&](unsigned w, int left) {
        return left >= 2 ? w : (left == 1 ? (w & 0xffffu) | (dd & 0xffff0000u) : dd);
      };
      for (int k0 = 0; k0 < gm; k0 += kOrd) {
        const int n = min(c - k0, kOrd);  // this lane's entries of the round
        uint4 v[4];                       // the four 16-byte reads issued first
#pragma unroll
        for (int u = 0; u < 4; ++u)
          v[u] = 8 * u < n ? reinterpret_cast<const uint4*>(own + k0)[u] : make_uint4(0, 0, 0, 0);
        unsigned cl = 0, ch = 0;  // entries so far of classes 0-3 and 4-7, 8 bits each
        unsigned free = n >= 32 ? FULL : n > 0 ? (1u << n) - 1u : 0u;  // steps not taken
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const unsigned w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
          if (k0 + 8 * u >= gm) break;
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const unsigned en = (q & 1) ? w[q >> 1] >> 16 : w[q >> 1] & 0xffffu;
            const int sh = 8 * (en & 3);
            const unsigned cc = (en & 4) ? ch : cl, ci = cc + (1u << sh);
            int k = ((en - lane) & 7) + 8 * ((cc >> sh) & 255);
            if (8 * u + q < n) {
              cl = (en & 4) ? cl : ci;
              ch = (en & 4) ? ci : ch;
              if (k > 31 || !((free >> (k & 31)) & 1u)) k = 31 - __clz(free);
              free ^= 1u << k;
              row[k] = (unsigned short)en;
            }
          }
        }
#pragma unroll
        for (int k = 0; k < kOrd; k += 4) {
          if (k0 + k >= gm) break;
          const uint2 w = *reinterpret_cast<const uint2*>(row + k);
          dst[EXAMD_IDX(b0 + (size_t)((k0 + k) >> 2) * 32, nbrick, st)] = make_uint2(pad(w.x, n - k), pad(w.y, n - k - 2));
        }
      }
    }
    if (tid == 0) {
      const int n = cw[3];
      atomicMax(&A.lw[LW_LMAX], n);
      if (n > lk) {
        A.lcount[tile] = -1;
        A.fb[atomicAdd(&A.lw[LW_FBN], 1)] = tile;
      } else {
        A.lcount[tile] = total;
      }
    }
    return false;
  }

  // (4) write-back: home atoms -> Fown, halo copies -> P[slot]
  for (int t = tid; t < total; t += blockDim.x) {
    const int ci = code[t];
    const int lx = ci & 31, ly = (ci >> 5) & 31, lz = (ci >> 10) & 31;
    const int slot = ((lx == 0 || lx == EX - 1) ? 1 : 0) | ((ly == 0 || ly == EY - 1) ? 2 : 0) |
                     ((lz == 0 || lz == EZ - 1) ? 4 : 0);
    const int e = lx + EX * (ly + EY * lz);
    const int64_t g = gfirst[e] + (t - lstart[e]);
    if (FP64 || FIX) {
      double* F = slot == 0 ? (double*)A.Fown : (double*)A.P + (size_t)(slot - 1) * 3 * A.N;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double f;
        if (FIX) {
          // the sum, times 2^-sf: C 2^coarse + r, C the coarse word and r the rest of the 64 bits, a signed
          // number; as h 2^32 + l with |h| < 2^53, so that one rounding is left
          const int C = fa[(6 + c) * cap + t], sh = A.fx.coarse - 32;
          const int rh = (int)((unsigned)fa[(3 + c) * cap + t] - ((unsigned)C << sh));
          const long long h = ((long long)C << sh) + rh;
          const unsigned l = (unsigned)fa[c * cap + t];
          const double d = fma((double)h, 0x1p32, (double)l);
          f = (h | l) ? __hiloint2double(__double2hiint(d) - (A.fx.sf << 20), __double2loint(d)) : 0.0;
        } else {
          f = fd[c * cap + t];
        }
        F[EXAMD_IDX(c * A.N + g, 3 * A.N, st)] = f;
      }
    } else {
      float4* F = slot == 0 ? (float4*)A.Fown : (float4*)A.P + (size_t)(slot - 1) * A.N;
      if (MODE == kRedoBig || MODE == kListBig) {
        // this copy's output was written by the first pass and by this tile
        // only (a copy's slot pattern is unique to one tile)
        const float x = fr[t], y = fr[cap + t], z = fr[2 * cap + t];
        if (x != 0.f || y != 0.f || z != 0.f) {
          const int64_t gg = EXAMD_IDX(g, A.N, st);
          float4 v = F[gg];
          v.x += x;
          v.y += y;
          v.z += z;
          F[gg] = v;
        }
      } else {
        float f[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
          f[c] = MODE == kRedoFull ? fmaf((float)fa[3 * t + c], kFixInv, fr[c * cap + t])
                                   : (float)fa[3 * t + c] * kFixInv;
        F[EXAMD_IDX(g, A.N, st)] = make_float4(f[0], f[1], f[2], 0.f);
      }
    }
  }

  // (5) per-tile energy / virial / counters
  if (ENERGY || COUNT) {
    // mixed form: exact integer sums (the same bits whatever the order) and the
    // rare large terms' FP32 ones; FP64 form: FP64 sums.  Two sums share a warp's
    // exchange, and warp 0 adds up the warps' (one thread's loop over all of them
    // and unneeded sums were 6 % of a small-box ensemble's instructions).
    long long* redl = (long long*)red;
    double e = 0.0, w = 0.0;
    if (ENERGY) {
      if (FP64 || FIX) {
        e = esum;
        w = FIX ? wsum * A.fx.wunit : wsum;
      }
    }
    __syncthreads();  // the queues are done with
    if (ENERGY) {
      if (FP64 || FIX) {
        e = warp_sum2(e, w);
        if ((lane & 15) == 0) red[8 * warp + (lane >> 4)] = e;
      } else {
        const long long v = warp_sum2(ek.v, wk.v);
        if ((lane & 15) == 0) redl[8 * warp + 2 + (lane >> 4)] = v;
        if (__any_sync(FULL, ek.side != 0.f || wk.side != 0.f)) e = warp_sum2((double)ek.side, (double)wk.side);
        if ((lane & 15) == 0) red[8 * warp + (lane >> 4)] = e;
      }
    }
    if (COUNT) {
      const long long c1 = warp_sum((long long)ncand), c2 = warp_sum((long long)nacc), c3 = warp_sum((long long)neval);
      if (lane == 0) {
        redl[8 * warp + 4] = c1;
        redl[8 * warp + 5] = c2;
        redl[8 * warp + 6] = c3;
      }
    }
    __syncthreads();
    if (warp == 0) {
      const int k = min(lane, nw - 1);
      const bool on = lane < nw;
      if (ENERGY) {
        const double se = red[8 * k], sw = red[8 * k + 1];
        double t = 0.0;
        if (FP64 || FIX || __any_sync(FULL, se != 0.0 || sw != 0.0)) t = warp_sum2(on ? se : 0.0, on ? sw : 0.0);
        if (!(FP64 || FIX))
          t += (double)warp_sum2(on ? redl[8 * k + 2] : 0ll, on ? redl[8 * k + 3] : 0ll) * 0x1.0p-32;
        if (lane == 0) A.tileE[tile] = t;
        if (lane == 16) A.tileW[tile] = t;
      }
      if (COUNT)
        for (int c = 0; c < 3; ++c) {
          const long long n = warp_sum(on ? redl[8 * k + 4 + c] : 0ll);
          if (lane == 0) A.tileC[3 * tile + c] = n;
        }
    }
  }
  return false;
}

template <bool FP64, bool MULTI, bool ENERGY, bool COUNT>
__global__ void __launch_bounds__(256, FP64 ? 3 : 4) k_pair(const PairArgs A) {
  pair_tile<FP64, MULTI, ENERGY, COUNT, kMain>(A, A.order[blockIdx.x]);
}

// The mixed form's enumeration with kWideWarps warps per CTA, for grids that one
// wave of 3 CTAs per SM holds: an SM then has 2 or 3 CTAs however few warps they
// are, and 12 warps instead of 8 shorten each.
template <bool MULTI, bool ENERGY>
__global__ void __launch_bounds__(32 * kWideWarps, 3) k_pair_wide(const PairArgs A) {
  pair_tile<false, MULTI, ENERGY, false, kMain, true, kFineParts>(A, A.order[blockIdx.x]);
}

// FP64 form: the first pass in fixed point; a tile with a term too large for it by
// the FP64 body, in the same CTA: all of them in a system with overlapping atoms
// (131,072 atoms at random, density 0.5, no least distance: 376 us a pass, 352 by
// the FP64 body alone; 942 where such tiles were finished here first and then
// listed for k_pair_redo64, one CTA an SM).
template <bool MULTI, bool ENERGY, bool COUNT, int PARTS, bool OWNG>
__global__ void __launch_bounds__(256, MULTI ? 3 : 4) k_pair_fix(const PairArgs A) {
  const int tile = A.order[blockIdx.x];
  if (pair_tile<false, MULTI, ENERGY, COUNT, kFixed, true, PARTS, OWNG>(A, tile)) {
    __syncthreads();
    pair_tile<true, MULTI, ENERGY, COUNT, kMain>(A, tile);
  }
}

// Pair-list mode: the forces of every tile from its list (fallback tiles
// return at once: the redo pass enumerates them).
template <bool MULTI, bool ENERGY, bool CUT>
__global__ void __launch_bounds__(256, 4) k_pair_list(const PairArgs A) {
  pair_tile<false, MULTI, ENERGY, false, kList, CUT>(A, A.order[blockIdx.x]);
}

// Pair-list mode: the lists of every tile, on the steps whose gate is set.
template <bool MULTI>
__global__ void __launch_bounds__(32 * kBuildWarps, 3) k_pair_build(const PairArgs A) {
  if (A.gate && !*A.gate) return;
  pair_tile<false, MULTI, false, false, kListBuild>(A, A.order[blockIdx.x]);
}

// Mixed form: the redo pass over the tiles that k_pair listed (normally none,
// and the blocks return at once).  The block that finishes last empties the
// list: every block has read its length (a read that its loop and barrier
// depend on) before its thread 0 counts the block done.  LIST (pair-list
// mode): the listed tiles' large terms are redone from their lists, and the
// fallback tiles (over capacity or with lists that did not fit when they were
// built) are computed in full by enumeration, every step until the next build.
template <bool MULTI, bool ENERGY, bool COUNT, bool LIST>
__global__ void __launch_bounds__(256, 3) k_pair_redo(const PairArgs A) {
  grid_trigger();
  grid_wait();
  const int n = *(volatile const int*)A.redo_n;
  const int nfb = LIST ? *(volatile const int*)&A.lw[LW_FBN] : 0;
  for (int j = blockIdx.x; j < n + nfb; j += gridDim.x) {
    const int w = j < n ? A.redo[j] : (A.fb[j - n] | kFullBit);
    if (w & kFullBit)
      pair_tile<false, MULTI, ENERGY, COUNT, kRedoFull>(A, w & ~kFullBit);
    else if (LIST)
      pair_tile<false, MULTI, false, false, kListBig>(A, w);
    else
      pair_tile<false, MULTI, false, false, kRedoBig>(A, w);
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (atomicAdd(A.redo_done, 1u) == gridDim.x - 1) {
      *A.redo_n = 0;
      *A.redo_done = 0;
    }
  }
}

// FP64 form: the tiles over the first pass's capacity.
template <bool MULTI, bool ENERGY, bool COUNT>
__global__ void __launch_bounds__(256, 3) k_pair_redo64(const PairArgs A) {
  grid_trigger();
  grid_wait();
  const int n = *(volatile const int*)A.redo_n;
  for (int j = blockIdx.x; j < n; j += gridDim.x) {
    pair_tile<true, MULTI, ENERGY, COUNT, kRedoFull>(A, A.redo[j] & ~kFullBit);
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (atomicAdd(A.redo_done, 1u) == gridDim.x - 1) {
      *A.redo_n = 0;
      *A.redo_done = 0;
    }
  }
}

template <bool FP64, bool MULTI>
static void* pick_enum_ec(const PairConfig& c) {
  if (c.energy) return c.count ? (void*)&k_pair<FP64, MULTI, true, true> : (void*)&k_pair<FP64, MULTI, true, false>;
  return c.count ? (void*)&k_pair<FP64, MULTI, false, true> : (void*)&k_pair<FP64, MULTI, false, false>;
}

// The enumeration's first pass.
static void* pick_enum(const PairConfig& c) {
  if (c.fp64) return c.multi ? pick_enum_ec<true, true>(c) : pick_enum_ec<true, false>(c);
  return c.multi ? pick_enum_ec<false, true>(c) : pick_enum_ec<false, false>(c);
}

// The first pass: in pair-list mode (the counters excepted, which the
// enumeration counts) the list pass.
static bool uses_list(const PairConfig& c) { return c.list && !c.fp64 && !c.count; }

template <bool MULTI, bool OWNG>
static void* pick_fix(const PairConfig& c) {
  constexpr int P = kUnitParts, F = kFineParts;
  if (c.count)
    return c.energy ? (void*)&k_pair_fix<MULTI, true, true, P, OWNG> : (void*)&k_pair_fix<MULTI, false, true, P, OWNG>;
  if (c.fine)
    return c.energy ? (void*)&k_pair_fix<MULTI, true, false, F, OWNG> : (void*)&k_pair_fix<MULTI, false, false, F, OWNG>;
  return c.energy ? (void*)&k_pair_fix<MULTI, true, false, P, OWNG> : (void*)&k_pair_fix<MULTI, false, false, P, OWNG>;
}

template <bool MULTI>
static void* pick_redo64(const PairConfig& c) {
  if (c.energy) return c.count ? (void*)&k_pair_redo64<MULTI, true, true> : (void*)&k_pair_redo64<MULTI, true, false>;
  return c.count ? (void*)&k_pair_redo64<MULTI, false, true> : (void*)&k_pair_redo64<MULTI, false, false>;
}

static void* pick(const PairConfig& c) {
  if (uses_wide(c)) {
    if (c.multi) return c.energy ? (void*)&k_pair_wide<true, true> : (void*)&k_pair_wide<true, false>;
    return c.energy ? (void*)&k_pair_wide<false, true> : (void*)&k_pair_wide<false, false>;
  }
  if (c.fix) return c.multi ? pick_fix<true, false>(c) : c.own_global ? pick_fix<false, true>(c) : pick_fix<false, false>(c);
  if (uses_list(c)) {
    if (c.cut) {
      if (c.multi) return c.energy ? (void*)&k_pair_list<true, true, true> : (void*)&k_pair_list<true, false, true>;
      return c.energy ? (void*)&k_pair_list<false, true, true> : (void*)&k_pair_list<false, false, true>;
    }
    if (c.multi) return c.energy ? (void*)&k_pair_list<true, true, false> : (void*)&k_pair_list<true, false, false>;
    return c.energy ? (void*)&k_pair_list<false, true, false> : (void*)&k_pair_list<false, false, false>;
  }
  return pick_enum(c);
}

static void* pick_build(const PairConfig& c) {
  return c.multi ? (void*)&k_pair_build<true> : (void*)&k_pair_build<false>;
}

template <bool MULTI, bool LIST>
static void* pick_redo_ec(const PairConfig& c) {
  if (c.energy)
    return c.count ? (void*)&k_pair_redo<MULTI, true, true, LIST> : (void*)&k_pair_redo<MULTI, true, false, LIST>;
  return c.count ? (void*)&k_pair_redo<MULTI, false, true, LIST> : (void*)&k_pair_redo<MULTI, false, false, LIST>;
}

static void* pick_redo(const PairConfig& c) {
  if (c.fix) return c.multi ? pick_redo64<true>(c) : pick_redo64<false>(c);
  if (uses_list(c)) return c.multi ? pick_redo_ec<true, true>(c) : pick_redo_ec<false, true>(c);
  return c.multi ? pick_redo_ec<true, false>(c) : pick_redo_ec<false, false>(c);
}

cudaError_t pair_prepare(const PairConfig& cfg, int smem_bytes) {
  cudaError_t e = cudaFuncSetAttribute(pick(cfg), cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  if (e != cudaSuccess || (cfg.fp64 && !cfg.fix)) return e;
  e = cudaFuncSetAttribute(pick_redo(cfg), cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
  if (e != cudaSuccess || !uses_list(cfg)) return e;
  return cudaFuncSetAttribute(pick_build(cfg), cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
}

cudaError_t launch_pair(const PairConfig& cfg, const PairArgs& a, int ntiles, int smem_bytes, cudaStream_t st) {
  if (ntiles <= 0) return cudaSuccess;
  void* fn = pick(cfg);
  void* args[] = {(void*)&a};
  // smem_bytes (the larger of the passes' needs) bounds every launch
  const int main_smem = main_smem_bytes(cfg, a.cap, a.ne_max, a.ext_max);
  if (main_smem > smem_bytes) return cudaErrorInvalidValue;
  const int warps = uses_wide(cfg) ? kWideWarps : cfg.warps;
  // (the list pass follows a conditional graph node or the list build: launched plainly)
  const bool chain = cfg.chain && !uses_list(cfg);
  cudaError_t e = launch_chained_ptr(chain, fn, dim3(ntiles), dim3(32 * warps), args, (size_t)main_smem, st);
  if (e != cudaSuccess || (cfg.fp64 && !cfg.fix)) return e;
  // the redo pass: a few blocks per SM at most; nothing to do in a thermal system
  const int redo_smem = redo_smem_bytes(cfg, a.cap_redo, a.ne_max, a.ext_max);
  if (redo_smem > smem_bytes) return cudaErrorInvalidValue;
  return launch_chained_ptr(chain, pick_redo(cfg), dim3(std::min(ntiles, kRedoBlocks)), dim3(32 * cfg.warps), args,
                            (size_t)redo_smem, st);
}

cudaError_t launch_pair_build(const PairConfig& cfg, const PairArgs& a, int ntiles, int smem_bytes, cudaStream_t st) {
  if (ntiles <= 0) return cudaSuccess;
  void* args[] = {(void*)&a};
  const int smem = build_smem_bytes(cfg, a.cap, a.ne_max, a.ext_max);
  if (smem > smem_bytes) return cudaErrorInvalidValue;
  return cudaLaunchKernel(pick_build(cfg), dim3(ntiles), dim3(32 * kBuildWarps), args, (size_t)smem, st);
}

}  // namespace examd
