// api.cu -- the C ABI (include/examd_gb300.h): context, buffers, step
// sequencing, CUDA-graph capture of the step loop.
//
// Host-side counterpart of the reference's setup and driver sequence:
// exaMD_domain_create (SRC/exaMD_utils.f90:167-190), the neighbour-slot and
// midpoint tables (SRC/exaMD_partitioning.f90:783-798,
// SRC/exaMD_module.f90:276-346) and the timed force call (exaMD.f90:241-253).
// The METIS partition of blocks over ranks (SRC/exaMD_partitioning.f90:65-455)
// becomes a fixed partition of cells into CTA tiles.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"

using namespace examd;

namespace {

// The 63 (slot_a, slot_b) block-pair classes of the midpoint method, slot =
// (ii+1) + 3(jj+1) + 9(kk+1) + 1 with ii fastest, 14 = home.  This table is
// the ownership rule itself, so it is carried as the same data
// (SRC/exaMD_module.f90:282-344).
const int kMidpointTable[63][2] = {
    {14, 14}, {14, 15}, {14, 16}, {14, 17}, {14, 18}, {14, 19}, {14, 20}, {14, 21}, {14, 22},
    {14, 23}, {14, 24}, {14, 25}, {14, 26}, {14, 27}, {10, 18}, {10, 27}, {11, 17}, {11, 18},
    {11, 25}, {11, 26}, {11, 27}, {12, 16}, {12, 17}, {12, 25}, {13, 15}, {13, 18}, {13, 24},
    {13, 27}, {15, 16}, {15, 19}, {15, 22}, {15, 25}, {16, 21}, {16, 24}, {17, 19}, {17, 20},
    {17, 21}, {18, 19}, {19, 5},  {19, 9},  {20, 5},  {20, 7},  {20, 8},  {20, 9},  {21, 5},
    {21, 7},  {22, 5},  {22, 6},  {22, 9},  {23, 5},  {24, 5},  {24, 4},  {24, 7},  {25, 5},
    {25, 3},  {25, 6},  {26, 5},  {26, 2},  {26, 3},  {27, 1},  {27, 2},  {27, 4},  {27, 5}};

void slot_offset(int s, int o[3]) {  // SRC/exaMD_partitioning.f90:786-795
  s -= 1;
  o[0] = s % 3 - 1;
  o[1] = (s / 3) % 3 - 1;
  o[2] = s / 9 - 1;
}

bool class_ok(int cls, int h) {  // home offset h keeps the home cell inside the tile
  switch (cls) {
    case 0: return h == 1;   // halo cell before the tile
    case 1: return h >= 0;   // first cell
    case 2: return true;     // interior
    case 3: return h <= 0;   // last cell
    default: return h == -1; // halo cell after the tile
  }
}

// Derive the row structure and the per-class ownership masks from the table.
// Returns false if the table does not have the expected shape.
bool build_own_lut(OwnLut& L, signed char (*rowsOut)[2] = nullptr, unsigned char (*byRow)[kRows] = nullptr) {
  std::memset(&L, 0, sizeof(L));
  std::vector<std::pair<int, int>> rows;
  std::map<std::pair<int, int>, std::map<int, std::array<int, 3>>> byrow;
  for (int p = 1; p < 63; ++p) {
    int a[3], b[3];
    slot_offset(kMidpointTable[p][0], a);
    slot_offset(kMidpointTable[p][1], b);
    int d[3] = {b[0] - a[0], b[1] - a[1], b[2] - a[2]};
    auto key = std::make_pair(d[1], d[2]);
    if (!byrow.count(key) && key != std::make_pair(0, 0)) rows.push_back(key);
    if (byrow[key].count(d[0])) return false;  // duplicate separation
    byrow[key][d[0]] = {-a[0], -a[1], -a[2]};  // home = A - slot_a
  }
  if (rows.size() != 12 || byrow.size() != 13) return false;
  rows.push_back({0, 0});
  for (int r = 0; r < kRows; ++r) {
    if (rowsOut) {
      rowsOut[r][0] = (signed char)rows[r].first;
      rowsOut[r][1] = (signed char)rows[r].second;
    }
    const auto& m = byrow[rows[r]];
    if (r < 12) {
      if (m.size() != 5) return false;
    } else if (m.size() != 2 || !m.count(1) || !m.count(2)) {
      return false;
    }
  }
  for (int cx = 0; cx < 5; ++cx)
    for (int cy = 0; cy < 5; ++cy)
      for (int cz = 0; cz < 5; ++cz) {
        const int cls = cx * 25 + cy * 5 + cz;
        for (int r = 0; r < kRows; ++r) {
          unsigned mask = 0;
          for (const auto& kv : byrow[rows[r]]) {
            const auto& h = kv.second;
            if (class_ok(cx, h[0]) && class_ok(cy, h[1]) && class_ok(cz, h[2])) mask |= 1u << (kv.first + 2);
          }
          if (r == kRows - 1 && class_ok(cx, 0) && class_ok(cy, 0) && class_ok(cz, 0)) mask |= 1u << 2;
          if (byRow) byRow[cls][r] = (unsigned char)mask;
          if (mask)
            L.ent[cls][L.nrow[cls]++] =
                (unsigned short)(mask | ((unsigned)(rows[r].first + 2) << 5) | ((unsigned)(rows[r].second + 2) << 8) |
                                 (r == kRows - 1 ? 1u << 11 : 0u));
        }
      }
  return true;
}

int round_block_length(double want, double* out, int* q_out, int* k_out) {
  if (!(want > 0.0) || !std::isfinite(want)) return EXAMD_ERR_ARG;
  // largest k with ceil(want * 2^k) < 2^14: c * bl then needs <= 24 bits
  int k = 13 - (int)std::floor(std::log2(want));
  double bl = 0.0;
  for (; k > -60; --k) {
    double q = std::ceil(want * std::ldexp(1.0, k));
    if (q < 16384.0) {
      bl = std::ldexp(q, -k);
      *q_out = (int)q;
      *k_out = k;
      break;
    }
  }
  if (!(bl >= want)) return EXAMD_ERR_ARG;
  *out = bl;  // = q * 2^-k
  return EXAMD_OK;
}

// r at which |F(r)| = 24 eps (2 s^12 - s^6) / r, s = sigma / r, falls to fmax
// (it falls monotonically from r -> 0 to its zero at 2^(1/6) sigma), squared
// and widened by 1e-4, which covers the rounding of a pair's r^2 and force.
double r2_of_force(double eps, double sigma, double fmax) {
  auto fmag = [&](double rr) {
    const double s6 = std::pow(sigma / rr, 6.0);
    return 24.0 * eps * (2.0 * s6 * s6 - s6) / rr;
  };
  double lo = 1e-3 * sigma, hi = std::pow(2.0, 1.0 / 6.0) * sigma;
  if (!(fmag(lo) > fmax)) {
    hi = lo;
  } else {
    for (int it = 0; it < 200; ++it) {
      const double mid = 0.5 * (lo + hi);
      (fmag(mid) > fmax ? lo : hi) = mid;
    }
  }
  return hi * hi * (1.0 + 1e-4);
}

// x >= 0 in units of 2^ue, modulo 2^64; exact for an x of at least 2^(ue + 52).
long long fixed_of(double x, int ue) {
  int e = 0;
  const unsigned long long m = (unsigned long long)std::ldexp(std::frexp(x, &e), 53);
  const int sh = e - 53 - ue;
  return (long long)(sh < 0 || sh > 63 ? 0ull : m << sh);
}

// The tables of the FP64 form's fixed-point pass (pair.cu, force_batch_fix), or
// false where the parameters do not suit it and the FP64 body computes every
// tile: pairs whose force at their cutoff falls below 2^-13 of the largest force
// scale eps / sigma (the sums' one unit would hold it to fewer bits than FP64
// does), pairs so small beside the longest cutoff (sigma below about a sixth of
// it), whose square is below 2^62 units, that their r^2 has less than FP64's bits
// (RMS error of contact pairs at sigmas 1 : 8 was 8.6e-15 where FP64 has 1.1e-15), a
// cutoff inside the range of the forces too large for the sums, or lengths and
// energies whose powers leave FP64's range.
bool build_fix(const LJTable& lj, const examd_params& p, double bl, FixTable& fx) {
  const int n2 = lj.nt * lj.nt;
  double rmax = 0.0, f0max = 0.0, fweak = INFINITY;  // fweak: the weakest pair's force at its cutoff (by its terms' size)
  for (int k = 0; k < n2; ++k) {
    rmax = std::max(rmax, p.rc[k]);
    f0max = std::max(f0max, p.eps[k] / p.sigma[k]);
    const double s6 = std::pow(p.sigma[k] / p.rc[k], 6.0);
    fweak = std::min(fweak, 24.0 * p.eps[k] * (s6 + 2.0 * s6 * s6) / p.rc[k]);
  }
  if (!std::isnormal(f0max)) return false;
  int f0 = std::ilogb(f0max);  // F0 = 2^f0
  if (std::ldexp(1.0, f0) < f0max) ++f0;
  fx.ue = std::ilogb(rmax) + 1 - 62;  // every separation within the cutoff is below 2^62 units
  const FixUnit* unit = nullptr;
  for (const FixUnit& u : kFixUnits)
    if (!unit && fweak >= std::ldexp(1.0, f0 - u.weak)) unit = &u;
  if (!unit) return false;
  fx.sf = unit->bits - f0;
  fx.coarse = unit->coarse;
  fx.atoms = unit->atoms;
  const double fbig = std::ldexp(1.0, unit->term + f0);
  const int w = 2 * fx.ue + 64;  // r^2 = D 2^w
  double r2big[EXAMD_MAX_TYPES * EXAMD_MAX_TYPES];
  double gmax = 0.0;
  for (int k = 0; k < n2; ++k) {
    r2big[k] = std::max(r2_of_force(p.eps[k], p.sigma[k], fbig), 1.001e-12);  // coincident atoms (kR2Min64) as well
    gmax = std::max(gmax, fbig / std::sqrt(r2big[k]));
  }
  if (!std::isnormal(gmax)) return false;
  const int sg = 61 - std::ilogb(gmax);  // |dg| 2^sg < 2^62
  fx.k0 = sg - fx.ue - fx.sf;
  fx.wunit = std::ldexp(1.0, w - sg);
  if (!std::isnormal(fx.wunit)) return false;
  // (the coarse word is formed from the product's top word: a step is at least 2^4 of its units)
  if (fx.k0 + fx.coarse - 96 < 4 || fx.k0 > 63) return false;
  for (int k = 0; k < n2; ++k) {
    FixPair& q = fx.p[k];
    const long double s2 = (long double)lj.p64[k].sig2, s6 = s2 * s2 * s2, e = (long double)p.eps[k];
    q.c6 = (double)std::ldexp(24.0L * e * s6, sg - 4 * w);
    q.c12 = (double)std::ldexp(48.0L * e * s6 * s6, sg - 7 * w);
    q.s6 = (double)std::ldexp(s6, -3 * w);
    q.e4 = lj.p64[k].eps4;
    q.eshift = lj.p64[k].eshift;
    const double lim = std::ldexp(lj.p64[k].rcut2, -w), big = std::ldexp(r2big[k], -w);
    if (!std::isnormal(q.c6) || !std::isnormal(q.c12) || !std::isnormal(q.s6) || !(big >= 0x1.8p52) ||
        !(lim < 0x1p61) || !(big < lim))
      return false;
    q.limh = (int)((long long)lim >> 32);
    q.bigh = (int)((long long)big >> 32) + 1;
    // The prefilter's cutoff covers the FP32 separations' rounding: relative to it, and absolute, to the cell edge (x
    // from the tile's centre, up to 11 edges away, y and z from the atoms' own rows: 80 2^-24 edges in all)
    const double wide = p.rc[k] + 5e-6 * bl;
    q.pre = std::max(lj.p32[k].rc2 * 1.0001f, (float)(wide * wide * 1.000001));
  }
  return true;
}

// Split of one box axis of nb cells into tiles of at most tile_len cells (an
// even split: tile_len or tile_len - 1 cells), so that the largest staged
// tile, which sizes shared memory, stays (tile_len + 2)^3 cells; every tile
// keeps >= 2 cells.  balance = 1: a last cell at least 1.5 edges wide (it
// absorbs the remainder of L / edge) counts as two cells in the split, so the
// tile that holds it has one cell fewer.  Writes nt + 1 starts, returns nt.
int split_axis(int nb, double last_width, int tile_len, int balance, int* starts) {
  const int nv = nb + (balance == 1 && last_width >= 1.5 ? 1 : 0);
  const int nt = std::max(1, std::min(nb / 2, (nv + tile_len - 1) / tile_len));
  for (int k = 0; k < nt; ++k) starts[k] = (int)((int64_t)k * nv / nt);
  starts[nt] = nb;
  if (nt > 1 && starts[nt] - starts[nt - 1] < 2)  // keep >= 2 cells: the even split
    for (int k = 0; k <= nt; ++k) starts[k] = (int)((int64_t)k * nb / nt);
  return nt;
}

// Home cells per tile and axis where the caller leaves it to the library: 4.
// The FP64 form, whose tiles take longer and whose results do not depend on
// them, takes smaller ones where 4^3 would leave SMs idle: 3 below four tiles an
// SM, 2 where even 3^3 gives less than one.  (Pair pass at 4 / 3 / 2, us: 1,000
// atoms in 8 / 27 / 64 tiles 44.8 / 27.1 / 17.1; 8,788 in 125 / 216 / 512
// 46 / 35 / 31; 32,000 in 343 / 729 / 2197 63 / 47 / 56; 87,808 in 1000 / 2197
// 100 / 98.)  Also 3 where a tile of 4^3 is too large for three CTAs on an SM
// (about 820 atoms with the headroom; expected from the mean density, the wide
// last cell and three standard deviations): 1M liquid, 4^3 / 3^3: rc 3.0 1561 /
// 1309, 500k at rc 3.0 764 / 639; below it, rc 2.75 1000 / 1151, rc 2.5 844 / 1027;
// and 2 where one of 3^3 would have more atoms than the fixed-point pass takes at
// such cutoffs (1M at rc 5, 3^3 / 2^3: 59.3
// ms by the FP64 body / 10.7).
// The mixed form keeps 4: its FP32 x coordinates are the tile's.
int default_tile(const examd_params& p, int nboxes, const examd_box* boxes, double bl, int sms) {
  if (p.precision != EXAMD_FP64) return 4;
  auto tiles = [&](int t) {
    double n = 0.0;
    for (int b = 0; b < nboxes; ++b) {
      double v = 1.0;
      for (int a = 0; a < 3; ++a) v *= std::ceil(std::floor(boxes[b].L[a] / bl) / t);
      n += v;
    }
    return n;
  };
  double most[2] = {0.0, 0.0};  // staged by the largest tile of 3^3 and of 4^3 cells
  for (int b = 0; b < nboxes; ++b)
    for (int t = 3; t <= 4; ++t) {
      double atoms = (double)boxes[b].natoms;
      for (int a = 0; a < 3; ++a) {
        const double cells = boxes[b].L[a] / bl;
        atoms *= std::min(1.0, (t + 2 + (cells - std::floor(cells))) / cells);
      }
      most[t - 3] = std::max(most[t - 3], (atoms + 3.0 * std::sqrt(atoms)) * 1.0625 + 32.0);
    }
  int t = most[1] <= 820.0 ? 4 : 3;
  if (tiles(4) < 4.0 * sms) t = tiles(3) >= sms ? 3 : 2;
  return t == 3 && most[0] > kFixUnits[2].atoms ? 2 : t;
}

}  // namespace

int examd_tile_split(int nb, double last_width, int tile_len, int tile_balance, int* starts, int* nt) {
  if (!starts || !nt || nb < 1 || nb >= 1024 || tile_len < 1 || tile_balance < 0 || tile_balance > 1 ||
      !(last_width >= 1.0) || !(last_width < 2.0))
    return EXAMD_ERR_ARG;
  *nt = split_axis(nb, last_width, tile_len, tile_balance, starts);
  return EXAMD_OK;
}

constexpr int kIoChunks = 4;            // host <-> device transfers of the force call, in chunks
// Energies of eager steps kept on the device before one copy: this many steps of
// them, or as many as fit in kEagerBytes per array (one at least).
constexpr int kEagerSlots = 32;
constexpr size_t kEagerBytes = (size_t)4 << 20;
int eager_slots(int nboxes) {
  return (int)std::min<size_t>(kEagerSlots, std::max<size_t>(1, kEagerBytes / (sizeof(double) * (size_t)nboxes)));
}
// Force calls at new positions of at most this many atoms go through the
// context's own page-locked arrays (two host copies of up to 393 KB) from the
// third call on, so that they replay one captured graph whatever the caller's
// arrays are: 1,000 atoms cost 104 us as some twenty separate calls, the GPU
// idle between them.
constexpr int64_t kSmallIo = 1 << 14;
constexpr int64_t kHostTypes = 1 << 14;  // atoms whose types are checked by the host
constexpr int64_t kIoMinChunk = 1 << 16;  // atoms; smaller calls use fewer chunks

struct examd_ctx {
  examd_params p{};
  int nboxes = 0;
  std::vector<examd_box> boxes;
  std::vector<BoxDev> bh;
  std::vector<int> tile0;  // nboxes + 1
  std::vector<int64_t> atom0;
  int64_t N = 0;
  int NC = 0, ntiles = 0, ne_max = 0, ext_max = 0;
  double bl = 0.0;
  LJTable lj{};
  FixTable fx{};
  PairConfig pc;
  bool fix = false;     // the system has a fixed-point pass (pc.fix: the present capacities leave room for it)
  int cap = 0, smem = 0, smem_limit = 0, sm_smem = 0;
  int cap_redo = 0;     // staged-atom capacity of the redo pass
  bool whole_headroom = false;  // never half of it (see keep_headroom)
  int dev = 0;
  cudaStream_t st = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr, e2 = nullptr, e3 = nullptr;
  std::string lasterr;

  // device buffers
  BoxDev* d_boxes = nullptr;
  int4* d_tiles = nullptr;
  int* d_order = nullptr;  // pair-kernel launch order of the tiles
  int* d_tile0 = nullptr;
  unsigned char* d_bmask = nullptr;
  double* X[2][3] = {};
  double* V[2][3] = {};
  int* meta[2] = {};
  int* id[2] = {};
  int cur = 0;
  float4* U = nullptr;
  int* cellS = nullptr;
  int* cellOld = nullptr;
  int* slot = nullptr;
  int* count = nullptr;
  int* cstart = nullptr;
  int* bsum = nullptr;
  void* Fown = nullptr;
  void* P = nullptr;
  double* tileE = nullptr;
  double* tileW = nullptr;
  long long* tileC = nullptr;
  int* redo = nullptr;  // tiles for the redo pass (large pair-force terms)
  int* redo_n = nullptr;  // [0] count, [1] done counter of the redo pass
  double* boxE = nullptr;  // per box (graph chunk: [chunk][nboxes])
  double* boxW = nullptr;
  double* boxKE = nullptr;
  int* status = nullptr;
  int* d_occ = nullptr;
  double* stage = nullptr;   // 3N doubles (AoS I/O)
  double* stage2 = nullptr;  // 3N doubles
  int* d_meta_in = nullptr;
  double* d_factor = nullptr;
  int64_t* d_atom0 = nullptr;
  double* keAtom = nullptr;
  double* partial = nullptr;  // chunk partial sums of the per-box reductions
  int* h_status = nullptr;    // pinned host copies of the status word and, behind it, of d_occ
  // caller-order I/O in chunks, copies on a second stream
  int* inv = nullptr;         // caller index -> sorted slot
  bool inv_valid = false;     // inv matches the current sorted order
  cudaStream_t st2 = nullptr;
  cudaStream_t stc = nullptr;  // pair-list mode: captures the rebuild into a conditional node's body
  cudaEvent_t ev_io[3 * kIoChunks + 1] = {};
  int maxc_atoms = 1, maxc_tiles = 1;
  int ebuf_steps = 0;
  double* h_e = nullptr;      // pinned copies of boxKE and boxE (ebuf_steps + 1 steps each), for the runs with energies
  // a step's energy sums run on the second stream: the events that order them
  // (kick done, pair pass done; kinetic sums done, potential sums done), and
  // whether the last two are to be waited for
  cudaEvent_t ev_side[4] = {};
  bool side_ke = false, side_pe = false;

  bool in_call = false;  // the work of a force call is being queued
  bool atoms_set = false;
  bool forces_valid = false;  // Fown/P hold F(X[cur])
  bool energy_valid = false;

  // pair-list mode (examd_params.pair_skin > 0): the offsets Ub of the last
  // build, the per-tile lists (lslots staged atoms of lk entries each) and
  // their counts, the staged atoms per tile, the fallback tiles and the list
  // words (ListWord); list_gen counts the reallocations of the lists (a
  // captured graph names one generation)
  bool list = false;
  float disp_thr2 = 0.f;  // rebuild when an atom moved more than this squared
  float4* Ub = nullptr;
  unsigned short* plist = nullptr;
  unsigned short* plraw = nullptr;   // the build's scratch (each atom's entries in staged order)
  unsigned short* plperm = nullptr;  // the staged atoms in the order of their entry counts
  unsigned short* plcnt = nullptr;
  int lk = 0, lslots = 0, list_gen = 0;
  int* lcount = nullptr;
  int* fb = nullptr;
  int* lw = nullptr;
  int* h_lw = nullptr;  // pinned host copy of the list words
  int64_t host_builds = 0;  // builds the host asked for (the device counts the others)

  // graph cache
  cudaGraphExec_t gexec = nullptr;
  int g_parity = -1, g_chunk = 0, g_energy = -1, g_cap = 0, g_list_gen = 0;
  double g_dt = 0.0;
  // the force call at new positions (examd_gpu_forces_at) as a CUDA graph,
  // one per parity of the sort's double buffer, for a caller that passes the
  // same pinned buffers every time (an MD driver's arrays)
  struct IoGraph {
    cudaGraphExec_t exec = nullptr;
    const void *pos = nullptr, *forces = nullptr, *epot = nullptr, *virial = nullptr;
    int accumulate = -1, cap = 0, cap_redo = 0, list_gen = 0;
  } io_graph[2], small_graph[2][4];  // small calls: by parity, then energies | accumulate << 1
  int small_calls = 0;      // small calls so far, up to 2
  double* h_io = nullptr;   // small calls: positions, forces, energies, virials (pinned)

  int cuda_fail(cudaError_t e, const char* what) {
    lasterr = std::string(what) + ": " + cudaGetErrorString(e);
    return EXAMD_ERR_CUDA;
  }
};

#define CK(call)                                                    \
  do {                                                              \
    cudaError_t _e = (call);                                        \
    if (_e != cudaSuccess) return ctx->cuda_fail(_e, #call);        \
  } while (0)

namespace {

template <class T>
int dalloc(examd_ctx* ctx, T** p, size_t count) {
  if (count == 0) count = 1;
  cudaError_t e = cudaMalloc((void**)p, count * sizeof(T));
  if (e != cudaSuccess) {
    ctx->lasterr = std::string("cudaMalloc: ") + cudaGetErrorString(e);
    *p = nullptr;
    return EXAMD_ERR_NOMEM;
  }
  return EXAMD_OK;
}

// The captured force calls, dropped (the buffers they name change).
void drop_io_graphs(examd_ctx* ctx) {
  auto drop = [](examd_ctx::IoGraph& g) {
    if (g.exec) cudaGraphExecDestroy(g.exec);
    g = examd_ctx::IoGraph{};
  };
  for (int b = 0; b < 2; ++b) {
    drop(ctx->io_graph[b]);
    for (auto& g : ctx->small_graph[b]) drop(g);
  }
}

void free_all(examd_ctx* ctx) {
  if (ctx->gexec) cudaGraphExecDestroy(ctx->gexec);
  ctx->gexec = nullptr;
  drop_io_graphs(ctx);
  void* ptrs[] = {ctx->d_boxes, ctx->d_tiles, ctx->d_order, ctx->d_tile0, ctx->d_bmask, ctx->U, ctx->cellS,
                  ctx->cellOld, ctx->slot, ctx->count, ctx->cstart, ctx->bsum,
                  ctx->Fown, ctx->P, ctx->tileE, ctx->tileW, ctx->tileC, ctx->boxE, ctx->boxW, ctx->boxKE,
                  ctx->status, ctx->d_occ, ctx->stage, ctx->stage2, ctx->d_meta_in, ctx->d_factor,
                  ctx->d_atom0, ctx->keAtom, ctx->partial, ctx->redo, ctx->redo_n,
                  ctx->Ub, ctx->plist, ctx->plraw, ctx->plperm, ctx->plcnt, ctx->lcount, ctx->fb, ctx->lw};
  for (void* q : ptrs)
    if (q) cudaFree(q);
  for (int b = 0; b < 2; ++b) {
    for (int a = 0; a < 3; ++a) {
      if (ctx->X[b][a]) cudaFree(ctx->X[b][a]);
      if (ctx->V[b][a]) cudaFree(ctx->V[b][a]);
    }
    if (ctx->meta[b]) cudaFree(ctx->meta[b]);
    if (ctx->id[b]) cudaFree(ctx->id[b]);
  }
  if (ctx->h_status) cudaFreeHost(ctx->h_status);
  if (ctx->h_lw) cudaFreeHost(ctx->h_lw);
  if (ctx->h_e) cudaFreeHost(ctx->h_e);
  if (ctx->h_io) cudaFreeHost(ctx->h_io);
  for (cudaEvent_t e : ctx->ev_side)
    if (e) cudaEventDestroy(e);
  if (ctx->inv) cudaFree(ctx->inv);
  for (cudaEvent_t e : ctx->ev_io)
    if (e) cudaEventDestroy(e);
  if (ctx->st2) cudaStreamDestroy(ctx->st2);
  if (ctx->stc) cudaStreamDestroy(ctx->stc);
  if (ctx->e0) cudaEventDestroy(ctx->e0);
  if (ctx->e1) cudaEventDestroy(ctx->e1);
  if (ctx->e2) cudaEventDestroy(ctx->e2);
  if (ctx->e3) cudaEventDestroy(ctx->e3);
  if (ctx->st) cudaStreamDestroy(ctx->st);
}

int status_to_code(int st) {
  if (st & ST_TYPE) return EXAMD_ERR_ARG;
  if (st & ST_PAIRFN) return EXAMD_ERR_PAIRFN;
  if (st & ST_NONFINITE) return EXAMD_ERR_NONFINITE;
  if (st & ST_OUTSIDE) return EXAMD_ERR_OUTSIDE;
  if (st & ST_OVERFLOW) return EXAMD_ERR_CELL_OVERFLOW;
  if (st & ST_TIMEOUT) return EXAMD_ERR_TIMEOUT;
  if (st & ST_BOUNDS) return EXAMD_ERR_CHECK;
  return EXAMD_OK;
}

// Largest staged-atom count of any tile (ext cells), for the smem capacity.
__global__ void k_tile_occupancy(const int4* __restrict__ tiles, const BoxDev* __restrict__ boxes,
                                 const int* __restrict__ cstart, int* __restrict__ occ) {
  __shared__ int part[32];
  const int tile = blockIdx.x;
  const int4 t0 = tiles[2 * tile], t1 = tiles[2 * tile + 1];
  const BoxDev& B = boxes[t0.x];
  const int EX = t1.x + 2, EY = t1.y + 2, EZ = t1.z + 2, NE = EX * EY * EZ;
  int s = 0;
  for (int e = threadIdx.x; e < NE; e += blockDim.x) {
    int lx = e % EX, rr = e / EX, ly = rr % EY, lz = rr / EY;
    int g[3] = {t0.y + lx - 1, t0.z + ly - 1, t0.w + lz - 1};
    for (int a = 0; a < 3; ++a) {
      if (g[a] < 0) g[a] += B.nb[a];
      if (g[a] >= B.nb[a]) g[a] -= B.nb[a];
    }
    int gc = B.cell0 + g[0] + B.nb[0] * (g[1] + B.nb[1] * g[2]);
    s += cstart[gc + 1] - cstart[gc];
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += part[w];
    atomicMax(&occ[0], t);
  }
}

}  // namespace

// --------------------------------------------------------------------------
extern "C" {

void examd_default_params(examd_params* p) {
  std::memset(p, 0, sizeof(*p));
  p->precision = EXAMD_FP64;
  p->ntypes = 1;
  p->eps[0] = 1.0;
  p->sigma[0] = 1.0;
  p->rc[0] = 2.5;
  p->mass[0] = 1.0;
}

const char* examd_gpu_strerror(int code) {
  switch (code) {
    case EXAMD_OK: return "ok";
    case EXAMD_ERR_OUTSIDE: return "position outside the box (block number out of range)";
    case EXAMD_ERR_ARG: return "invalid argument or parameter";
    case EXAMD_ERR_NB_TOO_SMALL: return "fewer than 5 cells on an axis: the 63-entry table would count pairs twice";
    case EXAMD_ERR_CELL_OVERFLOW: return "a tile holds more atoms than its shared-memory capacity";
    case EXAMD_ERR_NONFINITE: return "non-finite position";
    case EXAMD_ERR_TIMEOUT: return "a bounded device wait gave up";
    case EXAMD_ERR_CUDA: return "CUDA runtime error";
    case EXAMD_ERR_NOMEM: return "out of device or pinned memory";
    case EXAMD_ERR_STATE: return "invalid call order";
    case EXAMD_ERR_NO_DEVICE: return "no usable sm_103 CUDA device";
    case EXAMD_ERR_IO: return "file missing, unreadable or malformed";
    case EXAMD_ERR_PAIRFN: return "the pair function returned an error (e.g. coincident atoms)";
    case EXAMD_ERR_CHECK: return "an index check of the checked build failed";
    default: return "unknown status";
  }
}

const char* examd_gpu_last_error(examd_ctx* ctx) { return ctx ? ctx->lasterr.c_str() : ""; }

int examd_own_table(signed char* rows, unsigned char* lut) {
  if (!rows || !lut) return EXAMD_ERR_ARG;
  OwnLut L;
  return build_own_lut(L, (signed char(*)[2])rows, (unsigned char(*)[kRows])lut) ? EXAMD_OK : EXAMD_ERR_ARG;
}

int examd_host_alloc(void** ptr, int64_t bytes) {
  if (!ptr || bytes < 0) return EXAMD_ERR_ARG;
  return cudaHostAlloc(ptr, (size_t)std::max<int64_t>(bytes, 1), cudaHostAllocDefault) == cudaSuccess
             ? EXAMD_OK
             : EXAMD_ERR_NOMEM;
}
int examd_host_free(void* ptr) { return cudaFreeHost(ptr) == cudaSuccess ? EXAMD_OK : EXAMD_ERR_CUDA; }

int examd_gpu_create(const examd_params* params, int nboxes, const examd_box* boxes, examd_ctx** out) {
  if (!params || !boxes || !out || nboxes < 1) return EXAMD_ERR_ARG;
  *out = nullptr;
  const examd_params& p = *params;
  if (p.ntypes < 1 || p.ntypes > EXAMD_MAX_TYPES) return EXAMD_ERR_ARG;
  if (p.precision != EXAMD_FP64 && p.precision != EXAMD_MIXED) return EXAMD_ERR_ARG;
  if (p.potential < EXAMD_POT_LJ || p.potential > EXAMD_POT_WCA) return EXAMD_ERR_ARG;
  const int nt = p.ntypes;
  double rcmax = 0.0;
  for (int a = 0; a < nt; ++a)
    for (int b = 0; b < nt; ++b) {
      const int k = a * nt + b, kt = b * nt + a;
      if (!(p.eps[k] > 0) || !(p.sigma[k] > 0) || !(p.rc[k] > 0)) return EXAMD_ERR_ARG;
      if (p.eps[k] != p.eps[kt] || p.sigma[k] != p.sigma[kt] || p.rc[k] != p.rc[kt]) return EXAMD_ERR_ARG;
      rcmax = std::max(rcmax, p.rc[k]);
    }
  // pair-list mode: the cells must hold every pair within rc + skin in the
  // 63-entry table's reach, so their edge is at least (rc + skin) / 2
  const double skin = p.pair_skin;
  if (!(skin >= 0.0) || !std::isfinite(skin) || (skin > 0.0 && p.precision != EXAMD_MIXED)) return EXAMD_ERR_ARG;
  if (skin > 0.0 && skin < 1e-3) return EXAMD_ERR_ARG;  // below the displacement test's margin
  if (p.pair_list_capacity < 0 || p.pair_list_capacity > 1024 || p.pair_list_capacity % 8 != 0) return EXAMD_ERR_ARG;
  const double reach = rcmax + skin;
  double want = p.cell_edge > 0 ? p.cell_edge : 0.5 * reach;
  if (want < 0.5 * reach) return EXAMD_ERR_ARG;
  double bl;
  int blq = 0, blk = 0;
  if (round_block_length(want, &bl, &blq, &blk) != EXAMD_OK) return EXAMD_ERR_ARG;

  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1 || p.device < 0 || p.device >= ndev)
    return EXAMD_ERR_NO_DEVICE;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, p.device) != cudaSuccess) return EXAMD_ERR_NO_DEVICE;
  if (prop.major != 10 || prop.minor != 3) return EXAMD_ERR_NO_DEVICE;  // built for sm_103a only

  examd_ctx* ctx = new examd_ctx();
  ctx->p = p;
  ctx->nboxes = nboxes;
  ctx->boxes.assign(boxes, boxes + nboxes);
  ctx->bl = bl;
  ctx->dev = p.device;
  ctx->smem_limit = (int)prop.sharedMemPerBlockOptin;
  ctx->sm_smem = (int)prop.sharedMemPerMultiprocessor;
  cudaSetDevice(ctx->dev);

  // pair-kernel configuration
  ctx->pc.fp64 = p.precision == EXAMD_FP64;
  ctx->pc.multi = nt > 1;
  ctx->pc.cut = p.potential == EXAMD_POT_WCA;
  if (p.pair_tables < 0 || p.pair_tables > 2 || p.tile_balance < 0 || p.tile_balance > 1) {
    delete ctx;
    return EXAMD_ERR_ARG;
  }
  ctx->list = skin > 0.0;
  ctx->pc.list = ctx->list;
  // an atom that moved d since the build is tested in FP32 against skin/2
  // less a margin of 1e-4 that covers the offsets' rounding many times over
  ctx->disp_thr2 = ctx->list ? (float)((0.5 * skin - 1e-4) * (0.5 * skin - 1e-4)) : 0.f;
  ctx->pc.warps = p.warps > 0 ? p.warps : 8;
  if (ctx->pc.warps < 4 || ctx->pc.warps > 8) {
    delete ctx;
    return EXAMD_ERR_ARG;
  }
  int T[3];
  const int deftile = default_tile(p, nboxes, boxes, bl, prop.multiProcessorCount);
  for (int a = 0; a < 3; ++a) {
    T[a] = p.tile[a] > 0 ? p.tile[a] : deftile;
    if (T[a] < 2 || T[a] > 14) {
      delete ctx;
      return EXAMD_ERR_ARG;
    }
  }

  // LJ tables
  LJTable& lj = ctx->lj;
  lj.nt = nt;
  float rc2max = 0.f;
  lj.pot = p.potential;
  for (int k = 0; k < nt * nt; ++k) {
    const double e = p.eps[k], s = p.sigma[k], r = p.rc[k];
    lj.p64[k].sig2 = s * s;      // sig2 = prmvdw(1,2)**2   (user_func.f90:59)
    lj.p64[k].eps24 = 24.0 * e;  // eps24 = twentyfour*eps  (user_func.f90:58)
    lj.p64[k].eps4 = 4.0 * e;
    lj.p64[k].rc2 = r * r;       // prmvdw(1,5)**2           (user_func.f90:52)
    // the potential's own range and energy shift
    double rcut2 = r * r, eshift = 0.0;
    if (p.potential == EXAMD_POT_LJ_SHIFTED) {
      const double s6 = std::pow(s * s / (r * r), 3);
      eshift = 4.0 * e * s6 * (s6 - 1.0);
    } else if (p.potential == EXAMD_POT_WCA) {
      rcut2 = std::cbrt(2.0) * s * s;  // (2^(1/6) sigma)^2
      eshift = -e;                     // U(2^(1/6) sigma) = -eps
      if (rcut2 > r * r) {  // rc must cover the potential's range
        delete ctx;
        return EXAMD_ERR_ARG;
      }
    }
    lj.p64[k].rcut2 = rcut2;
    lj.p64[k].eshift = eshift;
    lj.p32[k].sig2 = (float)(s * s);
    lj.p32[k].m24eps = (float)(-24.0 * e);
    lj.p32[k].c4eps = (float)(4.0 * e);
    lj.p32[k].rc2 = (float)(r * r);
    // the mixed form's own range test only where the potential ends inside
    // rc (WCA); for the LJ forms the range is rc itself, which the candidate
    // test decides, in FP64 at the border (an FP32 re-test there would drop
    // a pair that the FP64 form applies)
    lj.p32[k].rcut2 = p.potential == EXAMD_POT_WCA ? (float)rcut2 : INFINITY;
    lj.p32[k].eshift = (float)eshift;
    lj.p32[k].rl2 = (float)((r + skin) * (r + skin));
    // (not below kR2Min32, so that a pair-function error is found among the large terms)
    lj.p32[k].r2big = std::max((float)r2_of_force(e, s, kFixMaxForce), 1e-12f);
    rc2max = std::max(rc2max, lj.p32[k].rc2);
  }
  lj.rc2max = rc2max;
  // pair-list mode: atoms may be up to skin/2 outside the cells they were
  // sorted into, so an enumeration between builds prunes at rc + skin/2
  // The margin covers the rounding of the FP32 coordinates, at most 18 cell
  // edges from the tile's centre: 1e-4, or 2e-5 of the edge where lengths are large
  const double margin = std::max(1e-4, 2e-5 * bl), reach_now = rcmax + 0.5 * skin + margin;
  lj.prune2 = (float)(reach_now * reach_now);
  lj.prune2_list = (float)((reach + margin) * (reach + margin));
  for (int a = 0; a < EXAMD_MAX_TYPES; ++a) {
    double m = (a < nt && p.mass[a] > 0) ? p.mass[a] : 1.0;
    lj.mass[a] = m;
    lj.minv[a] = 1.0 / m;
  }

  // (in larger cells the prefilter would pass too many candidates)
  ctx->fix = ctx->pc.fix = ctx->pc.fp64 && bl <= 8.0 * rcmax && build_fix(lj, p, bl, ctx->fx);

  // Tiles of a batch: the tile edge T is the densest box's.  A box with fewer
  // atoms per cell gets tiles up to 2 cells longer per axis, as long as its
  // expected staged atoms, (T + 2 + g)^3 per cell times its atoms per cell,
  // stay within the densest box's (the largest tile sizes shared memory for
  // the whole launch): fewer halo cells per home cell, the same footprint.
  double dens_max = 0.0;
  std::vector<double> dens(nboxes, 0.0);
  for (int b = 0; b < nboxes; ++b) {
    double cells = 1.0;
    for (int a = 0; a < 3; ++a) cells *= std::max(1.0, std::floor(boxes[b].L[a] / bl));
    dens[b] = (double)boxes[b].natoms / cells;
    dens_max = std::max(dens_max, dens[b]);
  }

  // boxes, cells, tiles
  std::vector<int4> tiles;
  std::vector<unsigned char> bmask;
  int cell0 = 0;
  int64_t a0 = 0;
  for (int b = 0; b < nboxes; ++b) {
    const examd_box& X = boxes[b];
    BoxDev B{};
    if (X.natoms < 0) {
      delete ctx;
      return EXAMD_ERR_ARG;
    }
    for (int a = 0; a < 3; ++a) {
      if (!(X.L[a] > 0) || !std::isfinite(X.L[a])) {
        delete ctx;
        return EXAMD_ERR_ARG;
      }
      B.L[a] = X.L[a];
      B.Li[a] = 1.0 / X.L[a];  // globalboxi = one/globalbox (SRC/exaMD_utils.f90:188)
      B.Lf[a] = (float)X.L[a];
      double q = X.L[a] / bl;  // nblocks_xyz = Int(globalbox/block_length) (:179)
      if (q < 5.0) {
        delete ctx;
        return EXAMD_ERR_NB_TOO_SMALL;
      }
      if (q >= 1024.0) {
        delete ctx;
        return EXAMD_ERR_ARG;
      }
      B.nb[a] = (int)q;
    }
    if (ctx->pc.fix)
      for (int a = 0; a < 3; ++a) {
        const int e = std::ilogb(B.L[a]);
        B.Lq[a] = fixed_of(B.L[a], ctx->fx.ue);
        B.qbit[a] = e - 52 - ctx->fx.ue;  // >= 10: L is more than twice the cutoff
        const double over = std::ldexp(B.L[a] - std::ldexp(1.0, e), -ctx->fx.ue);
        B.qthr[a] = over < 0x1p62 ? (long long)over : (1ll << 62);
      }
    B.bl = bl;
    B.bli = 1.0 / bl;
    B.blq = blq;
    B.blk = blk;
    for (int a = 0; a < 3; ++a) B.remf[a] = (float)(B.L[a] - B.nb[a] * bl);  // nb*bl is exact
    B.blf = (float)bl;
    B.blif = (float)(1.0 / bl);
    B.cell0 = cell0;
    B.tile0 = (int)tiles.size() / 2;
    int Tb[3] = {T[0], T[1], T[2]};
    for (int g = 2; g > 0 && dens[b] > 0.0; --g) {
      const double grown = (double)(T[0] + 2 + g) * (T[1] + 2 + g) * (T[2] + 2 + g) * dens[b];
      if (grown <= (double)(T[0] + 2) * (T[1] + 2) * (T[2] + 2) * dens_max) {
        for (int a = 0; a < 3; ++a) Tb[a] = T[a] + g;
        break;
      }
    }
    int starts[3][1025];
    for (int a = 0; a < 3; ++a) {
      const double wide = (B.L[a] - (B.nb[a] - 1) * bl) / bl;  // the last cell's width in edges
      B.nt[a] = split_axis(B.nb[a], wide, Tb[a], p.tile_balance, starts[a]);
      for (int k = 0; k < B.nt[a]; ++k)
        if (starts[a][k + 1] - starts[a][k] + 2 > kMaxExt) {
          delete ctx;
          return EXAMD_ERR_ARG;
        }
    }
    ctx->tile0.push_back(B.tile0);
    for (int kz = 0; kz < B.nt[2]; ++kz)
      for (int ky = 0; ky < B.nt[1]; ++ky)
        for (int kx = 0; kx < B.nt[0]; ++kx) {
          int4 d0 = make_int4(b, starts[0][kx], starts[1][ky], starts[2][kz]);
          int4 d1 = make_int4(starts[0][kx + 1] - starts[0][kx], starts[1][ky + 1] - starts[1][ky],
                              starts[2][kz + 1] - starts[2][kz], 0);
          tiles.push_back(d0);
          tiles.push_back(d1);
          ctx->ne_max = std::max(ctx->ne_max, (d1.x + 2) * (d1.y + 2) * (d1.z + 2));
          ctx->ext_max = std::max(ctx->ext_max, std::max(d1.x, std::max(d1.y, d1.z)) + 2);
        }
    // boundary mask per cell: first or last cell of its tile on each axis
    std::vector<unsigned char> edge[3];
    for (int a = 0; a < 3; ++a) {
      edge[a].assign(B.nb[a], 0);
      for (int k = 0; k < B.nt[a]; ++k) {
        edge[a][starts[a][k]] = 1;
        edge[a][starts[a][k + 1] - 1] = 1;
      }
    }
    for (int cz = 0; cz < B.nb[2]; ++cz)
      for (int cy = 0; cy < B.nb[1]; ++cy)
        for (int cx = 0; cx < B.nb[0]; ++cx)
          bmask.push_back((unsigned char)(edge[0][cx] | (edge[1][cy] << 1) | (edge[2][cz] << 2)));
    cell0 += B.nb[0] * B.nb[1] * B.nb[2];
    ctx->atom0.push_back(a0);
    a0 += X.natoms;
    ctx->bh.push_back(B);
  }
  ctx->tile0.push_back((int)tiles.size() / 2);
  ctx->atom0.push_back(a0);
  ctx->N = a0;
  ctx->NC = cell0;
  ctx->ntiles = (int)tiles.size() / 2;
  ctx->pc.fine = ctx->ntiles <= 16 * prop.multiProcessorCount;  // about four waves
  // where the caller leaves the warps to the library and three CTAs an SM hold every tile
  ctx->pc.wide = p.warps <= 0 && !ctx->pc.fp64 && !ctx->list && ctx->ntiles <= 3 * prop.multiProcessorCount;
  if (ctx->N >= (int64_t)1 << 31 || (int64_t)cell0 >= ((int64_t)1 << 31) - 1 ||
      (cell0 + kScanTileHost - 1) / kScanTileHost > 8192 || nboxes >= (1 << 23)) {
    delete ctx;
    return EXAMD_ERR_ARG;
  }
  // Launch order of the pair kernel: the tiles by estimated cost, costliest
  // first, so that the grid ends on its cheapest CTAs (longest processing
  // time first; the per-tile outputs keep the tile's index).  The estimate is
  // the tile's staged atoms plus twice its home atoms times the atoms per cell
  // (its pair work), from cell volumes: the last cell of an axis is wider.
  std::vector<int> order(ctx->ntiles);
  {
    std::vector<double> cost(ctx->ntiles);
    for (int t = 0; t < ctx->ntiles; ++t) {
      const int4 d0 = tiles[2 * t], d1 = tiles[2 * t + 1];
      const BoxDev& B = ctx->bh[d0.x];
      const int org[3] = {d0.y, d0.z, d0.w}, len[3] = {d1.x, d1.y, d1.z};
      double vh = 1.0, ve = 1.0;
      for (int a = 0; a < 3; ++a) {
        const double wide = (B.L[a] - (B.nb[a] - 1) * B.bl) / B.bl;  // the last cell's width in cell edges
        double h = 0.0, e = 0.0;
        for (int c = org[a] - 1; c <= org[a] + len[a]; ++c) {
          const int g = (c + B.nb[a]) % B.nb[a];
          const double w = g == B.nb[a] - 1 ? wide : 1.0;
          e += w;
          if (c >= org[a] && c < org[a] + len[a]) h += w;
        }
        vh *= h;
        ve *= e;
      }
      const double n = (double)boxes[d0.x].natoms * B.bl * B.bl * B.bl / (B.L[0] * B.L[1] * B.L[2]);
      cost[t] = n * (ve + 2.0 * vh * n);
    }
    for (int t = 0; t < ctx->ntiles; ++t) order[t] = t;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cost[x] > cost[y]; });
  }

  OwnLut lut;
  if (!build_own_lut(lut)) {
    delete ctx;
    return EXAMD_ERR_ARG;
  }
  int rc = EXAMD_OK;
#define ALLOC(ptr, cnt)                                   \
  do {                                                    \
    if ((rc = dalloc(ctx, &(ptr), (cnt))) != EXAMD_OK) {  \
      free_all(ctx);                                      \
      delete ctx;                                         \
      return rc;                                          \
    }                                                     \
  } while (0)
  if (upload_own_lut(lut) != cudaSuccess || cudaStreamCreateWithFlags(&ctx->st, cudaStreamNonBlocking) != cudaSuccess ||
      cudaEventCreate(&ctx->e0) != cudaSuccess || cudaEventCreate(&ctx->e1) != cudaSuccess ||
      cudaEventCreate(&ctx->e2) != cudaSuccess || cudaEventCreate(&ctx->e3) != cudaSuccess) {
    free_all(ctx);
    delete ctx;
    return EXAMD_ERR_CUDA;
  }
  if (cudaHostAlloc((void**)&ctx->h_status, 2 * sizeof(int), cudaHostAllocDefault) != cudaSuccess) {
    ctx->h_status = nullptr;
    free_all(ctx);
    delete ctx;
    return EXAMD_ERR_NOMEM;
  }
  *ctx->h_status = 0;
  bool io_ok = cudaStreamCreateWithFlags(&ctx->st2, cudaStreamNonBlocking) == cudaSuccess &&
               cudaStreamCreateWithFlags(&ctx->stc, cudaStreamNonBlocking) == cudaSuccess;
  for (cudaEvent_t& e : ctx->ev_side) io_ok = io_ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  for (cudaEvent_t& e : ctx->ev_io) io_ok = io_ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
  if (!io_ok) {
    free_all(ctx);
    delete ctx;
    return EXAMD_ERR_CUDA;
  }
  const size_t N = (size_t)ctx->N, NC = (size_t)ctx->NC;
  ALLOC(ctx->d_boxes, nboxes);
  ALLOC(ctx->d_tiles, tiles.size());
  ALLOC(ctx->d_order, ctx->ntiles);
  ALLOC(ctx->d_tile0, nboxes + 1);
  ALLOC(ctx->d_bmask, NC);
  for (int b = 0; b < 2; ++b) {
    for (int a = 0; a < 3; ++a) {
      ALLOC(ctx->X[b][a], N);
      ALLOC(ctx->V[b][a], N);
    }
    ALLOC(ctx->meta[b], N);
    ALLOC(ctx->id[b], N);
  }
  ALLOC(ctx->U, N);
  ALLOC(ctx->cellS, N);
  ALLOC(ctx->cellOld, N);
  ALLOC(ctx->slot, N);
  ALLOC(ctx->count, NC);
  ALLOC(ctx->cstart, NC + 1);
  ALLOC(ctx->bsum, 8192);
  if (ctx->pc.fp64) {
    double* f;
    ALLOC(f, 3 * N);
    ctx->Fown = f;
    ALLOC(f, 7 * 3 * N);
    ctx->P = f;
  } else {
    float4* f;
    ALLOC(f, N);
    ctx->Fown = f;
    ALLOC(f, 7 * N);
    ctx->P = f;
  }
  ALLOC(ctx->redo, std::max(1, ctx->ntiles));
  ALLOC(ctx->redo_n, 2);
  ALLOC(ctx->tileE, ctx->ntiles);
  ALLOC(ctx->tileW, ctx->ntiles);
  ALLOC(ctx->tileC, 3 * (size_t)ctx->ntiles);
  ALLOC(ctx->boxE, nboxes);
  ALLOC(ctx->boxW, nboxes);
  ALLOC(ctx->boxKE, nboxes);
  ALLOC(ctx->status, 1);
  ALLOC(ctx->d_occ, 2);
  ALLOC(ctx->stage, 3 * N);
  ALLOC(ctx->stage2, 3 * N);
  ALLOC(ctx->d_meta_in, N);
  ALLOC(ctx->d_factor, nboxes);
  ALLOC(ctx->d_atom0, nboxes + 1);
  ALLOC(ctx->keAtom, N);
  ALLOC(ctx->inv, N);
  if (ctx->list) {
    ALLOC(ctx->Ub, N);
    ALLOC(ctx->lcount, ctx->ntiles);
    ALLOC(ctx->fb, ctx->ntiles);
    ALLOC(ctx->lw, LW_WORDS);
    if (cudaHostAlloc((void**)&ctx->h_lw, LW_WORDS * sizeof(int), cudaHostAllocDefault) != cudaSuccess) {
      ctx->h_lw = nullptr;
      free_all(ctx);
      delete ctx;
      return EXAMD_ERR_NOMEM;
    }
  }
  {
    int64_t maxa = 1, maxt = 1;
    for (int b = 0; b < nboxes; ++b) {
      maxa = std::max<int64_t>(maxa, ctx->atom0[b + 1] - ctx->atom0[b]);
      maxt = std::max<int64_t>(maxt, ctx->tile0[b + 1] - ctx->tile0[b]);
    }
    ctx->maxc_atoms = red_chunks(maxa);
    ctx->maxc_tiles = red_chunks(maxt);
    ALLOC(ctx->partial, std::max((size_t)nboxes * ctx->maxc_atoms, (size_t)2 * nboxes * ctx->maxc_tiles));
  }
#undef ALLOC
  cudaStream_t st = ctx->st;
  bool ok = cudaMemcpyAsync(ctx->d_boxes, ctx->bh.data(), nboxes * sizeof(BoxDev), cudaMemcpyHostToDevice, st) ==
                cudaSuccess &&
            cudaMemcpyAsync(ctx->d_tiles, tiles.data(), tiles.size() * sizeof(int4), cudaMemcpyHostToDevice, st) ==
                cudaSuccess &&
            cudaMemcpyAsync(ctx->d_order, order.data(), order.size() * sizeof(int), cudaMemcpyHostToDevice, st) ==
                cudaSuccess &&
            cudaMemcpyAsync(ctx->d_tile0, ctx->tile0.data(), (nboxes + 1) * sizeof(int), cudaMemcpyHostToDevice,
                            st) == cudaSuccess &&
            cudaMemcpyAsync(ctx->d_bmask, bmask.data(), NC, cudaMemcpyHostToDevice, st) == cudaSuccess &&
            cudaMemcpyAsync(ctx->d_atom0, ctx->atom0.data(), (nboxes + 1) * sizeof(int64_t),
                            cudaMemcpyHostToDevice, st) == cudaSuccess &&
            cudaMemsetAsync(ctx->count, 0, NC * sizeof(int), st) == cudaSuccess &&
            cudaMemsetAsync(ctx->status, 0, sizeof(int), st) == cudaSuccess &&
            (!ctx->redo_n || cudaMemsetAsync(ctx->redo_n, 0, 2 * sizeof(int), st) == cudaSuccess) &&
            (!ctx->lw || cudaMemsetAsync(ctx->lw, 0, LW_WORDS * sizeof(int), st) == cudaSuccess) &&
            cudaStreamSynchronize(st) == cudaSuccess;
  if (!ok) {
    free_all(ctx);
    delete ctx;
    return EXAMD_ERR_CUDA;
  }
  *out = ctx;
  return EXAMD_OK;
}

void examd_gpu_destroy(examd_ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->dev);
  if (ctx->st) cudaStreamSynchronize(ctx->st);
  free_all(ctx);
  delete ctx;
}

}  // extern "C"

// --------------------------------------------------------------------------
namespace {

struct InCall {  // marks the queueing of a force call (its launches are chained)
  examd_ctx* ctx;
  bool was;
  explicit InCall(examd_ctx* c) : ctx(c), was(c->in_call) { c->in_call = true; }
  ~InCall() { ctx->in_call = was; }
};

inline unsigned nblk(int64_t n, int t = 256) { return (unsigned)std::max<int64_t>(1, (n + t - 1) / t); }

// Scan and final ordering after a counting pass; swaps the buffers.
// want_inv: also record the caller -> sorted map (for the caller-order I/O).
// Pair-list mode: the sorted arrays are copied back into the current buffer
// (a step loop captured as a graph names fixed buffers, and whether a step
// rebuilds is decided on the device), the offsets are kept as the build's
// Ub, the caller map is always recorded, and gate (a device word, or
// nullptr) makes the whole sequence conditional.
int finish_binning(examd_ctx* ctx, bool want_inv, const int* gate = nullptr) {
  cudaStream_t st = ctx->st;
  const int nc = ctx->NC;
  const int nsb = (nc + kScanTileHost - 1) / kScanTileHost;
  const int s = ctx->cur, d = 1 - ctx->cur;
  const bool list = ctx->list;
  if (list) want_inv = true;
  const bool chain = ctx->in_call && !list;  // (in pair-list mode these may be the body of a conditional node)
  if (nsb > 1)  // (one block has none before it)
    CK(launch_chained(chain, k_scan_reduce, nsb, 256, st, nc, ctx->count, ctx->bsum, gate));
  CK(launch_chained(chain, k_scan_final, nsb, 256, st, nc, ctx->count, ctx->bsum, ctx->cstart, gate));
  if (ctx->N > 0) {
    CK(launch_chained(chain, k_finalize, nblk(ctx->N), 256, st, ctx->N, ctx->cellOld, ctx->slot, ctx->cstart,
                      ctx->d_boxes, ctx->X[s][0], ctx->X[s][1], ctx->X[s][2], ctx->V[s][0], ctx->V[s][1],
                      ctx->V[s][2], ctx->meta[s], ctx->id[s], ctx->X[d][0], ctx->X[d][1], ctx->X[d][2], ctx->V[d][0],
                      ctx->V[d][1], ctx->V[d][2], ctx->meta[d], ctx->id[d], ctx->U, list ? ctx->Ub : nullptr,
                      ctx->cellS, want_inv ? ctx->inv : nullptr, ctx->NC, ctx->status, gate));
    if (list)
      k_copy_back<<<nblk(ctx->N), 256, 0, st>>>(ctx->N, ctx->X[d][0], ctx->X[d][1], ctx->X[d][2], ctx->V[d][0],
                                                 ctx->V[d][1], ctx->V[d][2], ctx->meta[d], ctx->id[d], ctx->X[s][0],
                                                 ctx->X[s][1], ctx->X[s][2], ctx->V[s][0], ctx->V[s][1],
                                                 ctx->V[s][2], ctx->meta[s], ctx->id[s], gate);
  }
  CK(cudaGetLastError());
  if (!list) ctx->cur = d;
  ctx->inv_valid = want_inv;
  return EXAMD_OK;
}

// Chunk c of n atoms for the caller-order I/O: [i0, i1).
int io_chunks(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>(kIoChunks, n / kIoMinChunk)); }
void io_range(int64_t n, int nch, int c, int64_t& i0, int64_t& i1) {
  i0 = n * c / nch;
  i1 = n * (c + 1) / nch;
}

// The caller -> sorted map of the current order, if the last binning did not
// record it.
cudaError_t ensure_inv(examd_ctx* ctx) {
  if (ctx->inv_valid || ctx->N == 0) return cudaSuccess;
  k_inverse<<<nblk(ctx->N), 256, 0, ctx->st>>>(ctx->N, ctx->id[ctx->cur], ctx->inv);
  ctx->inv_valid = true;
  return cudaGetLastError();
}

// The status word after work already synchronised: its copy to the pinned
// host word was queued before that synchronisation (queue_status).
int take_status(examd_ctx* ctx) {
  const int h = *ctx->h_status;
  if (h) {
    CK(cudaMemsetAsync(ctx->status, 0, sizeof(int), ctx->st));
    CK(cudaStreamSynchronize(ctx->st));
  }
  return status_to_code(h);
}

cudaError_t queue_status(examd_ctx* ctx) {
  return cudaMemcpyAsync(ctx->h_status, ctx->status, sizeof(int), cudaMemcpyDeviceToHost, ctx->st);
}

int check_status(examd_ctx* ctx) {
  CK(queue_status(ctx));
  CK(cudaStreamSynchronize(ctx->st));
  return take_status(ctx);
}

// Staged-atom capacities of a tile from the current binning: +25% + 64
// headroom for the redo pass and for the FP64 form without one (no fixed-point
// pass); +6% + 32 for a first pass with a redo pass behind it (a tile that
// outgrows it before the next update is computed in full by the redo pass, at
// the redo capacity).  In two parts, so that a run waits once per chunk: the
// occupancy queued to its pinned word, and the capacities from it.
int queue_occupancy(examd_ctx* ctx) {
  CK(cudaMemsetAsync(ctx->d_occ, 0, 2 * sizeof(int), ctx->st));
  k_tile_occupancy<<<ctx->ntiles, 128, 0, ctx->st>>>(ctx->d_tiles, ctx->d_boxes, ctx->cstart, ctx->d_occ);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(ctx->h_status + 1, ctx->d_occ, sizeof(int), cudaMemcpyDeviceToHost, ctx->st));
  return EXAMD_OK;
}

int apply_capacity(examd_ctx* ctx, bool* grew = nullptr) {
  if (grew) *grew = false;
  const int occ = ctx->h_status[1];
  PairConfig pc = ctx->pc;  // (the context changes only once a choice fits)
  int cap = 0, redo = 0, bytes = 0;
  auto fits = [&] {
    pc.own_global = pair_own_global(pc, cap, ctx->ne_max, ctx->ext_max, ctx->sm_smem);
    bytes = pair_smem_bytes(pc, cap, redo, ctx->ne_max, ctx->ext_max);
    return bytes <= ctx->smem_limit && (!pc.fix || cap <= ctx->fx.atoms);
  };
  auto up8 = [](int n) { return (n + 7) & ~7; };
  auto headroom = [&] {  // not below what the same pass has now
    redo = std::max(up8(occ + occ / 4 + 64), pc.fix == ctx->pc.fix ? ctx->cap_redo : 0);
    cap = pc.fp64 && !pc.fix ? redo : up8(occ + occ / 16 + 32);
    // The fixed-point pass (78 bytes an atom) with half the headroom where the whole of it costs a CTA per SM (1M
    // liquid 949 -> 844 us a pass, 500k at rc 3.0 719 -> 639)
    if (pc.fix && !ctx->whole_headroom) {
      pc.own_global = !pc.multi;
      const int least = up8(occ + occ / 32 + 16);
      const int n = pair_ctas(pc, least, ctx->ne_max, ctx->ext_max, ctx->sm_smem);
      while (cap > least && pair_ctas(pc, cap, ctx->ne_max, ctx->ext_max, ctx->sm_smem) < n) cap -= 8;
    }
    return fits();
  };
  auto exact = [&] {
    cap = redo = up8(occ);
    return fits();
  };
  // (the redo pass binds, or the fixed-point pass: the 12-warp CTAs' tables never do)
  pc.fix = ctx->fix;
  bool ok = headroom();
  if (pc.fix == ctx->pc.fix) {
    if (cap <= ctx->cap) return EXAMD_OK;
    ok = ok || exact();
  }
  if (!ok && pc.fix) {
    // The FP64 body has smaller tables; it takes every tile as long as the fixed-point pass does not fit the largest
    // with its headroom
    pc.fix = false;
    ok = headroom();
    if (!ctx->pc.fix && cap <= ctx->cap) return EXAMD_OK;
    ok = ok || exact();
  }
  if (!ok) return EXAMD_ERR_CELL_OVERFLOW;
  if (pc.fix == ctx->pc.fix && cap == ctx->cap && redo == ctx->cap_redo) return EXAMD_OK;
  // all variants used by this context (the attribute is the kernel's, shared
  // with every other context of the process: the device's limit, so that none
  // takes away what another needs)
  for (int e = 0; e < 2; ++e)
    for (int n = 0; n < 2; ++n) {
      pc.energy = e;
      pc.count = n;
      CK(pair_prepare(pc, ctx->smem_limit));
    }
  ctx->pc.fix = pc.fix;
  ctx->pc.own_global = pc.own_global;
  ctx->cap = cap;
  ctx->cap_redo = redo;
  ctx->smem = bytes;
  if (ctx->gexec) cudaGraphExecDestroy(ctx->gexec);
  ctx->gexec = nullptr;
  drop_io_graphs(ctx);
  if (grew) *grew = true;
  return EXAMD_OK;
}

PairArgs pair_args(examd_ctx* ctx) {
  PairArgs a{};
  a.tiles = ctx->d_tiles;
  a.order = ctx->d_order;
  a.boxes = ctx->d_boxes;
  a.cstart = ctx->cstart;
  a.U = ctx->U;
  a.X0 = ctx->X[ctx->cur][0];
  a.X1 = ctx->X[ctx->cur][1];
  a.X2 = ctx->X[ctx->cur][2];
  a.Fown = ctx->Fown;
  a.P = ctx->P;
  a.N = ctx->N;
  a.tileE = ctx->tileE;
  a.tileW = ctx->tileW;
  a.tileC = ctx->tileC;
  a.status = ctx->status;
  a.cap = ctx->cap;
  a.cap_redo = ctx->cap_redo;
  a.ne_max = ctx->ne_max;
  a.ext_max = ctx->ext_max;
  a.lj = ctx->lj;
  a.fx = ctx->fx;
  a.redo = ctx->redo;
  a.redo_n = ctx->redo_n;
  a.redo_done = (unsigned*)(ctx->redo_n + 1);
  a.list = ctx->plist;
  a.lraw = ctx->plraw;
  a.lperm = ctx->plperm;
  a.lcnt = ctx->plcnt;
  a.lcount = ctx->lcount;
  a.lk = ctx->lk;
  a.lslots = ctx->lslots;
  a.ntiles = ctx->ntiles;
  a.fb = ctx->fb;
  a.lw = ctx->lw;
  a.gate = nullptr;
  return a;
}

// Pair-list mode: the lists of every tile at the current cells.  gate: a
// device word that makes the build conditional (eager steps), or nullptr:
// build now, with the fallback list emptied first (host: a build the host
// asked for, counted here; otherwise the body of a captured rebuild, which
// the device counts).
int build_lists(examd_ctx* ctx, const int* gate, bool host = true) {
  if (!gate) CK(cudaMemsetAsync(ctx->lw + LW_FBN, 0, sizeof(int), ctx->st));
  if (!gate && host) ++ctx->host_builds;
  PairArgs a = pair_args(ctx);
  a.gate = gate;
  CK(launch_pair_build(ctx->pc, a, ctx->ntiles, ctx->smem, ctx->st));
  return EXAMD_OK;
}

// Pair-list mode: cells and lists rebuilt at the current positions (gate and
// host as for build_lists).
int rebuild(examd_ctx* ctx, const int* gate, bool host = true) {
  const int s = ctx->cur;
  if (ctx->N > 0) {
    k_bin_count<<<nblk(ctx->N), 256, 0, ctx->st>>>(ctx->N, ctx->X[s][0], ctx->X[s][1], ctx->X[s][2],
                                                    ctx->meta[s], ctx->d_boxes, ctx->cellOld, ctx->slot,
                                                    ctx->count, ctx->status, gate);
    CK(cudaGetLastError());
  }
  const int rc = finish_binning(ctx, true, gate);
  return rc ? rc : build_lists(ctx, gate, host);
}

// Pair-list mode, after new positions: the device decides whether some atom
// moved more than half the skin since the build (or a rebuild was asked
// for).  Eager, the rebuild's kernels run or return at once on that
// decision.  Under stream capture (the step loop's graphs, the captured
// force call) the rebuild is captured, ungated, as the body of a conditional
// graph node whose value the decision sets, so a step without a rebuild
// launches none of its kernels.
int maybe_rebuild(examd_ctx* ctx) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  CK(cudaStreamIsCapturing(ctx->st, &cs));
  if (cs != cudaStreamCaptureStatusActive) {
    k_list_decide<<<1, 1, 0, ctx->st>>>(ctx->lw, ctx->disp_thr2, cudaGraphConditionalHandle{}, 0);
    CK(cudaGetLastError());
    return rebuild(ctx, ctx->lw + LW_GATE);
  }
  cudaGraph_t g = nullptr;
  const cudaGraphNode_t* deps = nullptr;
  const cudaGraphEdgeData* edges = nullptr;
  size_t nd = 0;
  CK(cudaStreamGetCaptureInfo(ctx->st, &cs, nullptr, &g, &deps, &edges, &nd));
  cudaGraphConditionalHandle h;
  CK(cudaGraphConditionalHandleCreate(&h, g, 0, cudaGraphCondAssignDefault));
  k_list_decide<<<1, 1, 0, ctx->st>>>(ctx->lw, ctx->disp_thr2, h, 1);
  CK(cudaGetLastError());
  CK(cudaStreamGetCaptureInfo(ctx->st, &cs, nullptr, &g, &deps, &edges, &nd));
  cudaGraphNodeParams np{};
  np.type = cudaGraphNodeTypeConditional;
  np.conditional.handle = h;
  np.conditional.type = cudaGraphCondTypeIf;
  np.conditional.size = 1;
  cudaGraphNode_t node;
  CK(cudaGraphAddNode(&node, g, deps, edges, nd, &np));
  CK(cudaStreamUpdateCaptureDependencies(ctx->st, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
  // the body: the rebuild's kernels, captured from a stream of their own
  cudaGraph_t body = np.conditional.phGraph_out[0];
  CK(cudaStreamBeginCaptureToGraph(ctx->stc, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
  cudaStream_t main = ctx->st;
  ctx->st = ctx->stc;
  const int rc = rebuild(ctx, nullptr, false);
  ctx->st = main;
  cudaGraph_t captured = nullptr;
  const cudaError_t ce = cudaStreamEndCapture(ctx->stc, &captured);
  if (rc) return rc;
  if (ce != cudaSuccess) return ctx->cuda_fail(ce, "cudaStreamEndCapture (rebuild body)");
  return EXAMD_OK;
}

// Pair-list mode: lists of `want` entries per staged atom, for the current
// staged-atom capacity.  The captured graphs name the old lists, so they are
// dropped.
int set_list_capacity(examd_ctx* ctx, int want) {
  const int slots = (ctx->cap + 31) & ~31;
  if (want == ctx->lk && slots == ctx->lslots && ctx->plist) return EXAMD_OK;
  CK(cudaStreamSynchronize(ctx->st));
  for (unsigned short** q : {&ctx->plist, &ctx->plraw, &ctx->plperm, &ctx->plcnt}) {
    if (*q) cudaFree(*q);
    *q = nullptr;
  }
  ctx->lk = ctx->lslots = 0;
  const size_t atoms = (size_t)ctx->ntiles * (size_t)slots;
  int rc;
  if ((rc = dalloc(ctx, &ctx->plist, atoms * (size_t)want)) || (rc = dalloc(ctx, &ctx->plraw, atoms * (size_t)want)) ||
      (rc = dalloc(ctx, &ctx->plperm, atoms)) || (rc = dalloc(ctx, &ctx->plcnt, atoms)))
    return rc;
  ctx->lk = want;
  ctx->lslots = slots;
  ++ctx->list_gen;
  if (ctx->gexec) {
    cudaGraphExecDestroy(ctx->gexec);
    ctx->gexec = nullptr;
  }
  drop_io_graphs(ctx);
  return EXAMD_OK;
}

// Pair-list mode: the list words, read after the stream's work; the longest
// list since the last read is reset.
int queue_list_words(examd_ctx* ctx) {
  CK(cudaMemcpyAsync(ctx->h_lw, ctx->lw, LW_WORDS * sizeof(int), cudaMemcpyDeviceToHost, ctx->st));
  CK(cudaMemsetAsync(ctx->lw + LW_LMAX, 0, sizeof(int), ctx->st));
  return EXAMD_OK;
}

int read_list_words(examd_ctx* ctx) {
  const int rc = queue_list_words(ctx);
  if (rc) return rc;
  CK(cudaStreamSynchronize(ctx->st));
  return EXAMD_OK;
}

// entries per atom: a multiple of 8 (a list pass reads eight at a time), at
// most 1024 (the list pass's count histogram)
int list_capacity_for(int longest) { return std::min(((longest + longest / 5 + 8) + 7) & ~7, 1024); }

// Pair-list mode, after a binning with the atoms in their cells: the lists
// built now at a capacity that fits the atom with the most entries, with 20 %
// headroom (the first build at an estimate from the densest box: 1.6 times
// the pairs in half a sphere of radius rc + skin).
int init_lists(examd_ctx* ctx) {
  if (ctx->p.pair_list_capacity > 0) {  // the caller's capacity, never resized
    const int rc = set_list_capacity(ctx, ctx->p.pair_list_capacity);
    return rc ? rc : build_lists(ctx, nullptr);
  }
  if (!ctx->plist) {
    double rho = 0.0, reach = 0.0;
    for (int b = 0; b < ctx->nboxes; ++b)
      rho = std::max(rho, (double)ctx->boxes[b].natoms / (ctx->boxes[b].L[0] * ctx->boxes[b].L[1] * ctx->boxes[b].L[2]));
    for (int k = 0; k < ctx->lj.nt * ctx->lj.nt; ++k) reach = std::max(reach, std::sqrt((double)ctx->lj.p32[k].rl2));
    const double est = 1.6 * (2.0943951 * reach * reach * reach * rho) + 16.0;
    const int rc = set_list_capacity(ctx, list_capacity_for((int)std::min(est, 4096.0)));
    if (rc) return rc;
  } else {
    const int rc = set_list_capacity(ctx, ctx->lk);  // new slots if the staged-atom capacity grew
    if (rc) return rc;
  }
  for (int it = 0; it < 4; ++it) {
    int rc = build_lists(ctx, nullptr);
    if (rc) return rc;
    rc = read_list_words(ctx);
    if (rc) return rc;
    const int longest = ctx->h_lw[LW_LMAX];
    const int want = list_capacity_for(longest);
    if (longest <= ctx->lk && ctx->lk <= 2 * want) return EXAMD_OK;
    rc = set_list_capacity(ctx, want);  // grow to fit, or shrink an estimate far too large
    if (rc) return rc;
  }
  return EXAMD_OK;  // any tile still over its list is computed by enumeration
}

int run_pair(examd_ctx* ctx, bool energy, bool count, double* boxE = nullptr, double* boxW = nullptr,
             bool side = false, bool sums = true);

// Pair-list mode, between runs of steps: a tile with an atom whose list
// outgrew its capacity since the last check, or with more staged atoms than
// the lists have slots, is computed by enumeration meanwhile.  The lists get
// room for it: new lists, which a build at the current positions fills, after
// a fresh sort (a build needs every atom inside its cell), and the forces
// again in the new order.  A staged-atom capacity that grew within the slots
// makes the next step rebuild, so that the tiles over the old one get lists.
// (h_lw holds the list words.)
int update_lists(examd_ctx* ctx, bool cap_grew) {
  int rc;
  const int longest = ctx->h_lw[LW_LMAX];
  const bool fixed = ctx->p.pair_list_capacity > 0;
  const int want = fixed ? ctx->lk : std::max(ctx->lk, list_capacity_for(longest));
  if (want != ctx->lk || ctx->cap > ctx->lslots) {
    if ((rc = set_list_capacity(ctx, want)) || (rc = rebuild(ctx, nullptr)) || (rc = run_pair(ctx, false, false)))
      return rc;
    return read_list_words(ctx);
  }
  if (cap_grew) {
    const int one = 1;
    CK(cudaMemcpyAsync(ctx->lw + LW_FORCE, &one, sizeof(int), cudaMemcpyHostToDevice, ctx->st));
    CK(cudaStreamSynchronize(ctx->st));
  }
  return EXAMD_OK;
}

// The pair pass; with energy the per-box sums to boxE, boxW (nullptr: the
// context's), on the second stream for a step of a loop (side); sums = false
// leaves them to the caller.
int run_pair(examd_ctx* ctx, bool energy, bool count, double* boxE, double* boxW, bool side, bool sums) {
  PairConfig c = ctx->pc;
  c.energy = energy;
  c.count = count;
  c.chain = ctx->in_call || !(c.wide || side);
  if (ctx->side_pe) {  // the last step's sums read the tile energies that this pass writes
    CK(cudaStreamWaitEvent(ctx->st, ctx->ev_side[3], 0));
    ctx->side_pe = false;
  }
  CK(launch_pair(c, pair_args(ctx), ctx->ntiles, ctx->smem, ctx->st));
  if (!energy || !sums) return EXAMD_OK;
  cudaStream_t to = side ? ctx->st2 : ctx->st;
  if (side) {
    CK(cudaEventRecord(ctx->ev_side[1], ctx->st));
    CK(cudaStreamWaitEvent(to, ctx->ev_side[1], 0));
  }
  CK(launch_reduce_tiles(ctx->nboxes, ctx->d_tile0, ctx->maxc_tiles, ctx->tileE, ctx->tileW, ctx->partial,
                         boxE ? boxE : ctx->boxE, boxW ? boxW : ctx->boxW, to));
  if (side) {
    CK(cudaEventRecord(ctx->ev_side[3], to));
    ctx->side_pe = true;
  }
  return EXAMD_OK;
}

// The first stream waits for the energy sums queued on the second one.
int join_side(examd_ctx* ctx) {
  if (ctx->side_ke) CK(cudaStreamWaitEvent(ctx->st, ctx->ev_side[2], 0));
  if (ctx->side_pe) CK(cudaStreamWaitEvent(ctx->st, ctx->ev_side[3], 0));
  ctx->side_ke = ctx->side_pe = false;
  return EXAMD_OK;
}

StepArgs step_args(examd_ctx* ctx) {
  StepArgs s{};
  s.boxes = ctx->d_boxes;
  s.bmask = ctx->d_bmask;
  s.cellS = ctx->cellS;
  s.Fown = ctx->Fown;
  s.P = ctx->P;
  s.N = ctx->N;
  s.fp64 = ctx->pc.fp64;
  s.nc = ctx->NC;
  s.status = ctx->status;
  return s;
}

cudaPointerAttributes attributes(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();  // clear the sticky-free error of an unknown pointer
    a.type = cudaMemoryTypeUnregistered;
  }
  return a;
}

// Whether the kernels can use the caller's array of n doubles in place: its
// first and its last byte page-locked host memory at the same address on the
// device (part of an array may be registered), and doubles on their boundary.
bool in_place(const void* p, size_t n) {
  if (!p || n == 0 || reinterpret_cast<uintptr_t>(p) % sizeof(double)) return false;
  for (const char* q : {(const char*)p, (const char*)p + n * sizeof(double) - 1}) {
    const cudaPointerAttributes a = attributes(q);
    if (a.type != cudaMemoryTypeHost || a.devicePointer != q) return false;
  }
  return true;
}

bool pinned(const void* p, size_t n) { return !p || in_place(p, n); }

bool on_device(const void* p) { return p && attributes(p).type == cudaMemoryTypeDevice; }

// The pair path at the resident positions, then the forces to the caller.  A
// page-locked array of the caller is read and written across the link by the
// kernels themselves (at the copy engines' rate, 0.2 TB/s each way): no staging
// copy, no chunks, and their events between two kernels.  Other arrays in
// chunks of the caller's order: the device->host copy of chunk c (second stream)
// overlaps the gather of chunk c + 1.  With accumulate, the caller's forces
// come in on the second stream while the pair kernel runs.
// The work of the force call, queued on the context's streams; the second
// stream rejoins the first at the end (so the sequence can be captured).
int enqueue_forces(examd_ctx* ctx, double* forces, double* epot, double* virial, int accumulate) {
  const InCall in_call(ctx);
  cudaStream_t st = ctx->st, st2 = ctx->st2;
  const bool energy = epot || virial;
  const int64_t N = ctx->N;
  const int nch = io_chunks(N);
  cudaEvent_t* ev_acc = ctx->ev_io + 2 * kIoChunks;
  double* const df = in_place(forces, 3 * (size_t)N) ? forces : nullptr;
  if (forces && accumulate && N > 0 && !df) {
    CK(cudaEventRecord(ctx->ev_io[3 * kIoChunks], st));  // stage is free once earlier work is done
    CK(cudaStreamWaitEvent(st2, ctx->ev_io[3 * kIoChunks], 0));
    for (int c = 0; c < nch; ++c) {
      int64_t i0, i1;
      io_range(N, nch, c, i0, i1);
      CK(cudaMemcpyAsync(ctx->stage + 3 * i0, forces + 3 * i0, 3 * (i1 - i0) * sizeof(double),
                         cudaMemcpyHostToDevice, st2));
      CK(cudaEventRecord(ev_acc[c], st2));
    }
  }
  // (the energies too, where the arrays allow)
  const size_t nb = (size_t)ctx->nboxes;
  double *const de = in_place(epot, nb) ? epot : nullptr, *const dw = in_place(virial, nb) ? virial : nullptr;
  // with the forces written in place, the call's last kernel sums the energies
  // of boxes of one chunk and passes on the status word
  const bool tail_sums = df && N > 0 && energy && ctx->maxc_tiles == 1;
  int rc = run_pair(ctx, energy, false, de, dw, false, !tail_sums);
  if (rc) return rc;
  bool status_sent = false;
  if (df && N > 0) {
    ForcesTail tail;
    if (tail_sums) {
      tail.nboxes = ctx->nboxes;
      tail.tile0 = ctx->d_tile0;
      tail.tileE = ctx->tileE;
      tail.tileW = ctx->tileW;
      tail.boxE = de ? de : ctx->boxE;
      tail.boxW = dw ? dw : ctx->boxW;
    }
#ifndef EXAMD_CHECKED  // (there the kernel's own index checks write the word)
    tail.host_status = ctx->h_status;
    status_sent = true;
#endif
    CK(ensure_inv(ctx));
    CK(launch_forces_out(step_args(ctx), 0, N, ctx->inv, df, accumulate, tail, st));
  } else if (forces && N > 0) {
    CK(ensure_inv(ctx));
    for (int c = 0; c < nch; ++c) {
      int64_t i0, i1;
      io_range(N, nch, c, i0, i1);
      if (accumulate) CK(cudaStreamWaitEvent(st, ev_acc[c], 0));
      CK(launch_forces_out(step_args(ctx), i0, i1, ctx->inv, ctx->stage, accumulate, ForcesTail{}, st));
      CK(cudaEventRecord(ctx->ev_io[kIoChunks + c], st));
      CK(cudaStreamWaitEvent(st2, ctx->ev_io[kIoChunks + c], 0));
      CK(cudaMemcpyAsync(forces + 3 * i0, ctx->stage + 3 * i0, 3 * (i1 - i0) * sizeof(double),
                         cudaMemcpyDeviceToHost, st2));
    }
  }
  if (epot && !de) CK(cudaMemcpyAsync(epot, ctx->boxE, ctx->nboxes * sizeof(double), cudaMemcpyDeviceToHost, st));
  if (virial && !dw) CK(cudaMemcpyAsync(virial, ctx->boxW, ctx->nboxes * sizeof(double), cudaMemcpyDeviceToHost, st));
  if (forces && N > 0 && !df) {
    CK(cudaEventRecord(ctx->ev_io[3 * kIoChunks], st2));
    CK(cudaStreamWaitEvent(st, ctx->ev_io[3 * kIoChunks], 0));
  }
  if (!status_sent) CK(queue_status(ctx));
  return EXAMD_OK;
}

// Waits for the force call and takes its status word.
int finish_forces(examd_ctx* ctx) {
  CK(cudaStreamSynchronize(ctx->st));
  const int rc = take_status(ctx);
  if (rc) return rc;
  ctx->forces_valid = true;
  return EXAMD_OK;
}

int forces_common(examd_ctx* ctx, double* forces, double* epot, double* virial, int accumulate) {
  const int rc = enqueue_forces(ctx, forces, epot, virial, accumulate);
  return rc ? rc : finish_forces(ctx);
}

}  // namespace

extern "C" {

// For the autotuner's trials on one configuration: a shape that keeps its CTAs per
// SM only with half the headroom loses one as soon as the atoms move on (the 16.8M
// mixture, tuned on its lattice, took tiles of 6x4x4 that way, whose 800 atoms
// later left two CTAs an SM: 8.2e8 atom-steps/s in FP64, 9.8e8 in the 5x4x4 that
// the trials now pick).
__attribute__((visibility("hidden"))) void examd_keep_headroom(examd_ctx* ctx) { ctx->whole_headroom = true; }

int examd_gpu_set_atoms(examd_ctx* ctx, int64_t n, const double* pos, const int* type, const double* vel) {
  if (!ctx || (n > 0 && !pos) || n != ctx->N) return EXAMD_ERR_ARG;
  cudaSetDevice(ctx->dev);
  cudaStream_t st = ctx->st;
  // The types: up to kHostTypes atoms are checked here, more of them by the
  // kernel that makes the meta words (which then costs a wait; a host loop and a
  // host array of 16.8M words took 40 of the call's 65 ms).
  const bool host_check = n <= kHostTypes;
  if (type && host_check)
    for (int64_t i = 0; i < n; ++i)
      if (type[i] < 0 || type[i] >= ctx->p.ntypes) return EXAMD_ERR_ARG;
  CK(cudaMemsetAsync(ctx->status, 0, sizeof(int), st));
  if (n > 0) {
    CK(cudaMemcpyAsync(ctx->stage, pos, 3 * n * sizeof(double), cudaMemcpyHostToDevice, st));
    if (vel) CK(cudaMemcpyAsync(ctx->stage2, vel, 3 * n * sizeof(double), cudaMemcpyHostToDevice, st));
    if (type) CK(cudaMemcpyAsync(ctx->d_meta_in, type, n * sizeof(int), cudaMemcpyHostToDevice, st));
    k_make_meta<<<nblk(n), 256, 0, st>>>(n, ctx->nboxes, ctx->d_atom0, type != nullptr, ctx->p.ntypes, ctx->d_meta_in,
                                         ctx->status);
    CK(cudaGetLastError());
    if (type && !host_check) {  // nothing of the context's atoms has been touched yet
      CK(queue_status(ctx));
      CK(cudaStreamSynchronize(st));
      if (const int trc = take_status(ctx)) return trc;
    }
  }
  const int s = ctx->cur;
  if (n > 0) {
    k_load_bin<<<nblk(n), 256, 0, st>>>(n, ctx->stage, vel ? ctx->stage2 : nullptr, ctx->d_meta_in, ctx->d_boxes,
                                        ctx->p.strict_box, ctx->X[s][0], ctx->X[s][1], ctx->X[s][2], ctx->V[s][0],
                                        ctx->V[s][1], ctx->V[s][2], ctx->meta[s], ctx->id[s], ctx->cellOld,
                                        ctx->slot, ctx->count, ctx->status);
    CK(cudaGetLastError());
  }
  int rc = finish_binning(ctx, true);
  if (rc) return rc;
  CK(queue_status(ctx));
  if ((rc = queue_occupancy(ctx))) return rc;
  CK(cudaStreamSynchronize(st));
  rc = take_status(ctx);
  if (rc) return rc;
  rc = apply_capacity(ctx);
  if (rc) return rc;
  if (ctx->list) {
    CK(cudaMemsetAsync(ctx->lw, 0, LW_WORDS * sizeof(int), st));
    rc = init_lists(ctx);
    if (rc) return rc;
    rc = check_status(ctx);
    if (rc) return rc;
  }
  ctx->atoms_set = true;
  ctx->forces_valid = false;
  return EXAMD_OK;
}

int examd_gpu_forces(examd_ctx* ctx, double* forces, double* epot, double* virial, int accumulate) {
  if (!ctx) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  return forces_common(ctx, forces, epot, virial, accumulate);
}

}  // extern "C"

namespace {

// The force call at new positions, queued (see examd_gpu_forces_at).
int enqueue_forces_at(examd_ctx* ctx, const double* pos, double* forces, double* epot, double* virial,
                      int accumulate) {
  const InCall in_call(ctx);
  cudaStream_t st = ctx->st, st2 = ctx->st2;
  const int s = ctx->cur;
  const int64_t N = ctx->N;
  if (N > 0) {
    // positions read in place, or in chunks of the caller's order: the
    // host->device copy of chunk c + 1 (second stream) overlaps the gather and
    // binning count of chunk c
    CK(ensure_inv(ctx));
    const double* const dp = in_place(pos, 3 * (size_t)N) ? pos : nullptr;
    auto gather = [&](const double* src, int64_t i0, int64_t i1) {
      if (ctx->list)
        return launch_gather_pos_list(i0, i1, src, ctx->d_boxes, ctx->p.strict_box, ctx->X[s][0], ctx->X[s][1],
                                      ctx->X[s][2], ctx->meta[s], ctx->inv, ctx->cellS, ctx->U, ctx->Ub, ctx->lw,
                                      ctx->status, st);
      return launch_chained(true, k_gather_pos_bin_range, nblk(i1 - i0, kIoThreads), kIoThreads, st, i0, i1, src,
                            ctx->d_boxes, ctx->p.strict_box, ctx->X[s][0], ctx->X[s][1], ctx->X[s][2], ctx->meta[s],
                            ctx->inv, ctx->cellOld, ctx->slot, ctx->count, ctx->status);
    };
    if (dp) {
      CK(gather(dp, 0, N));
    } else {
      CK(cudaEventRecord(ctx->ev_io[3 * kIoChunks], st));
      CK(cudaStreamWaitEvent(st2, ctx->ev_io[3 * kIoChunks], 0));
      const int nch = io_chunks(N);
      for (int c = 0; c < nch; ++c) {
        int64_t i0, i1;
        io_range(N, nch, c, i0, i1);
        CK(cudaMemcpyAsync(ctx->stage2 + 3 * i0, pos + 3 * i0, 3 * (i1 - i0) * sizeof(double),
                           cudaMemcpyHostToDevice, st2));
        CK(cudaEventRecord(ctx->ev_io[c], st2));
        CK(cudaStreamWaitEvent(st, ctx->ev_io[c], 0));
        CK(gather(ctx->stage2, i0, i1));
      }
    }
  }
  int rc = ctx->list ? maybe_rebuild(ctx) : finish_binning(ctx, true);
  if (rc) return rc;
  return enqueue_forces(ctx, forces, epot, virial, accumulate);
}

int finish_forces_at_eager(examd_ctx* ctx, const double* pos, double* forces, double* epot, double* virial,
                           int accumulate) {
  const int rc = enqueue_forces_at(ctx, pos, forces, epot, virial, accumulate);
  return rc ? rc : finish_forces(ctx);
}

// The force call at new positions with pinned buffers, as a captured graph kept
// in g (of the current parity) while its buffers and capacities stay.
int forces_at_graph(examd_ctx* ctx, examd_ctx::IoGraph& g, const double* pos, double* forces, double* epot,
                    double* virial, int accumulate) {
  const bool hit = g.exec && g.pos == pos && g.forces == forces && g.epot == epot && g.virial == virial &&
                   g.accumulate == accumulate && g.cap == ctx->cap && g.cap_redo == ctx->cap_redo &&
                   g.list_gen == ctx->list_gen;
  if (!hit) {
    if (g.exec) cudaGraphExecDestroy(g.exec);
    g = examd_ctx::IoGraph{};
    const int parity = ctx->cur;
    cudaGraph_t graph;
    CK(cudaStreamBeginCapture(ctx->st, cudaStreamCaptureModeThreadLocal));
    int rc = enqueue_forces_at(ctx, pos, forces, epot, virial, accumulate);
    cudaError_t ce = cudaStreamEndCapture(ctx->st, &graph);
    ctx->cur = parity;  // capture only recorded the work
    if (rc) return rc;
    if (ce != cudaSuccess) return ctx->cuda_fail(ce, "cudaStreamEndCapture");
    ce = cudaGraphInstantiate(&g.exec, graph, 0);
    cudaGraphDestroy(graph);
    if (ce != cudaSuccess) {
      g.exec = nullptr;
      return ctx->cuda_fail(ce, "cudaGraphInstantiate");
    }
    g.pos = pos;
    g.forces = forces;
    g.epot = epot;
    g.virial = virial;
    g.accumulate = accumulate;
    g.cap = ctx->cap;
    g.cap_redo = ctx->cap_redo;
    g.list_gen = ctx->list_gen;
  }
  CK(cudaGraphLaunch(g.exec, ctx->st));
  if (!ctx->list) ctx->cur = 1 - ctx->cur;  // the host-side effects of the captured call
  ctx->inv_valid = true;
  return finish_forces(ctx);
}

// The same for at most kSmallIo atoms in any host arrays.
int forces_at_small(examd_ctx* ctx, const double* pos, double* forces, double* epot, double* virial, int accumulate) {
  const size_t n3 = 3 * (size_t)ctx->N, nb = (size_t)ctx->nboxes;
  if (!ctx->h_io && cudaHostAlloc((void**)&ctx->h_io, (2 * n3 + 2 * nb) * sizeof(double), cudaHostAllocDefault) !=
                        cudaSuccess) {
    ctx->h_io = nullptr;
    cudaGetLastError();
    return finish_forces_at_eager(ctx, pos, forces, epot, virial, accumulate);
  }
  double *hp = ctx->h_io, *hf = hp + n3, *he = hf + n3, *hv = he + nb;
  const bool energy = epot || virial;
  accumulate = accumulate && forces ? 1 : 0;
  std::memcpy(hp, pos, n3 * sizeof(double));
  if (accumulate) std::memcpy(hf, forces, n3 * sizeof(double));
  const int rc = forces_at_graph(ctx, ctx->small_graph[ctx->cur][(energy ? 1 : 0) | (accumulate << 1)], hp,
                                 forces ? hf : nullptr, energy ? he : nullptr, energy ? hv : nullptr, accumulate);
  if (rc == EXAMD_ERR_CUDA) return rc;
  if (forces) std::memcpy(forces, hf, n3 * sizeof(double));  // (with a bad status too, as an eager call)
  if (epot) std::memcpy(epot, he, nb * sizeof(double));
  if (virial) std::memcpy(virial, hv, nb * sizeof(double));
  return rc;
}

}  // namespace

extern "C" {

int examd_gpu_forces_at(examd_ctx* ctx, const double* pos, double* forces, double* epot, double* virial,
                        int accumulate) {
  if (!ctx || (ctx->N > 0 && !pos)) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  CK(ensure_inv(ctx));  // outside any captured sequence
  const size_t n3 = 3 * (size_t)ctx->N, nb = (size_t)ctx->nboxes;
  if (ctx->N > 0 && ctx->N <= kSmallIo && !on_device(pos) && !on_device(forces) && !on_device(epot) &&
      !on_device(virial)) {
    if (ctx->small_calls == 2) return forces_at_small(ctx, pos, forces, epot, virial, accumulate);
    ++ctx->small_calls;  // a context used for a call or two is not worth a capture
  }
  if (ctx->N < kIoMinChunk || !pinned(pos, n3) || !pinned(forces, n3) || !pinned(epot, nb) || !pinned(virial, nb))
    return finish_forces_at_eager(ctx, pos, forces, epot, virial, accumulate);
  // same pinned buffers as last time at this parity: replay the captured call
  return forces_at_graph(ctx, ctx->io_graph[ctx->cur], pos, forces, epot, virial, accumulate);
}

}  // extern "C"

namespace {

KickArgs kick_args(examd_ctx* ctx, double ckick, double dt, bool drift, double hk) {
  KickArgs k{};
  k.s = step_args(ctx);
  const int c = ctx->cur;
  for (int a = 0; a < 3; ++a) {
    k.X[a] = ctx->X[c][a];
    k.V[a] = ctx->V[c][a];
  }
  k.meta = ctx->meta[c];
  k.ckick = ckick;
  k.dt = dt;
  k.drift = drift;
  k.hk = hk;
  for (int t = 0; t < EXAMD_MAX_TYPES; ++t) {
    k.ckm[t] = ckick * ctx->lj.minv[t];
    k.hkm[t] = hk * ctx->lj.minv[t];
  }
  k.keAtom = ctx->keAtom;
  k.lj = ctx->lj;
  k.cellOld = ctx->cellOld;
  k.slot = ctx->slot;
  k.count = ctx->count;
  k.status = ctx->status;
  k.list = ctx->list;
  k.U = ctx->U;
  k.Ub = ctx->Ub;
  k.lw = ctx->lw;
  return k;
}

// One step after the first: kick(ck) + drift + bin, pair.  keSlot receives the
// kinetic energy at the start of this step, eSlot the potential energy after.
// Pair-list mode: the binning and the lists only on the steps that the
// device decides to rebuild.  The energy sums (four small kernels, a fifth of a
// 32,000-atom step when they stood between its kernels) run on the second
// stream beside the binning and the next kick.
int kick(examd_ctx* ctx, double ck, double dt, bool drift, double* keSlot) {
  if (ctx->side_ke) {  // the last step's sums read the per-atom energies that this kick writes
    CK(cudaStreamWaitEvent(ctx->st, ctx->ev_side[2], 0));
    ctx->side_ke = false;
  }
  CK(launch_kick(kick_args(ctx, ck, dt, drift, keSlot ? 0.5 * dt : 0.0), ctx->st));
  if (!keSlot) return EXAMD_OK;
  CK(cudaEventRecord(ctx->ev_side[0], ctx->st));
  CK(cudaStreamWaitEvent(ctx->st2, ctx->ev_side[0], 0));
  CK(launch_box_sums(ctx->nboxes, ctx->d_atom0, ctx->maxc_atoms, ctx->keAtom, ctx->partial, keSlot, ctx->st2));
  CK(cudaEventRecord(ctx->ev_side[2], ctx->st2));
  ctx->side_ke = true;
  return EXAMD_OK;
}

int step_once(examd_ctx* ctx, double ck, double dt, double* keSlot, double* eSlot, double* wSlot) {
  int rc = kick(ctx, ck, dt, true, keSlot);
  if (rc) return rc;
  rc = ctx->list ? maybe_rebuild(ctx) : finish_binning(ctx, false);
  if (rc) return rc;
  return run_pair(ctx, eSlot != nullptr, false, eSlot, wSlot, eSlot != nullptr);
}

int ensure_ebuf(examd_ctx* ctx, int steps, bool host) {
  if (steps <= ctx->ebuf_steps && (!host || ctx->h_e)) return EXAMD_OK;
  steps = std::max(steps, ctx->ebuf_steps);
  if (ctx->h_e) cudaFreeHost(ctx->h_e);
  ctx->h_e = nullptr;
  if (host && cudaHostAlloc((void**)&ctx->h_e, 2 * (size_t)(steps + 1) * ctx->nboxes * sizeof(double),
                            cudaHostAllocDefault) != cudaSuccess) {
    ctx->h_e = nullptr;
    cudaGetLastError();  // reported here, not by the next launch
    return EXAMD_ERR_NOMEM;
  }
  if (steps <= ctx->ebuf_steps) return EXAMD_OK;
  size_t n = (size_t)(steps + 1) * ctx->nboxes;
  int rc;
  double *e = nullptr, *w = nullptr, *ke = nullptr;  // (the old ones stay if there is no room)
  if ((rc = dalloc(ctx, &e, n)) || (rc = dalloc(ctx, &w, n)) || (rc = dalloc(ctx, &ke, n))) {
    cudaGetLastError();
    for (double* q : {e, w, ke})
      if (q) cudaFree(q);
    return rc;
  }
  for (double* q : {ctx->boxE, ctx->boxW, ctx->boxKE})
    if (q) cudaFree(q);
  ctx->boxE = e;
  ctx->boxW = w;
  ctx->boxKE = ke;
  ctx->ebuf_steps = steps;
  // every captured graph that names the old energy buffers is stale: the step
  // loop's and the force call's (whose energy variant writes and reads boxE,
  // boxW)
  if (ctx->gexec) {
    cudaGraphExecDestroy(ctx->gexec);
    ctx->gexec = nullptr;
  }
  drop_io_graphs(ctx);
  return EXAMD_OK;
}

// The steady-state step loop of `chunk` steps (merged kicks) as one CUDA
// graph for buffer parity `parity`, captured and instantiated unless the
// cached one already matches.  Captures only: no step runs.
int ensure_chunk_graph(examd_ctx* ctx, int chunk, double dt, bool wantE, int parity) {
  const bool stale = !ctx->gexec || ctx->g_parity != parity || ctx->g_chunk != chunk ||
                     ctx->g_energy != (int)wantE || ctx->g_dt != dt || ctx->g_cap != ctx->cap ||
                     ctx->g_list_gen != ctx->list_gen;
  if (!stale) return EXAMD_OK;
  if (ctx->gexec) cudaGraphExecDestroy(ctx->gexec);
  ctx->gexec = nullptr;
  const int nb = ctx->nboxes;
  const int saved = ctx->cur;
  if (const int rc = join_side(ctx)) return rc;  // (the graph's own first step waits for nothing outside it)
  ctx->cur = parity;
  cudaGraph_t g;
  CK(cudaStreamBeginCapture(ctx->st, cudaStreamCaptureModeThreadLocal));
  int src = EXAMD_OK;
  for (int j = 0; j < chunk && src == EXAMD_OK; ++j)
    src = step_once(ctx, dt, dt, wantE ? ctx->boxKE + (size_t)j * nb : nullptr,
                    wantE ? ctx->boxE + (size_t)j * nb : nullptr, wantE ? ctx->boxW + (size_t)j * nb : nullptr);
  if (src == EXAMD_OK) src = join_side(ctx);
  cudaError_t ce = cudaStreamEndCapture(ctx->st, &g);
  ctx->side_ke = ctx->side_pe = false;
  // capture advanced the host-side parity; the graph leaves it unchanged (chunk
  // even; pair-list mode: no step swaps the buffers)
  ctx->cur = saved;
  if (src != EXAMD_OK) return src;
  if (ce != cudaSuccess) return ctx->cuda_fail(ce, "cudaStreamEndCapture");
  ce = cudaGraphInstantiate(&ctx->gexec, g, 0);
  cudaGraphDestroy(g);
  if (ce != cudaSuccess) {
    ctx->gexec = nullptr;
    return ctx->cuda_fail(ce, "cudaGraphInstantiate");
  }
  ctx->g_parity = parity;
  ctx->g_chunk = chunk;
  ctx->g_energy = wantE;
  ctx->g_dt = dt;
  ctx->g_cap = ctx->cap;
  ctx->g_list_gen = ctx->list_gen;
  return EXAMD_OK;
}

}  // namespace

extern "C" {

int examd_gpu_run(examd_ctx* ctx, int nsteps, double dt, int graph_chunk, double* energies, examd_stats* stats) {
  if (!ctx || nsteps < 0 || !(dt > 0) || graph_chunk < 0) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  cudaStream_t st = ctx->st;
  const int nb = ctx->nboxes;
  const bool wantE = energies != nullptr;
  int chunk = graph_chunk > 0 ? (graph_chunk + 1) / 2 * 2 : 0;
  // eager steps' energies wait on the device too
  const int eager = eager_slots(nb), slots = std::max(chunk, wantE ? eager : 1) + 1;
  int rc = ensure_ebuf(ctx, slots, wantE);
  if (rc) return rc;
  if (!ctx->forces_valid) {
    rc = run_pair(ctx, false, false);
    if (rc) return rc;
    ctx->forces_valid = true;
  }
  if (nsteps == 0) return EXAMD_OK;
  const double h = 0.5 * dt;
  // Energies: slot j of boxE holds the potential energy after step first + j
  // (0-based), slot j of boxKE the kinetic energy before it, i.e. after step
  // first + j - 1; `held` slots are filled.  fetch() brings them to the caller
  // in one copy each (a copy per box and step took 0.36 of the 0.40 s that 41
  // steps of a 512-box ensemble took).
  int first = 0, held = 0;
  auto queue_energies = [&](int extra_ke) -> int {
    const size_t n = (size_t)held * nb, nk = (size_t)(held + extra_ke) * nb;
    double* he = ctx->h_e + (size_t)(ctx->ebuf_steps + 1) * nb;
    if (const int jrc = join_side(ctx)) return jrc;
    if (nk) CK(cudaMemcpyAsync(ctx->h_e, ctx->boxKE, nk * sizeof(double), cudaMemcpyDeviceToHost, st));
    if (n) CK(cudaMemcpyAsync(he, ctx->boxE, n * sizeof(double), cudaMemcpyDeviceToHost, st));
    return EXAMD_OK;
  };
  auto store_energies = [&](int extra_ke) {  // after the stream's work
    const double* he = ctx->h_e + (size_t)(ctx->ebuf_steps + 1) * nb;
    for (int j = 0; j < held + extra_ke; ++j)
      for (int b = 0; b < nb; ++b) {
        const size_t g = (size_t)(first + j);
        if (g > 0) energies[2 * ((g - 1) * nb + b)] = ctx->h_e[(size_t)j * nb + b];
        if (j < held) energies[2 * (g * nb + b) + 1] = he[(size_t)j * nb + b];
      }
    first += held;
    held = 0;
  };
  auto fetch = [&]() -> int {
    if (!wantE || held == 0) return EXAMD_OK;
    if (const int qrc = queue_energies(0)) return qrc;
    CK(cudaStreamSynchronize(st));
    store_energies(0);
    return EXAMD_OK;
  };
  auto slot = [&](double* p) { return wantE ? p + (size_t)held * nb : nullptr; };
  CK(cudaEventRecord(ctx->e0, st));
  // step 1: half kick + drift, then forces
  rc = step_once(ctx, h, dt, nullptr, slot(ctx->boxE), slot(ctx->boxW));
  if (rc) return rc;
  held = 1;
  int done = 1;
  // steady state: merged kicks v += dt F/m
  while (done < nsteps) {
    const int left = nsteps - done;
    if (chunk > 0 && left >= chunk) {
      if ((rc = fetch())) return rc;  // the graph writes the slots from the first
      first = done;
      rc = ensure_chunk_graph(ctx, chunk, dt, wantE, ctx->cur);
      if (rc) return rc;
      CK(cudaGraphLaunch(ctx->gexec, st));
      held = chunk;
      done += chunk;
      // the capacities may need to grow as the density fluctuates: the status
      // word, the occupancy, the list words and the energies in one wait
      CK(queue_status(ctx));
      if ((rc = queue_occupancy(ctx))) return rc;
      if (ctx->list && (rc = queue_list_words(ctx))) return rc;
      if (wantE && (rc = queue_energies(0))) return rc;
      CK(cudaStreamSynchronize(st));
      if (wantE) store_energies(0);
      rc = take_status(ctx);
      if (rc) return rc;
      bool grew = false;
      rc = apply_capacity(ctx, &grew);
      if (rc) return rc;
      if (ctx->list && (rc = update_lists(ctx, grew))) return rc;
    } else {
      if (wantE && held >= eager && (rc = fetch())) return rc;
      if (held == 0) first = done;
      rc = step_once(ctx, dt, dt, slot(ctx->boxKE), slot(ctx->boxE), slot(ctx->boxW));
      if (rc) return rc;
      held += 1;
      done += 1;
    }
  }
  // closing half kick: v(t_n) = v(t_n - h) + h F/m
  if (held == 0) first = nsteps;
  if ((rc = kick(ctx, h, dt, false, slot(ctx->boxKE)))) return rc;
  if (wantE && (rc = queue_energies(1))) return rc;
  CK(cudaEventRecord(ctx->e1, st));
  CK(queue_status(ctx));
  CK(cudaStreamSynchronize(st));
  if (wantE) store_energies(1);
  rc = take_status(ctx);
  if (rc) return rc;
  ctx->forces_valid = true;
  if (stats) {
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, ctx->e0, ctx->e1));
    std::memset(stats, 0, sizeof(*stats));
    stats->ms = ms;
    stats->steps = nsteps;
    if (wantE) {
      for (int b = 0; b < nb; ++b) {
        stats->ekin += energies[2 * ((size_t)(nsteps - 1) * nb + b)];
        stats->epot += energies[2 * ((size_t)(nsteps - 1) * nb + b) + 1];
      }
    }
  }
  return EXAMD_OK;
}

int examd_gpu_prepare_run(examd_ctx* ctx, double dt, int graph_chunk, int energies) {
  if (!ctx || !(dt > 0) || graph_chunk < 0) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  const int chunk = graph_chunk > 0 ? (graph_chunk + 1) / 2 * 2 : 0;
  int rc = ensure_ebuf(ctx, std::max(chunk, energies ? eager_slots(ctx->nboxes) : 1) + 1, energies != 0);
  if (rc) return rc;
  if (!ctx->forces_valid) {
    rc = run_pair(ctx, false, false);
    if (rc) return rc;
    rc = check_status(ctx);
    if (rc) return rc;
    ctx->forces_valid = true;
  }
  if (chunk == 0) return EXAMD_OK;
  // the run's first step flips the sort's double buffer: its graph chunks
  // run at the other parity (pair-list mode: at this one)
  rc = ensure_chunk_graph(ctx, chunk, dt, energies != 0, ctx->list ? ctx->cur : 1 - ctx->cur);
  if (rc) return rc;
  CK(cudaStreamSynchronize(ctx->st));
  return EXAMD_OK;
}

int examd_gpu_time_phases(examd_ctx* ctx, int nsteps, double dt, double* ms) {
  if (!ctx || nsteps < 1 || !(dt > 0) || !ms) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  cudaStream_t st = ctx->st;
  int rc;
  if (!ctx->forces_valid) {
    rc = run_pair(ctx, false, false);
    if (rc) return rc;
    ctx->forces_valid = true;
  }
  double acc[3] = {0.0, 0.0, 0.0};
  for (int k = 0; k < nsteps; ++k) {
    // one steady-state step (merged kick), as the captured loop runs it
    CK(cudaEventRecord(ctx->e0, st));
    CK(launch_kick(kick_args(ctx, dt, dt, true, 0.0), st));
    CK(cudaEventRecord(ctx->e1, st));
    rc = ctx->list ? maybe_rebuild(ctx) : finish_binning(ctx, false);
    if (rc) return rc;
    CK(cudaEventRecord(ctx->e2, st));
    rc = run_pair(ctx, false, false);
    if (rc) return rc;
    CK(cudaEventRecord(ctx->e3, st));
    CK(cudaStreamSynchronize(st));
    float t01 = 0.f, t12 = 0.f, t23 = 0.f;
    CK(cudaEventElapsedTime(&t01, ctx->e0, ctx->e1));
    CK(cudaEventElapsedTime(&t12, ctx->e1, ctx->e2));
    CK(cudaEventElapsedTime(&t23, ctx->e2, ctx->e3));
    acc[0] += t01;
    acc[1] += t12;
    acc[2] += t23;
  }
  rc = check_status(ctx);
  if (rc) return rc;
  for (int a = 0; a < 3; ++a) ms[a] = acc[a] / nsteps;
  return EXAMD_OK;
}

int examd_gpu_time_rebuild(examd_ctx* ctx, int reps, double* ms) {
  if (!ctx || reps < 1 || !ms) return EXAMD_ERR_ARG;
  if (!ctx->list) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  CK(cudaEventRecord(ctx->e0, ctx->st));
  for (int r = 0; r < reps; ++r) {
    const int rc = rebuild(ctx, nullptr);
    if (rc) return rc;
  }
  CK(cudaEventRecord(ctx->e1, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  float t = 0.f;
  CK(cudaEventElapsedTime(&t, ctx->e0, ctx->e1));
  *ms = t / reps;
  ctx->forces_valid = false;  // the sorted order changed
  return check_status(ctx);
}

int examd_gpu_list_info(examd_ctx* ctx, int64_t* builds, int* capacity, int* longest, int* fallback_tiles) {
  if (!ctx) return EXAMD_ERR_ARG;
  int64_t b = 0;
  int c = 0, l = 0, f = 0;
  if (ctx->list) {
    cudaSetDevice(ctx->dev);
    const int rc = read_list_words(ctx);
    if (rc) return rc;
    b = ctx->h_lw[LW_BUILDS] + ctx->host_builds;
    c = ctx->lk;
    l = ctx->h_lw[LW_LMAX];
    f = ctx->h_lw[LW_FBN];
  }
  if (builds) *builds = b;
  if (capacity) *capacity = c;
  if (longest) *longest = l;
  if (fallback_tiles) *fallback_tiles = f;
  return EXAMD_OK;
}

int examd_gpu_get_state(examd_ctx* ctx, double* pos, double* vel) {
  if (!ctx) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  const int c = ctx->cur;
  if (pos) {
    CK(launch_state_out(ctx->N, ctx->X[c], ctx->id[c], ctx->stage, ctx->st));
    CK(cudaMemcpyAsync(pos, ctx->stage, 3 * ctx->N * sizeof(double), cudaMemcpyDeviceToHost, ctx->st));
  }
  if (vel) {
    CK(launch_state_out(ctx->N, ctx->V[c], ctx->id[c], ctx->stage2, ctx->st));
    CK(cudaMemcpyAsync(vel, ctx->stage2, 3 * ctx->N * sizeof(double), cudaMemcpyDeviceToHost, ctx->st));
  }
  CK(cudaStreamSynchronize(ctx->st));
  return EXAMD_OK;
}

int examd_gpu_kinetic(examd_ctx* ctx, double* ekin) {
  if (!ctx || !ekin) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  const int c = ctx->cur;
  CK(launch_kinetic(ctx->N, ctx->nboxes, ctx->d_atom0, ctx->maxc_atoms, ctx->V[c], ctx->meta[c], ctx->lj,
                    ctx->keAtom, ctx->partial, ctx->boxKE,
                    ctx->st));
  CK(cudaMemcpyAsync(ekin, ctx->boxKE, ctx->nboxes * sizeof(double), cudaMemcpyDeviceToHost, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  return EXAMD_OK;
}

int examd_gpu_scale_velocities(examd_ctx* ctx, const double* factor) {
  if (!ctx || !factor) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  const int c = ctx->cur;
  CK(cudaMemcpyAsync(ctx->d_factor, factor, ctx->nboxes * sizeof(double), cudaMemcpyHostToDevice, ctx->st));
  CK(launch_scale_v(ctx->N, ctx->V[c], ctx->meta[c], ctx->d_factor, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  return EXAMD_OK;
}

int examd_gpu_time_forces(examd_ctx* ctx, int reps, double* ms, double* kernel_ms) {
  if (!ctx || reps < 1) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  cudaStream_t st = ctx->st;
  int rc = run_pair(ctx, false, false);  // warm-up
  if (rc) return rc;
  CK(cudaEventRecord(ctx->e0, st));
  for (int r = 0; r < reps; ++r) {
    rc = run_pair(ctx, false, false);
    if (rc) return rc;
  }
  CK(cudaEventRecord(ctx->e1, st));
  CK(cudaStreamSynchronize(st));
  float t = 0.f;
  CK(cudaEventElapsedTime(&t, ctx->e0, ctx->e1));
  if (ms) *ms = t;
  if (kernel_ms) *kernel_ms = t / reps;
  rc = check_status(ctx);
  if (rc) return rc;
  ctx->forces_valid = true;
  return EXAMD_OK;
}

int examd_gpu_counters(examd_ctx* ctx, int64_t* candidates, int64_t* accepted, int64_t* evaluated,
                       int64_t* tiles, int64_t* max_tile_atoms) {
  if (!ctx) return EXAMD_ERR_ARG;
  if (!ctx->atoms_set) return EXAMD_ERR_STATE;
  cudaSetDevice(ctx->dev);
  int rc;
  // pair-list mode: the counts are the enumeration's, which needs every atom
  // inside its cell: a fresh sort and lists first
  if (ctx->list && (rc = rebuild(ctx, nullptr))) return rc;
  rc = run_pair(ctx, false, true);
  if (rc) return rc;
  std::vector<long long> c(3 * (size_t)ctx->ntiles);
  CK(cudaMemcpyAsync(c.data(), ctx->tileC, c.size() * sizeof(long long), cudaMemcpyDeviceToHost, ctx->st));
  int occ = 0;
  CK(cudaMemsetAsync(ctx->d_occ, 0, 2 * sizeof(int), ctx->st));
  k_tile_occupancy<<<ctx->ntiles, 128, 0, ctx->st>>>(ctx->d_tiles, ctx->d_boxes, ctx->cstart, ctx->d_occ);
  CK(cudaGetLastError());
  CK(cudaMemcpyAsync(&occ, ctx->d_occ, sizeof(int), cudaMemcpyDeviceToHost, ctx->st));
  CK(cudaStreamSynchronize(ctx->st));
  rc = check_status(ctx);
  if (rc) return rc;
  long long s1 = 0, s2 = 0, s3 = 0;
  for (int t = 0; t < ctx->ntiles; ++t) {
    s1 += c[3 * t];
    s2 += c[3 * t + 1];
    s3 += c[3 * t + 2];
  }
  if (candidates) *candidates = s1;
  if (accepted) *accepted = s2;
  if (evaluated) *evaluated = s3;
  if (tiles) *tiles = ctx->ntiles;
  if (max_tile_atoms) *max_tile_atoms = occ;
  ctx->forces_valid = true;
  return EXAMD_OK;
}

}  // extern "C"
