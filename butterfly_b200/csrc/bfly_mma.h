// Butterfly products of large problems as matrix products on the tensor cores (tcgen05).
//
// The stages of a product are cut into groups whose column bits fit a window of six bits.  Inside a window the
// stages of a group, twelve of them where two blocks meet at their turning point, are ONE dense 64 x 64 matrix per
// block of 64 columns ("operator").  A pass multiplies tiles of 128 rows by these operators; the backward multiplies the
// gradient by the transposed operator and accumulates the gradient of the whole operator, g^T x over the rows, which
// a small kernel takes apart into the gradients of the stages afterwards.  Per pass a tile crosses shared memory once,
// whatever the number of stages.  The operators' arithmetic takes 1152 clocks of a tile (2432 in the backward) where the
// tile's trip through HBM takes 2900 (4300).
//
// Precision.  A float32 value, scaled (kMmaScale), is the exact sum of three bfloat16 slices (8 + 8 + 8 bits).  Operators are multiplied out in
// float64 and cut into four parts, the first of few bits.  Nine of the twelve products are formed (the others are below
// 2^-25 of the whole) and summed in float32 by size.  tcgen05 cuts its sums towards zero, so those that count are kept
// exact or short (bfly_mma.cu).
//
// Range.  Operators and slices stand for the stages only while values are ordinary: no infinities or NaN, which spread stage
// by stage, nothing that overflows halfway.  Rows, gradients and activations from 2^40 on, operators (or products of some of
// their stages) from 2^20 on and sums that overflow raise a flag, whatever else they are; behind the passes the phase
// kernels are launched too and run if the flag is up (bfly_driver.h).  Their results, from the caller's tensors, then
// replace everything.
//
// Columns are counted in floats here: complex rows are rows of 2n floats whose bit 0 tells real from imaginary parts,
// always inside the window, and a complex operator of 32 x 32 is a real one of 64 x 64.
//
// Between passes rows live in planes of their own layout, (stack, row tile, column, 128 rows): every column of a tile
// is 512 contiguous bytes, so that a window of any column bits is read and written in long runs.  Only the first read
// and the last write of a product see the caller's rows; groups at the ends keep the low column bits in the window.
//
// This header: planning and parameter blocks, plain C++.  Kernels: bfly_mma.cu.
#pragma once
#include <algorithm>
#include <cstring>
#include <vector>

#include "bfly_plan.h"

namespace bfly {

constexpr int kMmaWin = 6;                    // bits of a window: operators are 64 x 64
constexpr int kMmaCols = 1 << kMmaWin;
constexpr int kMmaRows = 128;                 // rows of a tile (the lanes of tensor memory)
constexpr int kMmaMaxStages = 12;             // radix-2 stages a group may hold (a radix-4 factor counts as two)
constexpr int kMmaMaxGroups = 8;
constexpr int kMmaParts = 4;                  // bfloat16 parts of an operator
constexpr int kMmaImageBytes = kMmaParts * kMmaCols * kMmaCols * 2;  // one operator, swizzled as tcgen05 reads it
constexpr int kMmaRowBits = 40, kMmaOpBits = 20;             // rows below 2^40, operators below 2^20
// Rows and operators enter the products times 2^24 each: the last of a value's 24 bits, 2^-149 at the least, is then a normal
// bfloat16 (which have the exponents of float32, and 8 bits).  From 2^40 and 2^20 up to there nothing overflows either.
constexpr int kMmaScale = 24;
constexpr size_t kMmaHead = 256;              // in front of what a forward leaves and of a backward's work space: the flag
constexpr int kMmaBwMaxCtas = 160;            // most CTAs of a backward pass (one per SM)
constexpr int kMmaSlotFloats = 2 * kMmaCols * kMmaCols;      // an operator gradient as a CTA leaves it: two halves to be added
struct MmaStage {
  uint32_t tw_off;       // element offset of the factor's twiddles inside one stack
  uint8_t lbit, gbit;    // lowest bit the factor acts on: in the window, in the row (elements)
  uint8_t radix, which;
};
// Window: float column bits [0, ib) and [b0, b0 + 6 - ib).
struct MmaGeom {
  int ib, b0, log_nf;
  int sib;  // 2^sib CTAs walk the same row tiles of neighbouring blocks (mma_cta_of)
  BFLY_HD int mid() const { return b0 - ib; }
  // first column of block q of the row (the blocks are numbered by the bits outside the window)
  BFLY_HD int base(int q) const { return ((q & ((1 << mid()) - 1)) << ib) | ((q >> mid()) << (b0 + kMmaWin - ib)); }
  BFLY_HD int col(int j) const { return (j & ((1 << ib) - 1)) | ((j >> ib) << b0); }
};
struct MmaGroup {
  int t0, t1;  // stages
  MmaGeom geo;
  int nst;
  int passive; // element window bits no stage of the group acts on
  MmaStage st[kMmaMaxStages];
};

// Row tiles of a block by 2^log_tiles: `count` parts, whose operator gradients (and column sums) are added up in float64.
struct MmaParts {
  int log_tiles, count;
  BFLY_HD int of(int tile) const { return tile >> log_tiles; }
  BFLY_HD bool ends(int tile) const { return ((tile + 1) & ((1 << log_tiles) - 1)) == 0; }
  BFLY_HD bool begins(int tile) const { return tile > 0 && (tile & ((1 << log_tiles) - 1)) == 0; }
};

// Rows of the caller: (row, stack, column) at p[row * sB + stack * sS + column], columns from `cols` on read as zero and
// are not written.  flat > 0: the stacks are side by side in one matrix of `flat` columns, the last ones cut short.
struct MmaRowsIO {
  float* p;
  int64_t sB, sS;
  int cols, flat;
  int align;  // bytes every row start is a multiple of (4, 8, 16 or 32)
};
BFLY_HD int mma_cols(const MmaRowsIO& r, int stack, int log_nf) {
  if (r.flat <= 0) return r.cols;
  const int left = r.flat - stack * (1 << log_nf);
  return left < r.cols ? (left < 0 ? 0 : left) : r.cols;
}

struct MmaPass {
  MmaGeom geo;
  int S, B, nq, nt;       // stacks, rows, blocks of a row, row tiles
  MmaParts parts;
  const uint8_t* images;  // operators of the group, (stack, block)
  // forward: in -> out.  backward: gradient in -> out, x the activation that entered the group.  *_t: a plane instead of rows
  const float* in_t;
  float* out_t;
  const float* x_t;
  MmaRowsIO in, out, x;
  int reduce;             // backward: add to the output rows (their stack stride is 0)
  const float* bias;      // forward: bias[stack * nf + column] for flat positions below bias_len
  int bias_len;
  float* slots;           // backward: operator gradients (mma_slot)
  float* bias_slots;      // backward: column sums of the incoming gradient, 64 per slot; may be null
  int* flag;              // set to 1 for values that are not ordinary
  const int* kept_flag;   // backward: the forward's, taken over; may be null
};

struct MmaPrep {
  const void* tw[2];
  int64_t tw_stack[2];
  int S, nq, ng;
  uint8_t* images;        // (group, stack, block)
  int* flag;
  MmaGroup g[kMmaMaxGroups];
};
struct MmaPost {
  const void* tw[2];
  void* dtw[2];
  int64_t tw_stack[2];
  int S, nq, nt, ng, ctas;
  MmaParts parts;
  int last_group, group[kMmaMaxGroups];  // number of the product's last group, and of g[i] (by the launch)
  const float* slots;     // (group, slot)
  int64_t slots_group;    // floats from a group to the next
  const float* bias_slots;
  int* flag;
  float* dbias;           // with bias_slots: column sums of the last group's incoming gradient
  int dbias_len;
  MmaGroup g[kMmaMaxGroups];
};

// Work of a pass: tiles numbered (stack, block, row tile); CTA c of G takes [W c / G, W (c + 1) / G), so that it keeps an
// operator over many row tiles.  mma_cta_of: the CTA that takes tile w.  With geo.sib, CTAs and blocks count in groups of
// 2^sib, one block to a CTA of the group.
BFLY_HD int64_t mma_first_tile(int64_t W, int G, int c) { return W * c / G; }
BFLY_HD int mma_cta_of(int64_t W, int G, int64_t w) { return (int)(((w + 1) * G + W - 1) / W) - 1; }
// CTAs of a pass, and where group c of them leaves its sums over part `part` of a block's row tiles (MmaParts): all three walk
// up, so that no two sums share a slot.  Where a CTA begins with a part that is not a block's first, the slot in front of its own
// stays free, and the CTA writes zeros there: the slots of a block are those from its first CTA's and part's to its last.
BFLY_HD int mma_ctas(const MmaGeom& geo, int64_t tiles, int most) { return (int)(tiles < most ? tiles : most) >> geo.sib << geo.sib; }
BFLY_HD int64_t mma_slot(const MmaGeom& geo, const MmaParts& parts, int64_t block, int part, int c) {
  return (((block >> geo.sib) * parts.count + part + c) << geo.sib) | (block & ((1 << geo.sib) - 1));
}

// ------------------------------------------------------------------ host planning

// Cut the stages into groups: fewest passes, and groups at the ends of the product that keep at least eight floats
// (32 bytes, a sector) of a row together: pieces of 16 bytes cost a pass about a third more, shorter ones multiply it.
inline bool mma_groups(const std::vector<Stage>& st, int F, int log_n, std::vector<MmaGroup>& out) {
  const int ns = (int)st.size(), log_nf = log_n + F;
  if (log_nf < kMmaWin) return false;
  std::vector<double> best(ns + 1, 1e30);
  std::vector<int> from(ns + 1, -1);
  std::vector<MmaGeom> geo(ns + 1);
  best[0] = 0;
  for (int j = 0; j < ns; ++j) {
    if (best[j] >= 1e29) continue;
    int lo = 32, hi = 0, weight = 0;
    for (int e = j + 1; e <= ns; ++e) {
      const Stage& s = st[e - 1];
      lo = std::min(lo, s.bit + F);
      hi = std::max(hi, s.bit + F + (s.radix == 4 ? 2 : 1));
      weight += s.radix == 4 ? 2 : 1;
      MmaGeom g{kMmaWin, kMmaWin, log_nf, 0};
      if (hi > kMmaWin) { g.ib = kMmaWin - (hi - lo); g.b0 = lo; }
      if (g.ib < F || weight > kMmaMaxStages) break;
      const double rough = g.ib >= 5 ? 0 : g.ib == 4 ? 0.1 : g.ib == 3 ? 0.2 : g.ib == 2 ? 1.5 : g.ib == 1 ? 3.0 : 6.0;
      const double cost = best[j] + 1 + (j == 0 ? rough : 0) + (e == ns ? rough : 0);
      if (cost < best[e] - 1e-9) { best[e] = cost; from[e] = j; geo[e] = g; }
    }
  }
  if (from[ns] < 0) return false;
  out.clear();
  for (int e = ns; e > 0; e = from[e]) {
    MmaGroup g;
    std::memset(&g, 0, sizeof(g));
    g.t0 = from[e]; g.t1 = e; g.geo = geo[e];
    g.passive = (kMmaCols >> F) - 1;
    for (int k = g.t0; k < e; ++k) {
      MmaStage& m = g.st[g.nst++];
      const int fb = st[k].bit + F;
      m.tw_off = st[k].tw_off;
      m.gbit = (uint8_t)st[k].bit;
      m.lbit = (uint8_t)((fb < g.geo.ib ? fb : fb - g.geo.b0 + g.geo.ib) - F);
      m.radix = (uint8_t)st[k].radix;
      m.which = (uint8_t)st[k].which;
      g.passive &= ~((st[k].radix == 4 ? 3 : 1) << m.lbit);
    }
    // Pieces of the caller's rows below a cache line: the CTAs that share lines keep together, so that L2 joins the pieces.
    if ((g.t0 == 0 || g.t1 == ns) && g.geo.ib < 5 && g.geo.mid() >= 2) g.geo.sib = 2;
    out.push_back(g);
  }
  std::reverse(out.begin(), out.end());
  return (int)out.size() <= kMmaMaxGroups;
}

// A float32 sum over the tiles of a long run is off by its roundings: normal values, rows of 4096 columns, gradient of the factors
// 1.7e-7 for 16384 rows and 2.6e-7 for 49152 in one part, 1.3e-7 and 1.8e-7 in parts of 32 tiles (phases 3.3e-7, 5.5e-7).  A
// part more costs a slot, 32 KB written and read where its rows are 2 MB.  Runs of up to 48 tiles (148 CTAs share the work) stay whole; few blocks, whose slots one CTA
// each has to add up, get longer parts.
inline MmaParts mma_parts(int64_t blocks, int64_t nt) {
  MmaParts p{30, 1};
  const int64_t run = std::min(nt, (blocks * nt + 147) / 148);
  if (run > 48) p.log_tiles = blocks < 16 ? 7 : 5;
  p.count = (int)(((nt - 1) >> p.log_tiles) + 1);
  return p;
}

struct MmaLayout {
  std::vector<MmaGroup> g;
  int F, log_nf, nq;
  int64_t nt;                   // row tiles
  MmaParts parts;
  size_t plane;                 // bytes of a plane
  size_t images;                // operators of all groups
  size_t slots, bias_slots;     // backward: operator gradients of all groups, bias sums
  size_t slots_per_group(int S) const { return (size_t)S * nq * parts.count + kMmaBwMaxCtas; }
  // what a forward leaves: the flag, the activations between the groups, the operators
  size_t kept() const { return kMmaHead + (g.size() - 1) * plane + images; }
  // work space of a backward that starts from that (a gradient plane), and of one that makes it itself (the gradient takes
  // the place of the last activations)
  size_t bw_bytes(bool from_kept) const { return slots + bias_slots + (from_kept ? kMmaHead + (g.size() > 1 ? plane : 0) : kept()); }
};

}  // namespace bfly
