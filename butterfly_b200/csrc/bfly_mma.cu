// Kernels of the products that run on the tensor cores; bfly_mma.h explains the method.
//
//   bfly_mma_prep_kernel   operators of all groups, multiplied out in float64, as bfloat16 slices
//   bfly_mma_pass_kernel   one pass: forward, or backward (gradient through the transposed operator, operator gradient)
//   bfly_mma_post_kernel   operator gradients -> gradients of the stages
#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>
#include <type_traits>

#include "bfly_fast.h"
#include "bfly_mma.h"
#include "bfly_tma.h"

namespace bfly {
namespace {

// ------------------------------------------------------------------ tcgen05

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, 128-byte swizzle.  K-major operands: rows of 128 bytes (64 K values), `sbo` bytes
// between groups of eight rows.  MN-major operands: blocks of 64 M (N) values by 8 K, `sbo` bytes between blocks along K,
// `lbo` along M (N).
__device__ __forceinline__ uint64_t mma_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr & 0x3ffff) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Instruction descriptor: bfloat16 operands, float32 accumulator, M = 128; ta / tb: operand is MN-major.
__host__ __device__ constexpr uint32_t mma_idesc(int N, int ta, int tb) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)ta << 15) | ((uint32_t)tb << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kMmaRows >> 4) << 24);
}
// Called by a whole warp, which elects the thread that issues: the operands then stay in uniform registers.  (Issued from
// a branch that one thread takes, an instruction cost about 80 clocks, 4000 for a tile of the backward.)
__device__ __forceinline__ void mma_issue(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n .reg .pred p, q;\n elect.sync _|q, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n"
      " @q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n @q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_before_sync() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after_sync() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld8(uint32_t addr, float* v) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "r"(addr));
}

// tcgen05 cuts the sum of every instruction (16 products and the accumulator) to 24 bits towards zero: half a unit of the
// last place on average, always towards zero, where rounding has no mean.  A constant that puts the mean back is wrong
// wherever nothing was cut, so the sums that count are kept exact instead: the largest part of an operator entry is a
// multiple of 1/16 of the largest entry of its row and column (bfly_mma_prep_kernel), four bits at most beside the eight of
// the rows' first slice, and values down to 2^-9 of the largest of 64 add up within 24 bits.  What is cut from the other
// products is a sixteenth of a unit.

// ------------------------------------------------------------------ values and slices

// Eight neighbouring float32 values, times 2^kMmaScale, as their three bfloat16 slices, 16 bytes each.  The first slice cuts (rounding would
// turn the largest finite values into infinities), the second rounds, the third is what is left: exact.  `probe`: the largest
// magnitudes so far (a bfloat16 pair of any signs).
__device__ __forceinline__ void split8(const float* v, uint4& s1, uint4& s2, uint4& s3, uint32_t& probe) {
  uint32_t a1[4], a2[4], a3[4];
  uint64_t minus, scale;
  asm("mov.b64 %0, {%1, %1};" : "=l"(scale) : "f"((float)(1 << kMmaScale)));
  asm("mov.b64 %0, {%1, %1};" : "=l"(minus) : "f"(-1.f));
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint64_t x, h, r;
    uint32_t u, w, ru, rw;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(v[2 * i]), "f"(v[2 * i + 1]));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(x) : "l"(x), "l"(scale));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(u), "=r"(w) : "l"(x));
    a1[i] = __byte_perm(u, w, 0x7632);
    asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(probe) : "r"(probe), "r"(a1[i]));
    asm("mov.b64 %0, {%1, %2};" : "=l"(h) : "r"(u & 0xffff0000u), "r"(w & 0xffff0000u));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(h), "l"(minus), "l"(x));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(ru), "=r"(rw) : "l"(r));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(a2[i]) : "f"(__uint_as_float(rw)), "f"(__uint_as_float(ru)));
    asm("mov.b64 %0, {%1, %2};" : "=l"(h) : "r"(a2[i] << 16), "r"(a2[i] & 0xffff0000u));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(h), "l"(minus), "l"(r));
    asm("mov.b64 {%0, %1}, %2;" : "=r"(ru), "=r"(rw) : "l"(r));
    a3[i] = __byte_perm(ru, rw, 0x7632);
  }
  s1 = make_uint4(a1[0], a1[1], a1[2], a1[3]);
  s2 = make_uint4(a2[0], a2[1], a2[2], a2[3]);
  s3 = make_uint4(a3[0], a3[1], a3[2], a3[3]);
}
__device__ __forceinline__ bool beyond(uint32_t probe) {
  constexpr uint32_t most = (127 + kMmaScale + kMmaRowBits) << 7;
  return (probe & 0x7fff) >= most || ((probe >> 16) & 0x7fff) >= most;
}

// Where a CTA is: stack, first column of its block, row tile.
struct Spot { int stack, cbase, tile; };

__device__ __forceinline__ void load8(const float* src, float* v) {  // 32-byte aligned
  asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "l"(src) : "memory");
}

// Eight window columns of a row that are no 32 bytes in one piece, or not all there: all of the thread's units at once, in
// the widest pieces that the window and the rows' alignment allow.  (One unit after the other, the 1.6 % of the tiles that
// meet a cut column held 970 us against 530 for a layer of 4088 and one of 4096 columns.)
template <int PIECE, int N> __device__ __forceinline__ void load_pieces(const float* src, const MmaPass& p, int j0, int c0, int cols, int64_t rows, int64_t step, int stride, float (*v)[8]) {
#pragma unroll
  for (int i = 0; i < 8; i += PIECE) {
    const int d = p.geo.col(j0 + i);
    const bool in = c0 + d < cols;
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const float* q = src + k * step + d;
      const bool there = in && k * stride < rows;
      if (PIECE == 4) {
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        if (there) w = *reinterpret_cast<const float4*>(q);
        v[k][i] = w.x; v[k][i + 1] = w.y; v[k][i + 2] = w.z; v[k][i + 3] = w.w;
      } else {
        v[k][i] = there ? *q : 0.f;
      }
    }
  }
}

// A thread's share of a tile: four units of eight values that are neighbours in memory.  Unit u: rows 8 (u % 16) .. of
// window column u / 16 in a plane, window columns 8 (u % 8) .. of row u / 8 in the caller's rows.
constexpr int kCutThreads = 256, kUnits = kMmaRows * 8 / kCutThreads;
template <bool PLANE>
__device__ __forceinline__ void load_tile(const float* __restrict__ plane, const MmaRowsIO& io, const MmaPass& p, const Spot& at, int t, float (*v)[8]) {
  if (PLANE) {
    const float* src = plane + ((((int64_t)at.stack * p.nt + at.tile) << p.geo.log_nf) + at.cbase + p.geo.col(t >> 4)) * kMmaRows + (t & 15) * 8;
#pragma unroll
    for (int k = 0; k < kUnits; ++k) load8(src + p.geo.col(k * (kCutThreads / 16)) * kMmaRows, v[k]);
    return;
  }
  constexpr int stride = kCutThreads / 8;
  const int64_t r = (int64_t)at.tile * kMmaRows + (t >> 3), step = io.sB * stride, rows = p.B - r;
  const int j0 = (t & 7) * 8, cols = mma_cols(io, at.stack, p.geo.log_nf), c = at.cbase + p.geo.col(j0);
  const float* src = io.p + r * io.sB + at.stack * io.sS + at.cbase;
  if (p.geo.ib >= 3 && io.align >= 32 && cols % 8 == 0) {
#pragma unroll
    for (int k = 0; k < kUnits; ++k) {
      if (c < cols && k * stride < rows) {
        load8(src + p.geo.col(j0) + k * step, v[k]);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[k][i] = 0.f;
      }
    }
  } else if (p.geo.ib >= 2 && io.align >= 16 && cols % 4 == 0) {
    load_pieces<4, kUnits>(src, p, j0, at.cbase, cols, rows, step, stride, v);
  } else {
    load_pieces<1, kUnits>(src, p, j0, at.cbase, cols, rows, step, stride, v);
  }
}

// Operand of a tile in shared memory, 48 KB: from a plane [row half][slice][column][64 rows], from rows [slice][row][64
// columns]; 128-byte lines whose 16-byte chunks are swizzled.
constexpr uint32_t kOpBytes = 3 * kMmaRows * kMmaCols * 2;
template <bool PLANE> __device__ __forceinline__ void store_unit(uint8_t* op, int u, const float* v, uint32_t& probe) {
  uint4 s1, s2, s3;
  split8(v, s1, s2, s3, probe);
  uint8_t* d;
  constexpr int slice = PLANE ? 8192 : 16384;
  if (PLANE) {
    const int col = u >> 4, seg = u & 15;
    d = op + (seg >> 3) * 24576 + col * 128 + (((seg & 7) ^ (col & 7)) << 4);
  } else {
    const int row = u >> 3;
    d = op + row * 128 + (((u & 7) ^ (row & 7)) << 4);
  }
  *reinterpret_cast<uint4*>(d) = s1;
  *reinterpret_cast<uint4*>(d + slice) = s2;
  *reinterpret_cast<uint4*>(d + 2 * slice) = s3;
}

// rows x operator (TRANS: transposed operator).  Accumulators of 64 columns: slice 1 of the rows and part 1 of the operator,
// the largest products, into d, and behind them 12 21, 13 22 31 and 14 23 32, each about a 2^-5th to 2^-9th of the one
// before.  An instruction takes its operands' bytes / 128 clocks (measured: N = 64 48, 128 64, 192 96, so 256 128): 1152 for a tile.
template <bool PLANE, bool TRANS> __device__ __forceinline__ void issue_transform(uint32_t d, uint32_t op, uint32_t img) {
  constexpr uint32_t slice = PLANE ? 8192 : 16384;
  constexpr uint32_t i128 = mma_idesc(128, PLANE, TRANS), i192 = mma_idesc(192, PLANE, TRANS), i256 = mma_idesc(256, PLANE, TRANS);
  const uint64_t a0 = PLANE ? mma_desc(op, 24576, 1024) : mma_desc(op, 16, 1024);
  const uint64_t b0 = TRANS ? mma_desc(img, 8192, 1024) : mma_desc(img, 16, 1024);
  constexpr uint64_t as = slice >> 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const uint64_t a = a0 + k * ((PLANE ? 2048 : 32) >> 4), b = b0 + k * ((TRANS ? 2048 : 32) >> 4);
    mma_issue(d, a, b, i256, k > 0);
    mma_issue(d + 64, a + as, b, i192, true);
    mma_issue(d + 128, a + 2 * as, b, i128, true);
  }
}

// g^T x over the tile's rows, two slices of g stacked in the lanes.  Columns 0 .. of d: g1 x x1 of rows 0 .. 63 in the lower
// lanes, 64 .. the same of rows 64 .. 127 (what lands in the upper lanes, g2 x x1, is not used): short sums, taken out after
// every tile.  128 .. and 192 ..: all other products, g1|g2 x (x2|x3) and g2|g3 x x1, are 2^-8 as large and run on (`keep`).
// 1280 clocks for a tile.
template <bool GP, bool XP> __device__ __forceinline__ void issue_outer(uint32_t d, uint32_t g, uint32_t x, bool keep) {
  constexpr uint32_t i64 = mma_idesc(64, !GP, !XP), i128 = mma_idesc(128, !GP, !XP);
  constexpr uint64_t gs = (GP ? 8192 : 16384) >> 4, xs = (XP ? 8192 : 16384) >> 4;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t go = GP ? (k >> 2) * 24576 + (k & 3) * 32 : k * 2048, xo = XP ? (k >> 2) * 24576 + (k & 3) * 32 : k * 2048;
    const uint64_t a = mma_desc(g + go, GP ? 16 : 16384, 1024), b = mma_desc(x + xo, XP ? 16 : 16384, 1024);
    mma_issue(d + (k >> 2) * 64, a, b, i64, (k & 3) > 0);
    mma_issue(d + 128, a, b + xs, i128, keep || k > 0);
    mma_issue(d + 128, a + gs, b, i64, true);
  }
}

// Eight columns of what issue_transform left.
__device__ __forceinline__ void load_transform(uint32_t d, float* y) {
  float a[8], b[8], c[8];
  tmem_ld8(d, y);
  tmem_ld8(d + 64, a);
  tmem_ld8(d + 128, b);
  tmem_ld8(d + 192, c);
  wait_ld();
#pragma unroll
  for (int i = 0; i < 8; ++i) y[i] = (y[i] + (a[i] + (b[i] + c[i]))) * (1.f / ((int64_t)1 << 2 * kMmaScale));
}

// N results of a thread's row (window columns j0 ..) into a plane: a warp writes 128 bytes of a column at a time.
template <int N> __device__ __forceinline__ void store_plane(float* plane, const MmaPass& p, const Spot& at, int row, int j0, const float* y) {
  float* base = plane + ((((int64_t)at.stack * p.nt + at.tile) << p.geo.log_nf) + at.cbase + p.geo.col(j0)) * kMmaRows + row;
#pragma unroll
  for (int i = 0; i < N; ++i) base[p.geo.col(i) * kMmaRows] = y[i];
}

// The same into the caller's rows.  A warp's 32 rows turn through `turn` (16-byte chunks of N columns, swizzled) so that
// N / 4 lanes write 4 N neighbouring bytes of a row; straight from the registers every lane wrote 32 bytes of its own, and
// a tile took 3500 clocks.
template <int N> __device__ __forceinline__ void store_rows(const MmaRowsIO& io, const MmaPass& p, const Spot& at, int row0, int j0, const float* y,
                                                             uint8_t* turn, bool reduce, const float* bias) {
  constexpr int C = N / 4;  // chunks of a row
  const int lane = threadIdx.x & 31, cols = mma_cols(io, at.stack, p.geo.log_nf), chunk = lane % C;
  auto place = [](int r, int c) { return (r * C + (c ^ (C == 8 ? r & 7 : (r >> 1) & 3))) * 16; };
  if (C < 8 && p.geo.ib >= 3 && io.align >= 32 && !reduce && at.cbase + p.geo.col(j0 + N - 8) + 8 <= cols) {
    const int64_t r = (int64_t)at.tile * kMmaRows + row0 + lane;
    float* out = io.p + r * io.sB + at.stack * io.sS;
    if (r < p.B) {
#pragma unroll
      for (int h = 0; h < N; h += 8)
        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out + at.cbase + p.geo.col(j0 + h)), "f"(y[h]), "f"(y[h + 1]),
                     "f"(y[h + 2]), "f"(y[h + 3]), "f"(y[h + 4]), "f"(y[h + 5]), "f"(y[h + 6]), "f"(y[h + 7]) : "memory");
    }
    return;
  }
#pragma unroll
  for (int c = 0; c < C; ++c)
    *reinterpret_cast<float4*>(turn + place(lane, c)) = make_float4(y[4 * c], y[4 * c + 1], y[4 * c + 2], y[4 * c + 3]);
  __syncwarp();
  const int j = j0 + 4 * chunk, c0 = at.cbase + p.geo.col(j);
  const bool piece = p.geo.ib >= 2 && io.align >= 16 && c0 + 4 <= cols;
  float add[4] = {0.f, 0.f, 0.f, 0.f};
  if (bias) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t f = ((int64_t)at.stack << p.geo.log_nf) + at.cbase + p.geo.col(j + i);
      if (f < p.bias_len) add[i] = __ldg(bias + f);
    }
  }
  int64_t r = (int64_t)at.tile * kMmaRows + row0 + lane / C;
  float* out = io.p + r * io.sB + at.stack * io.sS;
#pragma unroll
  for (int k = 0; k < C; ++k, r += 32 / C, out += 32 / C * io.sB) {
    float4 v = *reinterpret_cast<const float4*>(turn + place(k * (32 / C) + lane / C, chunk));
    v.x += add[0]; v.y += add[1]; v.z += add[2]; v.w += add[3];
    if (r >= p.B) continue;
    if (piece) {
      if (reduce) asm volatile("red.global.v4.f32.add [%0], {%1, %2, %3, %4};" ::"l"(out + c0), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
      else *reinterpret_cast<float4*>(out + c0) = v;
    } else {
      const float w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int c = at.cbase + p.geo.col(j + i);
        if (c < cols) {
          if (reduce) atomicAdd(out + c, w[i]);
          else out[c] = w[i];
        }
      }
    }
  }
  __syncwarp();
}

// ------------------------------------------------------------------ passes
//
// One CTA per SM, its warps in three roles that hand tiles on through mbarriers: eight warps fetch tiles into registers and
// cut them into operand slices, one issues the matrix products, eight take the results out of tensor memory.  What a tile
// needs most after HBM is shared memory: of the backward's 4300 clocks (64 KB in and 32 KB out at an SM's share of HBM)
// the products take 2432 of its time and the writing of their operands 770.  So values go straight from registers into
// slices (through a staging copy in shared memory they would take 1020 clocks more: 180 us against 162 for a pass of
// 16384 x 4096), and all loads of an operand are issued at once (a register load waits on one of six counters, with
// whatever younger load shares it).  All warps through all steps, one after the other: 290 us.

constexpr int kCutWarps = kCutThreads / 32, kStoreWarps = 8;
constexpr int kStoreWarp0 = kCutWarps, kIssueWarp = kCutWarps + kStoreWarps;
constexpr int kPassThreads = 32 * (kIssueWarp + 4);  // whole warpgroups, which the register split asks for
// Row tiles after which the small products of the operator gradient are taken out too.  Every instruction cuts their sum, and a
// long sum of one sign loses 4.4e-9 of the whole per tile: 16384 rows of 4096 positive values, gradient of the factors 1.84e-7
// off after 32 tiles, 7.5e-8 after 8, 6.2e-8 after 4 (phases 1.3e-7), at the same time (924 us a training step).
constexpr int kFlushTiles = 4;
// Registers of a thread, by role.  All threads start with 96 (65536 / 640 in steps of eight); the shares add up to that.
constexpr int kCutRegs = 136, kStoreRegs = 88, kIssueRegs = 32;
static_assert(128 * (2 * kCutRegs + 2 * kStoreRegs + kIssueRegs) <= kPassThreads * 96, "register split");

// Shared memory: a pass has only the places that it uses.  Up to 195 KB leave 60 KB of the SM to the loads on their way, a
// few bytes more leave 28 (three backward passes of 16384 x 4096: 643 us so, 562 within).
template <bool BW, bool IN_P, bool OUT_P> struct PassMem {
  static constexpr int stages = 2;                // first operand; the backward's second has one place
  static constexpr uint32_t x = stages * kOpBytes;
  static constexpr uint32_t image = x + (BW ? kOpBytes : 0);
  static constexpr int turn_cols = BW ? 16 : 32;  // columns that turn at once on their way to the caller's rows
  static constexpr uint32_t turn = image + kMmaImageBytes;
  static constexpr uint32_t sums = turn + (OUT_P ? 0 : kStoreWarps * 32 * turn_cols * 4);
  static constexpr uint32_t control = sums + (BW && !IN_P ? kCutWarps * 64 * 4 : 0);
};
// Tensor memory: the transformed tile in 256 columns, twice in the forward; the operator gradient in 256.
constexpr uint32_t kOuterCol = 256;

struct Control {
  uint64_t gfull[2], gempty[2];  // operand tile (backward: first operand): written, read by the products
  uint64_t xfull;                // backward, second operand: written (read: pfull)
  uint64_t dfull[2], dempty[2];  // transformed tile in tensor memory: complete, taken out
  uint64_t pfull, pempty;        // operator gradient: complete for a tile, taken out
  uint64_t sync;                 // all warps that cut
  uint32_t tmem;
  int failed;                    // a wait ran out
};
template <typename M> constexpr uint32_t pass_bytes() { return M::control + (uint32_t)sizeof(Control); }

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Bounded; once a wait of any role has run out, all end.
__device__ __forceinline__ bool await(Control* ctl, uint64_t* bar, uint32_t parity) {
  const uint32_t b = smem_u32(bar);
  for (int i = 0; i < kTmaSpinLimit; ++i) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done) : "r"(b), "r"(parity) : "memory");
    if (done) return true;
    if ((i & 63) == 63 && *reinterpret_cast<volatile int*>(&ctl->failed)) return false;
  }
  *reinterpret_cast<volatile int*>(&ctl->failed) = 1;
  return false;
}
// The same for a whole warp, which goes on together.
__device__ __forceinline__ bool await_warp(Control* ctl, uint64_t* bar, uint32_t parity) { return __all_sync(0xffffffffu, await(ctl, bar, parity)); }
// All warps of a role; bounded like every other wait.
__device__ __forceinline__ bool role_sync(Control* ctl, uint64_t* bar, uint32_t& turn) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(bar);
  return await_warp(ctl, bar, turn++ & 1);
}

// The tiles of a CTA in order.
struct Walk {
  int64_t w, end;
  int block, nt, nq;
  Spot at;
  __device__ Walk(const MmaPass& p) : nt(p.nt), nq(p.nq) {
    const int sib = p.geo.sib, G = gridDim.x >> sib, c = blockIdx.x >> sib;
    const int64_t W = ((int64_t)p.S * p.nq >> sib) * p.nt;
    w = mma_first_tile(W, G, c);
    end = mma_first_tile(W, G, c + 1);
    block = ((int)(w / nt) << sib) + (blockIdx.x & ((1 << sib) - 1));
    at = Spot{block / nq, p.geo.base(block % nq), (int)(w % nt)};
  }
  __device__ bool more() const { return w < end; }
  __device__ bool last_of_part(const MmaParts& p) const { return at.tile + 1 == nt || w + 1 == end || p.ends(at.tile); }
  __device__ void next(const MmaPass& p) {
    ++w;
    if (++at.tile == nt) {
      block += 1 << p.geo.sib;
      at = Spot{block / nq, p.geo.base(block % nq), 0};
    }
  }
};

template <int REGS> __device__ __forceinline__ void registers_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS)); }
template <int REGS> __device__ __forceinline__ void registers_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS)); }

template <bool BW, bool IN_P, bool X_P, bool OUT_P>
__global__ void __launch_bounds__(kPassThreads, 1) bfly_mma_pass_kernel(const __grid_constant__ MmaPass p, int* err) {
  typedef PassMem<BW, IN_P, OUT_P> Mem;
  constexpr uint32_t DBUF = BW ? 1 : 2;      // transformed tiles tensor memory holds
  constexpr uint32_t ST = Mem::stages;
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t* img = sm + Mem::image;
  Control* ctl = reinterpret_cast<Control*>(sm + Mem::control);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (smem_u32(sm) & 1023) {  // what the swizzle of the operands counts from
    if (tid == 0) *err = 2;
    return;
  }
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&ctl->gfull[i]), kCutWarps);
      mbar_init(smem_u32(&ctl->gempty[i]), 1);
      mbar_init(smem_u32(&ctl->dfull[i]), 1);
      mbar_init(smem_u32(&ctl->dempty[i]), kStoreWarps);
    }
    mbar_init(smem_u32(&ctl->xfull), kCutWarps);
    mbar_init(smem_u32(&ctl->pfull), 1);
    mbar_init(smem_u32(&ctl->pempty), kStoreWarps);
    mbar_init(smem_u32(&ctl->sync), kCutWarps);
    ctl->failed = 0;
    if (BW && blockIdx.x == 0 && p.kept_flag && *p.kept_flag) *p.flag = 1;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kIssueWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&ctl->tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = __shfl_sync(0xffffffffu, ctl->tmem, 0);
  Walk at(p);

  if (warp < kCutWarps) {
    // ---------------- fetch, cut into slices
    registers_up<kCutRegs>();
    float bsum[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) bsum[i] = 0.f;
    uint32_t turn = 0, i = 0, probe = 0;
    int held = -1;       // block whose operator shared memory holds
    // Tile i, whose values are there: its place, and its operator if that is another than the last tile's.
    auto place = [&](int block) -> bool {
      const uint32_t s = i % ST;
      if (i >= ST && !await_warp(ctl, &ctl->gempty[s], (i / ST - 1) & 1)) return false;
      if (block != held) {  // the products with the former operator are done, and so is who else reads it
        if (i >= 1 && !await_warp(ctl, &ctl->gempty[(i - 1) % ST], ((i - 1) / ST) & 1)) return false;
        if (i >= 1 && !await_warp(ctl, &ctl->dempty[(i - 1) % DBUF], ((i - 1) / DBUF) & 1)) return false;
        const uint4* src = reinterpret_cast<const uint4*>(p.images + (int64_t)block * kMmaImageBytes);
#pragma unroll 2
        for (int k = tid; k < kMmaImageBytes / 16; k += kCutThreads) reinterpret_cast<uint4*>(img)[k] = __ldg(src + k);
        held = block;
      }
      return true;
    };
    auto cut = [&](auto plane, uint8_t* op, float (*v)[8], uint64_t* full) {
#pragma unroll
      for (int u = 0; u < kUnits; ++u) store_unit<decltype(plane)::value>(op, tid + u * kCutThreads, v[u], probe);
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(full);
    };
    float va[kUnits][8], vb[kUnits][8];
    if constexpr (!BW) {  // two tiles on their way
      Walk ahead(p);
      load_tile<IN_P>(p.in_t, p.in, p, ahead.at, tid, va);
      ahead.next(p);
      if (ahead.more()) load_tile<IN_P>(p.in_t, p.in, p, ahead.at, tid, vb);
      auto step = [&](float (*v)[8]) -> bool {
        if (!place(at.block)) return false;
        cut(std::integral_constant<bool, IN_P>(), sm + (i % ST) * kOpBytes, v, &ctl->gfull[i % ST]);
        at.next(p);
        ahead.next(p);
        if (ahead.more()) load_tile<IN_P>(p.in_t, p.in, p, ahead.at, tid, v);
        ++i;
        return at.more();
      };
      while (step(va) && step(vb)) {}
    } else {
      load_tile<IN_P>(p.in_t, p.in, p, at.at, tid, va);
      load_tile<X_P>(p.x_t, p.x, p, at.at, tid, vb);
      for (; at.more(); ++i) {
        if (!place(at.block)) break;
        const int block = at.block;
        const bool last = at.last_of_part(p.parts);
        const int part = p.parts.of(at.at.tile);
        at.next(p);
        uint8_t* op = sm + (i % ST) * kOpBytes;
        cut(std::integral_constant<bool, IN_P>(), op, va, &ctl->gfull[i % ST]);
        if (!IN_P) {
#pragma unroll
          for (int u = 0; u < kUnits; ++u)
#pragma unroll
            for (int e = 0; e < 8; ++e) bsum[e] += va[u][e];
        }
        if (at.more()) load_tile<IN_P>(p.in_t, p.in, p, at.at, tid, va);
        if (i >= 1 && !await_warp(ctl, &ctl->pfull, (i - 1) & 1)) break;
        cut(std::integral_constant<bool, X_P>(), sm + Mem::x, vb, &ctl->xfull);
        if (at.more()) load_tile<X_P>(p.x_t, p.x, p, at.at, tid, vb);
        if (!IN_P && last) {
          if (p.bias_slots) {  // column sums of the block's rows: this thread has columns 8 (tid % 8) ..
            float* sums = reinterpret_cast<float*>(sm + Mem::sums);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              bsum[e] += __shfl_xor_sync(0xffffffffu, bsum[e], 8);
              bsum[e] += __shfl_xor_sync(0xffffffffu, bsum[e], 16);
              if (lane < 8) sums[warp * 64 + lane * 8 + e] = bsum[e];
            }
            if (!role_sync(ctl, &ctl->sync, turn)) break;
            if (tid < 64) {
              float v = 0.f;
              for (int k = 0; k < kCutWarps; ++k) v += sums[k * 64 + tid];
              p.bias_slots[mma_slot(p.geo, p.parts, block, part, blockIdx.x >> p.geo.sib) * 64 + tid] = v;
            }
            if (!role_sync(ctl, &ctl->sync, turn)) break;
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) bsum[e] = 0.f;
        }
      }
    }
    if (beyond(probe)) *p.flag = 1;
  } else if (warp >= kIssueWarp) {
    registers_down<kIssueRegs>();
    // ---------------- issue the products
    if (warp != kIssueWarp) at.w = at.end;
    int kept = 0;  // tiles whose small products of the operator gradient tensor memory holds
    for (uint32_t i = 0; at.more(); ++i) {
      const uint32_t d = i % DBUF, s = i % ST, op = smem_u32(sm) + s * kOpBytes;
      if (!await_warp(ctl, &ctl->gfull[s], (i / ST) & 1)) break;
      if (i >= DBUF && !await_warp(ctl, &ctl->dempty[d], (i / DBUF - 1) & 1)) break;
      fence_after_sync();
      issue_transform<IN_P, BW>(tmem + d * 256, op, smem_u32(img));
      mma_commit(smem_u32(&ctl->dfull[d]));
      if (BW) {
        if (!await_warp(ctl, &ctl->xfull, i & 1)) break;
        if (i >= 1 && !await_warp(ctl, &ctl->pempty, (i - 1) & 1)) break;
        fence_after_sync();
        issue_outer<IN_P, X_P>(tmem + kOuterCol, op, smem_u32(sm + Mem::x), kept > 0);
        mma_commit(smem_u32(&ctl->pfull));
        kept = kept + 1 == kFlushTiles || at.last_of_part(p.parts) ? 0 : kept + 1;
      }
      mma_commit(smem_u32(&ctl->gempty[s]));
      at.next(p);
    }
  } else {
    // ---------------- take the results out
    registers_down<kStoreRegs>();
    const int e = warp - kStoreWarp0, row = (e & 3) * 32 + lane, j0 = (e >> 2) * 32;
    const uint32_t lanes = (uint32_t)((e & 3) * 32) << 16;
    float acc[BW ? 32 : 1];  // operator gradient: row `row` (two slices of the incoming gradient), columns j0 ..
#pragma unroll
    for (int i = 0; i < (BW ? 32 : 1); ++i) acc[i] = 0.f;
    if (BW && p.parts.begins(at.at.tile)) {  // a free slot in front
      const int64_t free = mma_slot(p.geo, p.parts, at.block, p.parts.of(at.at.tile) - 1, blockIdx.x >> p.geo.sib);
      float* dst = p.slots + free * kMmaSlotFloats + row * kMmaCols + j0;
#pragma unroll
      for (int c = 0; c < 32; c += 4) *reinterpret_cast<float4*>(dst + c) = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.bias_slots && e == 0) {
        p.bias_slots[free * kMmaCols + lane] = 0.f;
        p.bias_slots[free * kMmaCols + lane + 32] = 0.f;
      }
    }
    int kept = 0;
    for (uint32_t i = 0; at.more(); ++i) {
      const uint32_t d = i % DBUF;
      if (!await_warp(ctl, &ctl->dfull[d], (i / DBUF) & 1)) break;
      fence_after_sync();
      const Spot now = at.at;
      constexpr int NY = Mem::turn_cols;  // columns of a row at a time (the backward has no registers for all 32)
#pragma unroll
      for (int c0 = 0; c0 < 32; c0 += NY) {
        float y[NY];
#pragma unroll
        for (int h = 0; h < NY; h += 8) load_transform(tmem + d * 256 + lanes + j0 + c0 + h, y + h);
        if (c0 + NY == 32) {
          fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(&ctl->dempty[d]);
        }
        if (OUT_P) store_plane<NY>(p.out_t, p, now, row, j0 + c0, y);
        else store_rows<NY>(p.out, p, now, row - lane, j0 + c0, y, sm + Mem::turn + e * 32 * NY * 4, BW && p.reduce != 0, BW ? nullptr : p.bias);
      }
      if (BW) {
        if (!await_warp(ctl, &ctl->pfull, i & 1)) break;
        fence_after_sync();
        const bool last = at.last_of_part(p.parts), flush = ++kept == kFlushTiles || last;
        auto take = [&](uint32_t col, bool use) {  // (all warps together: a branch around the loads cost 30 us of 560)
#pragma unroll
          for (int h = 0; h < 4; ++h) {
            float v[8], w[8];
            tmem_ld8(tmem + kOuterCol + col + lanes + j0 + 8 * h, v);
            tmem_ld8(tmem + kOuterCol + col + 64 + lanes + j0 + 8 * h, w);
            wait_ld();
#pragma unroll
            for (int c = 0; c < 8; ++c)
              if (use) acc[BW ? 8 * h + c : 0] += v[c] + w[c];
          }
        };
        take(0, row < kMmaCols);
        if (flush) {
          kept = 0;
          take(128, true);
        }
        fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&ctl->pempty);
        if (last) {  // the part's last tile here: leave its sums
          float* dst = p.slots + mma_slot(p.geo, p.parts, at.block, p.parts.of(at.at.tile), blockIdx.x >> p.geo.sib) * kMmaSlotFloats + row * kMmaCols + j0;
#pragma unroll
          for (int c = 0; c < (BW ? 32 : 0); c += 4) *reinterpret_cast<float4*>(dst + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
#pragma unroll
          for (int c = 0; c < (BW ? 32 : 1); ++c) acc[c] = 0.f;
        }
      }
      at.next(p);
    }
  }
  fence_before_sync();
  __syncthreads();
  if (tid == 0 && ctl->failed) *err = 1;
  if (warp == kIssueWarp) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

// ------------------------------------------------------------------ operators and their gradients

struct cd { double re, im; };
constexpr double kKept = (double)(1ll << 40);  // products of some factors, below 2^20, keep 24 bits down to 2^-166
template <bool CPLX> struct Num;
template <> struct Num<false> {
  typedef double T; typedef float S;
  static constexpr int W = 64;
  static __device__ double one(bool o) { return o ? 1.0 : 0.0; }
  static __device__ double up(float a) { return a; }
  static __device__ float down(double a) { return (float)a; }
  static __device__ double times(double a, double s) { return a * s; }
  static __device__ double fma(double a, double b, double c) { return ::fma(a, b, c); }   // a b + c
  static __device__ double fmac(double a, double b, double c) { return ::fma(a, b, c); }  // conj(a) b + c
  static __device__ bool below(double a, double most) { return fabs(a) < most; }
  static __device__ double zero() { return 0.0; }
  static __device__ double add(double a, double b) { return a + b; }
  static __device__ double shuffle(double v, int h) { return __shfl_xor_sync(0xffffffffu, v, h); }
};
template <> struct Num<true> {
  typedef cd T; typedef float2 S;
  static constexpr int W = 32;
  static __device__ cd one(bool o) { return cd{o ? 1.0 : 0.0, 0.0}; }
  static __device__ cd up(float2 a) { return cd{a.x, a.y}; }
  static __device__ float2 down(cd a) { return make_float2((float)a.re, (float)a.im); }
  static __device__ cd times(cd a, double s) { return cd{a.re * s, a.im * s}; }
  static __device__ cd fma(cd a, cd b, cd c) { return cd{::fma(a.re, b.re, ::fma(-a.im, b.im, c.re)), ::fma(a.re, b.im, ::fma(a.im, b.re, c.im))}; }
  static __device__ cd fmac(cd a, cd b, cd c) { return cd{::fma(a.re, b.re, ::fma(a.im, b.im, c.re)), ::fma(a.re, b.im, ::fma(-a.im, b.re, c.im))}; }
  static __device__ bool below(cd a, double most) { return fabs(a.re) < most && fabs(a.im) < most; }
  static __device__ cd zero() { return cd{0.0, 0.0}; }
  static __device__ cd add(cd a, cd b) { return cd{a.re + b.re, a.im + b.im}; }
  static __device__ cd shuffle(cd v, int h) { return cd{__shfl_xor_sync(0xffffffffu, v.re, h), __shfl_xor_sync(0xffffffffu, v.im, h)}; }
};

// Threads of the operator kernels: a warp takes a unit of a factor (W / radix of them), its lanes the columns.  A radix-4
// factor needs too many registers for 1024 threads.
__host__ __device__ constexpr int op_threads(bool cplx, bool four) { return cplx || four ? 512 : 1024; }

// First window row of unit u of a factor, and where its twiddles are.
__device__ __forceinline__ int unit_row(int lbit, int radix, int u) { return insert_zeros(u, lbit, radix == 4 ? 2 : 1); }
template <bool CPLX> __device__ __forceinline__ int64_t unit_twiddle(const MmaStage& m, const MmaGeom& geo, int cbase, int row) {
  const int c = (cbase + geo.col(row << (CPLX ? 1 : 0))) >> (CPLX ? 1 : 0);
  return (int64_t)m.tw_off + (m.radix == 4 ? (int64_t)delete_2bits(c, m.gbit) * 16 : (int64_t)delete_bit(c, m.gbit) * 4);
}

// Twiddles of all factors of a block, side by side in shared memory in float64: one trip to memory instead of one per
// factor.  A radix-2 factor has 2 W entries in a block, a radix-4 factor 4 W and counts as two.
template <bool CPLX>
__device__ void gather_twiddles(typename Num<CPLX>::T* dst, const MmaGroup& g, int cbase, int stack, const void* const* tw, const int64_t* tw_stack) {
  typedef typename Num<CPLX>::S S;
  constexpr int W = Num<CPLX>::W;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int k = 0, off = 0; k < g.nst; ++k) {
    const MmaStage m = g.st[k];
    const int count = W * m.radix, lg = m.radix == 4 ? 4 : 2;
    if (k % (blockDim.x / 32) == warp) {  // a warp to a factor, its loads together
      const S* src = static_cast<const S*>(tw[m.which]) + (int64_t)stack * tw_stack[m.which];
#pragma unroll 4
      for (int i = lane; i < count; i += 32)
        dst[off + i] = Num<CPLX>::up(src[unit_twiddle<CPLX>(m, g.geo, cbase, unit_row(m.lbit, m.radix, i >> lg)) + (i & ((1 << lg) - 1))]);
    }
    off += count;
  }
}

// work (W x W) <- factor x work, and a float32 copy of it times kKept (keep may be null); are the results below 2^kMmaOpBits?
template <bool CPLX, int RAD>
__device__ __forceinline__ bool apply_stage(typename Num<CPLX>::T* work, int lbit, const typename Num<CPLX>::T* tw, typename Num<CPLX>::S* keep) {
  typedef Num<CPLX> N;
  constexpr int W = N::W;
  const int lane = threadIdx.x & 31, d = W << lbit;
  bool fine = true;
  for (int u = threadIdx.x >> 5; u < W / RAD; u += blockDim.x >> 5) {
    typename N::T t[RAD * RAD];
#pragma unroll
    for (int i = 0; i < RAD * RAD; ++i) t[i] = tw[u * RAD * RAD + i];
    const int at = unit_row(lbit, RAD, u) * W + lane;
#pragma unroll
    for (int c = at; c < at + W; c += 32) {
      typename N::T x[RAD];
#pragma unroll
      for (int i = 0; i < RAD; ++i) x[i] = work[c + i * d];
#pragma unroll
      for (int o = 0; o < RAD; ++o) {
        typename N::T a = N::zero();
#pragma unroll
        for (int i = 0; i < RAD; ++i) a = N::fma(t[o * RAD + i], x[i], a);
        work[c + o * d] = a;
        fine &= N::below(a, (double)(1 << kMmaOpBits));
        if (keep) keep[c + o * d] = N::down(N::times(a, kKept));
      }
    }
  }
  return fine;
}
template <bool CPLX, bool FOUR>
__device__ __forceinline__ bool apply_stage(typename Num<CPLX>::T* work, const MmaStage& m, const typename Num<CPLX>::T* tw, typename Num<CPLX>::S* keep) {
  return FOUR && m.radix == 4 ? apply_stage<CPLX, 4>(work, m.lbit, tw, keep) : apply_stage<CPLX, 2>(work, m.lbit, tw, keep);
}

// Latency: at most twelve short stages with a barrier each; blocks of all groups run side by side.
template <bool CPLX, bool FOUR>
__global__ void __launch_bounds__(op_threads(CPLX, FOUR)) bfly_mma_prep_kernel(const __grid_constant__ MmaPrep p) {
  typedef Num<CPLX> N;
  constexpr int W = N::W, T = op_threads(CPLX, FOUR);
  __shared__ typename N::T work[W * W];
  __shared__ typename N::T tw[kMmaMaxStages * 2 * W];
  const MmaGroup& g = p.g[blockIdx.z];
  const int q = blockIdx.x, s = blockIdx.y, cbase = g.geo.base(q);
  gather_twiddles<CPLX>(tw, g, cbase, s, p.tw, p.tw_stack);
  for (int i = threadIdx.x; i < W * W; i += T) work[i] = N::one(i / W == i % W);
  __syncthreads();
  bool fine = true;
  for (int k = 0, off = 0; k < g.nst; ++k) {
    const MmaStage m = g.st[k];
    fine &= apply_stage<CPLX, FOUR>(work, m, tw + off, (typename N::S*)nullptr);
    off += W * m.radix;
    __syncthreads();
  }
  if (!fine) *p.flag = 1;
  // Parts of an entry v (scaled): v to a multiple of 2^(E - 3), where 2^E is at most the largest entry of its row or its column, the
  // larger of the two (exact sums, see above), and three bfloat16 slices of the rest.
  __shared__ int top[2][kMmaCols];  // exponents of the largest entries of a row, a column
  auto entry = [&](int j, int i) -> double {
    if constexpr (CPLX) {
      const cd z = work[(j >> 1) * W + (i >> 1)];
      return ((j & 1) == (i & 1) ? z.re : ((j & 1) ? z.im : -z.im)) * (1 << kMmaScale);
    } else {
      return work[j * W + i] * (1 << kMmaScale);
    }
  };
  if (threadIdx.x < 2 * kMmaCols) top[threadIdx.x / kMmaCols][threadIdx.x % kMmaCols] = -1100;
  __syncthreads();
  static_assert(T % kMmaCols == 0 && kMmaCols % 32 == 0, "a thread stays in its column, a warp in a row");
  int column = -1100;
  for (int it = threadIdx.x; it < kMmaCols * kMmaCols; it += T) {
    const int e = ((__double2hiint(entry(it / kMmaCols, it % kMmaCols)) >> 20) & 0x7ff) - 1023, row = __reduce_max_sync(0xffffffffu, e);
    column = max(column, e);
    if ((threadIdx.x & 31) == 0) atomicMax(&top[0][it / kMmaCols], row);
  }
  atomicMax(&top[1][threadIdx.x % kMmaCols], column);
  __syncthreads();
  uint8_t* img = p.images + (((int64_t)blockIdx.z * p.S + s) * p.nq + q) * kMmaImageBytes;
  for (int it = threadIdx.x; it < kMmaCols * 8; it += T) {
    const int j = it >> 3, ch = it & 7;
    uint32_t sl[kMmaParts][4];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int i = ch * 8 + e, E = min(max(max(top[0][j], top[1][i]), -120), 120);
      double left = entry(j, i);
#pragma unroll
      for (int k = 0; k < kMmaParts; ++k) {
        float f = (float)left;
        if (k == 0) f = (float)(rint(left * __hiloint2double((1023 + 3 - E) << 20, 0)) * __hiloint2double((1023 - 3 + E) << 20, 0));
        uint32_t r;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(0.f), "f"(f));
        left -= (double)__uint_as_float(r << 16);
        sl[k][e >> 1] = (e & 1) ? sl[k][e >> 1] | (r << 16) : (r & 0xffffu);
      }
    }
#pragma unroll
    for (int k = 0; k < kMmaParts; ++k)
      *reinterpret_cast<uint4*>(img + k * 8192 + j * 128 + ((ch ^ (j & 7)) << 4)) = make_uint4(sl[k][0], sl[k][1], sl[k][2], sl[k][3]);
  }
}

// Sums over a warp of N values each: value i ends up in the lanes whose number is i modulo N.  Every exchange halves the
// values a lane still holds.
template <bool CPLX, int N> __device__ __forceinline__ typename Num<CPLX>::T warp_sums(typename Num<CPLX>::T* a) {
  typedef Num<CPLX> M;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int h = N / 2; h; h >>= 1) {
    const bool upper = lane & h;
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const typename M::T give = upper ? a[i] : a[i + h], hold = upper ? a[i + h] : a[i];
      a[i] = M::add(hold, M::shuffle(give, h));
    }
  }
  typename M::T v = a[0];
#pragma unroll
  for (int h = N; h < 32; h <<= 1) v = M::add(v, M::shuffle(v, h));
  return v;
}

// One factor of the way back: its gradient (G R^H) where it has entries, and G <- (factor)^H G.
template <bool CPLX, int RAD>
__device__ __forceinline__ void unstack_stage(typename Num<CPLX>::T* G, const typename Num<CPLX>::S* R, const MmaStage& m, const MmaGeom& geo, int cbase,
                                              const typename Num<CPLX>::T* tw, typename Num<CPLX>::S* dtw) {
  typedef Num<CPLX> N;
  typedef typename N::T T;
  constexpr int W = N::W;
  const int lane = threadIdx.x & 31, d = W << m.lbit;
  for (int u = threadIdx.x >> 5; u < W / RAD; u += blockDim.x >> 5) {
    const int r0 = unit_row(m.lbit, RAD, u), at = r0 * W + lane;
    T a[RAD * RAD];
#pragma unroll
    for (int i = 0; i < RAD * RAD; ++i) a[i] = N::zero();
#pragma unroll
    for (int c = 0; c < W; c += 32) {
      T g[RAD], r[RAD];
#pragma unroll
      for (int i = 0; i < RAD; ++i) {
        g[i] = G[at + c + i * d];
        r[i] = R ? N::times(N::up(R[at + c + i * d]), 1.0 / kKept) : N::one(r0 + (i << m.lbit) == c + lane);
      }
#pragma unroll
      for (int o = 0; o < RAD; ++o)
#pragma unroll
        for (int i = 0; i < RAD; ++i)
          a[o * RAD + i] = N::fmac(r[i], g[o], a[o * RAD + i]);
      if (R) {
#pragma unroll
        for (int i = 0; i < RAD; ++i) {
          T t = N::zero();
#pragma unroll
          for (int o = 0; o < RAD; ++o) t = N::fmac(tw[(u * RAD + o) * RAD + i], g[o], t);
          G[at + c + i * d] = t;
        }
      }
    }
    const T v = warp_sums<CPLX, RAD * RAD>(a);
    if (lane < RAD * RAD) dtw[unit_twiddle<CPLX>(m, geo, cbase, r0) + lane] = N::down(v);
  }
}

// Gradients of a group's factors from the gradient of their product, for one block: with R the product of the factors
// before a factor and G the gradient of the product up to it, its own gradient is (G R^H) where it has entries, and G
// continues as (factor)^H G.  R before every factor is kept (float32, times kKept); G runs in float64.
template <bool CPLX, bool FOUR>
__global__ void __launch_bounds__(op_threads(CPLX, FOUR)) bfly_mma_post_kernel(const __grid_constant__ MmaPost p) {
  typedef Num<CPLX> N;
  typedef typename N::T T;
  typedef typename N::S S;
  constexpr int W = N::W, THREADS = op_threads(CPLX, FOUR);
  extern __shared__ __align__(16) uint8_t raw[];
  T* G = reinterpret_cast<T*>(raw);
  T* tw = G + W * W;
  S* R = reinterpret_cast<S*>(tw + kMmaMaxStages * 2 * W);  // before factor k: R + (k - 1) W W
  const MmaGroup& g = p.g[blockIdx.z];
  const int q = blockIdx.x, s = blockIdx.y, cbase = g.geo.base(q), tid = threadIdx.x;
  // what the CTAs of the backward pass left for this block; on its way while R is made
  const int sib = g.geo.sib, ctas = (p.ctas >> sib);
  const int64_t block = (int64_t)s * p.nq + q, first = (block >> sib) * p.nt, tiles = ((int64_t)p.S * p.nq >> sib) * p.nt;
  const int64_t slot0 = mma_slot(g.geo, p.parts, block, 0, mma_cta_of(tiles, ctas, first));
  const int64_t slot1 = mma_slot(g.geo, p.parts, block, p.parts.of(p.nt - 1), mma_cta_of(tiles, ctas, first + p.nt - 1));
  constexpr int PER = kMmaCols * kMmaCols / THREADS;  // entries of a thread, neighbours
  const float* slots = p.slots + p.group[blockIdx.z] * p.slots_group + slot0 * kMmaSlotFloats + tid * PER;
  double sum[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) sum[i] = 0.0;
#pragma unroll 2
  for (int64_t slot = slot0; slot <= slot1; slot += 1 << sib, slots += kMmaSlotFloats << sib) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < PER; i += 4) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(slots + h * kMmaCols * kMmaCols + i));
        sum[i] += (double)v.x; sum[i + 1] += (double)v.y; sum[i + 2] += (double)v.z; sum[i + 3] += (double)v.w;
      }
  }
  bool fine = true;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    fine &= isfinite(sum[i]);
    sum[i] *= 1.0 / ((int64_t)1 << 2 * kMmaScale);
  }
  if (!fine) *p.flag = 1;
  gather_twiddles<CPLX>(tw, g, cbase, s, p.tw, p.tw_stack);
  for (int i = tid; i < W * W; i += THREADS) G[i] = N::one(i / W == i % W);
  __syncthreads();
  int off = 0;
  for (int k = 0; k + 1 < g.nst; ++k) {
    const MmaStage m = g.st[k];
    apply_stage<CPLX, FOUR>(G, m, tw + off, R + k * W * W);
    off += W * m.radix;
    __syncthreads();
  }
  if constexpr (CPLX) {  // a thread holds eight columns of one real row; the two rows of a complex one are 64 / 8 threads apart
    cd z[PER / 2];
#pragma unroll
    for (int i = 0; i < PER / 2; ++i) {
      const double re = sum[2 * i], im = sum[2 * i + 1], re2 = __shfl_xor_sync(0xffffffffu, re, kMmaCols / PER), im2 = __shfl_xor_sync(0xffffffffu, im, kMmaCols / PER);
      z[i] = cd{re + im2, re2 - im};  // (row, row) + (row + 1, row + 1), (row + 1, row) - (row, row + 1) in the even row
    }
    const int row = tid * PER / kMmaCols, col = tid * PER % kMmaCols / 2;
    if (row % 2 == 0)
#pragma unroll
      for (int i = 0; i < PER / 2; ++i) G[row / 2 * W + col + i] = ((row / 2) ^ (col + i)) & g.passive ? N::zero() : z[i];
  } else {
    const int row = tid * PER / W, col = tid * PER % W;
#pragma unroll
    for (int i = 0; i < PER; ++i) G[row * W + col + i] = (row ^ (col + i)) & g.passive ? N::zero() : sum[i];  // (columns no factor brings together)
  }
  if (p.bias_slots && p.group[blockIdx.z] == p.last_group && tid < kMmaCols) {
    double v = 0.0;
    for (int64_t slot = slot0; slot <= slot1; slot += 1 << sib) v += (double)p.bias_slots[slot * kMmaCols + tid];
    const int64_t f = ((int64_t)s << g.geo.log_nf) + cbase + g.geo.col(tid);
    if (f < p.dbias_len) p.dbias[f] = (float)v;
  }
  __syncthreads();
  for (int k = g.nst - 1; k >= 0; --k) {
    const MmaStage m = g.st[k];
    S* dtw = static_cast<S*>(p.dtw[m.which]) + (int64_t)s * p.tw_stack[m.which];
    const S* Rk = k > 0 ? R + (k - 1) * W * W : nullptr;
    if (FOUR && m.radix == 4) unstack_stage<CPLX, 4>(G, Rk, m, g.geo, cbase, tw + off, dtw);
    else unstack_stage<CPLX, 2>(G, Rk, m, g.geo, cbase, tw + off, dtw);
    if (k > 0) off -= W * g.st[k - 1].radix;
    __syncthreads();
  }
}

// ------------------------------------------------------------------ launches

// Room for `bytes` of dynamic shared memory, the most that any launch of the kernel asks for: set once per device, since
// threads with launches of different sizes would undo one another's setting.
struct SmemOnce {
  std::mutex mu;
  bool done[64] = {false};
  template <typename K> int operator()(K kernel, uint32_t bytes) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return BFLY_E_NODEVICE;
    std::lock_guard<std::mutex> lk(mu);
    if (done[dev]) return BFLY_OK;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) {
      cudaGetLastError();
      return BFLY_E_CUDA;
    }
    done[dev] = true;
    return BFLY_OK;
  }
};
int launched() { return cudaGetLastError() == cudaSuccess ? BFLY_OK : BFLY_E_CUDA; }

template <bool BW, bool IN_P, bool X_P, bool OUT_P> int pass_launch(const MmaPass& p, int ctas, cudaStream_t stream, int* err) {
  constexpr uint32_t bytes = pass_bytes<PassMem<BW, IN_P, OUT_P>>();
  static_assert(bytes <= 227 * 1024, "shared memory of a CTA");
  static SmemOnce smem;
  if (int rc = smem(bfly_mma_pass_kernel<BW, IN_P, X_P, OUT_P>, bytes)) return rc;
  bfly_mma_pass_kernel<BW, IN_P, X_P, OUT_P><<<ctas, kPassThreads, bytes, stream>>>(p, err);
  return launched();
}

// `stages`: most factors of a group, whose products the kernel keeps.
template <bool CPLX, bool FOUR> int post_launch(const MmaPost& p, int stages, cudaStream_t stream) {
  constexpr int W = Num<CPLX>::W, size = CPLX ? 8 : 4;
  auto bytes = [](int stages) { return (uint32_t)(size * (2 * W * W + 2 * kMmaMaxStages * 2 * W + (stages - 1) * W * W)); };
  static SmemOnce smem;
  if (int rc = smem(bfly_mma_post_kernel<CPLX, FOUR>, bytes(kMmaMaxStages))) return rc;
  bfly_mma_post_kernel<CPLX, FOUR><<<dim3(p.nq, p.S, p.ng), op_threads(CPLX, FOUR), bytes(stages), stream>>>(p);
  return launched();
}

}  // namespace

static bool has_radix4(const MmaGroup* g, int n) {
  for (int i = 0; i < n; ++i)
    for (int k = 0; k < g[i].nst; ++k)
      if (g[i].st[k].radix == 4) return true;
  return false;
}

int mma_prep_launch(const MmaPrep& p, bool cplx, cudaStream_t stream) {
  const dim3 grid(p.nq, p.S, p.ng);
  const bool four = has_radix4(p.g, p.ng);
  if (cplx) bfly_mma_prep_kernel<true, true><<<grid, op_threads(true, true), 0, stream>>>(p);
  else if (four) bfly_mma_prep_kernel<false, true><<<grid, op_threads(false, true), 0, stream>>>(p);
  else bfly_mma_prep_kernel<false, false><<<grid, op_threads(false, false), 0, stream>>>(p);
  return launched();
}

int mma_fw_launch(const MmaPass& p, int sms, cudaStream_t stream, int* err) {
  const int ctas = mma_ctas(p.geo, (int64_t)p.S * p.nq * p.nt, sms);
  if (p.in_t) return p.out_t ? pass_launch<false, true, false, true>(p, ctas, stream, err) : pass_launch<false, true, false, false>(p, ctas, stream, err);
  return p.out_t ? pass_launch<false, false, false, true>(p, ctas, stream, err) : pass_launch<false, false, false, false>(p, ctas, stream, err);
}

int mma_bw_launch(const MmaPass& p, int most, cudaStream_t stream, int* err) {
  const int ctas = mma_ctas(p.geo, (int64_t)p.S * p.nq * p.nt, most);
  if (p.in_t && p.x_t && p.out_t) return pass_launch<true, true, true, true>(p, ctas, stream, err);
  if (p.in_t && !p.x_t && !p.out_t) return pass_launch<true, true, false, false>(p, ctas, stream, err);
  if (!p.in_t && p.x_t && p.out_t) return pass_launch<true, false, true, true>(p, ctas, stream, err);
  if (!p.in_t && !p.x_t && !p.out_t) return pass_launch<true, false, false, false>(p, ctas, stream, err);
  return BFLY_E_ARG;
}

// Groups of few factors need less shared memory (two CTAs to an SM up to seven), so they go in a launch of their own.
int mma_post_launch(const MmaPost& all, bool cplx, cudaStream_t stream, int* launches) {
  for (int many = 1; many >= 0; --many) {
    MmaPost p = all;
    p.ng = 0;
    int stages = 1;
    for (int i = 0; i < all.ng; ++i)
      if ((all.g[i].nst > 7) == (many != 0)) {
        p.group[p.ng] = i;
        p.g[p.ng++] = all.g[i];
        stages = std::max(stages, all.g[i].nst);
      }
    if (!p.ng) continue;
    const int rc = cplx ? post_launch<true, true>(p, stages, stream)
                   : has_radix4(p.g, p.ng) ? post_launch<false, true>(p, stages, stream) : post_launch<false, false>(p, stages, stream);
    if (rc) return rc;
    ++*launches;
  }
  return BFLY_OK;
}

}  // namespace bfly
