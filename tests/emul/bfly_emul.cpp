// Test helper, not product code: runs the CUDA kernels' per-thread tile routines on the
// host, one simulated thread at a time, behind the same driver that plans the GPU
// launches.  It exists to check planning and index arithmetic on a machine without a
// GPU; the shipped library never falls back to it.
//
// Build: g++ -O2 -std=c++17 -fPIC -shared -I butterfly_b200/csrc tests/emul/bfly_emul.cpp -o tests/emul/libbfly_emul.so
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "bfly_core.h"
#include "bfly_bw2.h"
#include "bfly_bw3.h"
#include "bfly_driver.h"
#include "bfly_glue.h"

using namespace bfly;

namespace {

long g_fw2_calls = 0;  // launches the emulator ran through the packed-pair forward path
long g_bw3_calls = 0;  // ... and through the packed-pair backward phase path

// The accumulators of every sub-group and thread, summed two by two over the thread bits of mask(j) (fold_threads).
template <int N, typename T = float, typename MASK, typename LD>
std::vector<T> fold_rows(int nsg, int nthr, MASK mask, LD ld) {
  std::vector<T> w((size_t)nsg * nthr * N);
  for (int j = 0; j < nsg; ++j) {
    T* a = &w[(size_t)j * nthr * N];
    for (int tid = 0; tid < nthr; ++tid) ld(j, tid, a + (size_t)tid * N);
    for (int b = 1; b < nthr; b <<= 1)
      if (mask(j) & b)
        for (int tid = 0; tid < nthr; ++tid)
          if (!(tid & b))
            for (int k = 0; k < N; ++k)
              a[(size_t)tid * N + k] = a[(size_t)(tid ^ b) * N + k] = add1(a[(size_t)tid * N + k], a[(size_t)(tid ^ b) * N + k]);
  }
  return w;
}

struct EmulExec {
  int sms = 7;       // odd on purpose: exercises ragged row slices
  int threads_ = 64;  // simulated block size (any power of two)
  int num_sms() const { return sms; }
  int threads() const { return threads_; }
  bool bw2 = true;   // exercise the second-generation backward where the driver selects it
  bool has_bw2(size_t /*elem_size*/, int kw) const { return bw2 && kw == 2; }

  // packed-pair forward kernel: boxes copied by plain loops, groups run thread by thread in plan
  // order (a valid schedule of the device kernel's barriers)
  bool fw2 = true;
  int run_fw2(const Fw2Params& p_in, int /*ctas_per_sm*/) {
    if (!fw2) return kFw2Declined;
    Fw2Params p = p_in;
    const int n = 1 << p.log_n;
    if (p.view && ((p.panel.lseg != p.panel.logC && p.panel.lseg != 5) || p.bias)) return kFw2Declined;
    if (p.x_cols < n && (p.x_cols < 32 || p.x_cols % 4 != 0)) return kFw2Declined;  // what the descriptors and the cut block's copies refuse
    if (p.out && p.out_cols % 32 != 0) return kFw2Declined;
    p.has_out = p.out != nullptr;
    if (!p.has_out) p.out_cols = n;
    ++g_fw2_calls;
    for (int64_t e = 0; e < fw2_pack_entries(p); ++e) fw2_pack_one(p, e);  // the re-ordering kernel
    std::vector<float> tile((size_t)p.R * n);
    const int64_t ntiles = fw2_num_tiles(p);
    auto box_copy = [&](bool load, const float* src, float* dst, int64_t sB, int64_t sS, int cols, int stack, int row0) {
      for (int r = 0; r < p.R; ++r)
        for (int c = 0; c < n; ++c) {
          float& t = tile[fw2_tile_index(p.R, r, c)];
          const int row = row0 + r;
          const bool in = row < p.B && c < cols;
          // a panel view addresses (panel, local column) -> real column of the one real stack
          const int64_t at = p.view ? (int64_t)row * sB + fw2_view_col(p, stack, c) : (int64_t)row * sB + (int64_t)stack * sS + c;
          if (load) t = in ? src[at] : 0.f;
          else if (in) dst[at] = t;
        }
    };
    for (int64_t t = 0; t < ntiles; ++t) {
      const int stack = (int)(t % p.S), row0 = (int)(t / p.S) * p.R;
      box_copy(true, p.x, nullptr, p.x_sB, p.x_sS, std::min(p.x_cols, n), stack, row0);
      for (int gi = 0; gi < p.ngroups; ++gi) {
        for (int tid = 0; tid < fw2_threads(p); ++tid) {
          f2 T[48];
          fw2_fetch_tw(p, p.g[gi], stack, tid, T);
          if (tid & 1) fw2_group_dispatch<true>(p, p.g[gi], tile.data(), tid, T);  // both row-loop forms
          else fw2_group_dispatch<false>(p, p.g[gi], tile.data(), tid, T);
        }
        if (p.g[gi].emit) box_copy(false, nullptr, p.snap[p.g[gi].emit - 1], p.view ? (int64_t)p.view_row : (int64_t)p.S * n, n, n, stack, row0);
      }
      if (p.has_out && p.bias)  // the store epilogue of the device kernel
        for (int r = 0; r < p.R; ++r)
          for (int c = 0; c < n; ++c)
            if (stack * n + c < p.bias_len) tile[fw2_tile_index(p.R, r, c)] += p.bias[stack * n + c];
      if (p.has_out) box_copy(false, nullptr, p.out, p.out_sB, p.out_sS, p.out_cols, stack, row0);
    }
    return BFLY_OK;
  }

  // packed-pair backward phase: the device kernel's steps, thread by thread, accumulators in a heap array
  bool bw3 = true;
  bool can_run_bw3(const Bw3Params& p) const {
    const BwParams<float>& q = p.b;
    // what the TMA descriptors would refuse: widths that are not whole 32-column blocks, and, for
    // panels made of strided segments, rows that are not whole groups of segments
    if (!bw3 || !q.vec_x || !q.vec_g || !q.vec_o || q.xin_cols % 32 || q.gin_cols % 32 || q.gout_cols % 32) return false;
    if (q.xin_cols < 32 || q.gin_cols < 32 || q.gout_cols < 32 || (q.gin_flat > 0 && q.gin_flat != q.S << q.log_n)) return false;
    if (q.vr > 0) return q.log_n >= 5 && (kBw3Rows << q.vr) <= 256;  // whole rows, as many as a box takes
    if (q.panel.lseg != q.panel.logC) {
      const int grp = 1 << q.panel.pb;
      for (int cols : {q.xin_cols, q.gin_cols, q.gout_cols})
        if (cols % grp != 0 && cols >= grp) return false; else if (cols < grp) return false;
    }
    return true;
  }
  int run_bw3(const Bw3Params& p) {
    if (!can_run_bw3(p)) return kFw2Declined;
    const BwParams<float>& q = p.b;
    ++g_bw3_calls;
    const int C = 1024, nthr = kBw3Threads;
    std::vector<float> smem((size_t)(q.nsg + 1) * kBw3Rows * C);
    float* smX = smem.data();
    float* smG = smem.data() + (size_t)q.nsg * kBw3Rows * C;
    std::vector<uint32_t> meta((size_t)q.nsg * nthr * 4 + 8);
    std::vector<float> accmem((size_t)nthr * kBw3MaxSg * 64);
    std::vector<float> pf((size_t)nthr * 64);  // per-thread fetch buffers (twiddles, accumulators of the next step)
    const int nctas = bw_num_ctas(q);
    for (int cta = 0; cta < nctas; ++cta) {
      int pbase, stack, rb, re;
      bw_cta_coords(q, cta, pbase, stack, rb, re);
      std::vector<Acc3Host> accs(nthr);
      for (int tid = 0; tid < nthr; ++tid) {
        accs[tid].mem = accmem.data() + (size_t)tid * kBw3MaxSg * 64;
        bw3_init(p, accs[tid], meta.data(), stack, pbase, tid);
        bw3_prefetch(p, accs[tid], 0, pf.data() + (size_t)tid * 64, pf.data() + (size_t)tid * 64 + 32);
      }
      for (int row0 = rb; row0 < re; row0 += kBw3Rows) {
        for (int tid = 0; tid < nthr; ++tid) {
          tile_load_v<float>(q.xin, q.xin_sB, q.xin_sS, q.xin_cols, q.B_rows, stack, row0, kBw3Rows, q.panel, pbase, true, q.log_n, q.vr, smX, tid, nthr);
          tile_load_v<float>(q.gin, q.gin_sB, q.gin_sS, q.gin_cols, q.B_rows, stack, row0, kBw3Rows, q.panel, pbase, true, q.log_n, q.vr, smG, tid, nthr);
        }
        if (q.dbias)  // column sums of the gradient tile as it arrived
          for (int r = 0; r < kBw3Rows; ++r)
            for (int l = 0; l < C; ++l) {
              const int flat = stack * (1 << q.log_n) + q.panel.col(pbase, l);
              if (flat < q.dbias_len) q.dbias[flat] += smG[r * C + swz<2>(l)];
            }
        for (int step = 0; step < bw3_num_steps(q.nsg); ++step)
          for (int tid = 0; tid < nthr; ++tid)
            bw3_step(p, accs[tid], meta.data(), step, smem.data(), tid, pf.data() + (size_t)tid * 64, pf.data() + (size_t)tid * 64 + 32);
        if (q.gout_reduce) {  // the device kernel's reduce-add store
          for (int r = 0; r < kBw3Rows; ++r)
            for (int l = 0; l < C; ++l) {
              const int at = q.panel.col(pbase, l), col = at & ((1 << q.log_n) - 1);
              const int64_t row = ((int64_t)(row0 + r) << q.vr) + (at >> q.log_n);
              if (row < q.B_rows && col < q.gout_cols) q.gout[row * q.gout_sB + (int64_t)stack * q.gout_sS + col] += smG[r * C + swz<2>(l)];
            }
        } else {
          for (int tid = 0; tid < nthr; ++tid)
            tile_store_v<float>(q.gout, q.gout_sB, q.gout_sS, q.gout_cols, q.B_rows, stack, row0, kBw3Rows, q.panel, pbase, true, q.log_n, q.vr, smG, tid, nthr);
        }
      }
      const std::vector<float> folded = fold_rows<32>(q.nsg, nthr, [&](int j) { return bw_row_threads(q, p.sg[j].ubit, 7); },
                                                      [&](int j, int tid, float* w) { accs[tid].ld32(j * 64 + 32, w); });
      for (int tid = 0; tid < nthr; ++tid)
        bw3_flush(p, accs[tid], stack, pbase, tid, [&](int j, float* w) {
          std::copy_n(&folded[(size_t)(j * nthr + tid) * 32], 32, w);
          return !(tid & bw_row_threads(q, p.sg[j].ubit, 7));
        });
    }
    return BFLY_OK;
  }

  template <typename T> int run_fw(const FwParams<T>& p) {
    const int C = 1 << p.panel.logC;
    std::vector<T> sm((size_t)p.R * C);
    std::vector<uint16_t> tab((size_t)p.ngroups * p.tab_slots * threads_ + 1);
    for (int tid = 0; tid < threads_; ++tid) fw_build_table<T>(p, tab.data(), tid, threads_);
    const int64_t ntiles = fw_num_tiles(p);
    const int64_t n = (int64_t)1 << p.log_n;
    for (int64_t tile = 0; tile < ntiles; ++tile) {
      int row0, stack, pbase;
      fw_tile_coords(p, tile, row0, stack, pbase);
      for (int tid = 0; tid < threads_; ++tid) {
        if (p.glue.x_real) tile_load_real(p.glue.x_real, p.x_sB, p.x_sS, p.x_cols, p.B_rows, stack, row0, p.R, p.panel.logC, sm.data(), tid, threads_, p.vr);
        else tile_load_v<T>(p.x, p.x_sB, p.x_sS, p.x_cols, p.B_rows, stack, row0, p.R, p.panel, pbase, p.vec_in != 0, p.log_n, p.vr, sm.data(), tid, threads_);
      }
      // the kernel's gather pass: wide rows of the same width, three at a time: every thread reads, barrier, every thread writes
      auto permute_rows = [&](const int32_t* perm, const T* diag) {
        constexpr int kWide = sizeof(T) == 8 ? 11 : 12, kSlots = 64, RB = 3;
        if ((1 << kWide) > kSlots * threads_) { std::fprintf(stderr, "emulated gathers need %d threads\n", (1 << kWide) / kSlots); std::abort(); }
        std::vector<T> v((size_t)threads_ * RB * kSlots);
        std::vector<uint32_t> plan((size_t)threads_ * kSlots);
        std::vector<int> cnt(threads_);
        const int mask = (int)n - 1;
        for (int tid = 0; tid < threads_; ++tid)
          cnt[tid] = tile_permute_plan<T, kSlots>(p.panel.logC, perm, p.glue.colbit, tid, threads_, plan.data() + (size_t)tid * kSlots, mask, kWide);
        for (int left = p.R << p.panel.logC, r = 0; left > 0; left -= RB << kWide, r += RB) {
          for (int tid = 0; tid < threads_; ++tid)
            tile_permute_read<T, kSlots, RB>(sm.data(), r, p.panel.logC, diag, plan.data() + (size_t)tid * kSlots, cnt[tid], v.data() + (size_t)tid * RB * kSlots, mask, kWide, left);
          for (int tid = 0; tid < threads_; ++tid)
            tile_permute_write<T, kSlots, RB>(sm.data(), r, plan.data() + (size_t)tid * kSlots, cnt[tid], v.data() + (size_t)tid * RB * kSlots, kWide, left);
        }
      };
      if (p.glue.any_in()) permute_rows(p.glue.in_perm, nullptr);
      for (int g = 0; g < p.ngroups; ++g) {
        for (int tid = 0; tid < threads_; ++tid)
          fw_group_dispatch<T, 4, 0, 0>(p, g, sm.data(), tab.data(), p.R, stack, pbase, tid, threads_);
        if (p.g[g].emit)
          for (int tid = 0; tid < threads_; ++tid)
            tile_store_v<T>(p.snap[p.g[g].emit - 1], (int64_t)p.S * n, n, (int)n, p.B_rows, stack, row0, p.R, p.panel, pbase, true, p.log_n, p.vr, sm.data(), tid, threads_);
      }
      if (p.bias)
        for (int tid = 0; tid < threads_; ++tid)
          tile_add_bias<T>(sm.data(), p.R, p.panel, pbase, p.bias, stack * (int)n, p.bias_len, (int)n - 1, tid, threads_);
      if (p.glue.out_perm) permute_rows(p.glue.out_perm, p.glue.out_diag);
      const bool scaled = p.glue.out_diag && !p.glue.out_perm;  // a diagonal alone goes with the store
      for (int tid = 0; tid < threads_; ++tid) {
        if (scaled && p.glue.out_real)
          tile_store_scaled<T>(p.glue.out_real, p.out_sB, p.out_sS, p.out_cols, p.B_rows, stack, row0, p.R, p.panel.logC, p.log_n, p.vr,
                               p.glue.out_diag, sm.data(), tid, threads_);
        else if (scaled)
          tile_store_scaled<T>(p.out, p.out_sB, p.out_sS, p.out_cols, p.B_rows, stack, row0, p.R, p.panel.logC, p.log_n, p.vr,
                               p.glue.out_diag, sm.data(), tid, threads_);
        else if (p.glue.out_real)
          tile_store_real(p.glue.out_real, p.out_sB, p.out_sS, p.out_cols, p.B_rows, stack, row0, p.R, p.panel.logC, sm.data(), tid, threads_, p.vr);
        else if (p.out)
          tile_store_v<T>(p.out, p.out_sB, p.out_sS, p.out_cols, p.B_rows, stack, row0, p.R, p.panel, pbase, p.vec_out != 0, p.log_n, p.vr, sm.data(), tid, threads_);
      }
    }
    return BFLY_OK;
  }

  // second-generation backward: same step routines as the device kernel, accumulators in a heap array
  template <typename T, int KW> int run_bw2(const BwParams<T>& p) {
    constexpr int N = BwTwn<KW>::value;
    const int C = 1 << p.panel.logC;
    const int nthr = C >> KW;
    // one buffer, as on the device: nsg snapshot tiles followed by the gradient tile
    std::vector<T> smem((size_t)(p.nsg + 1) * kBw2Rows * C);
    struct View { T* ptr; T* data() const { return ptr; } };
    const View smX{smem.data()}, smG{smem.data() + (size_t)p.nsg * kBw2Rows * C};
    std::vector<uint32_t> meta((size_t)p.nsg * kBw2Meta * nthr);
    std::vector<T> accmem((size_t)nthr * 2 * kMaxSg * N);
    const int nctas = bw_num_ctas(p);
    for (int cta = 0; cta < nctas; ++cta) {
      int pbase, stack, rb, re;
      bw_cta_coords(p, cta, pbase, stack, rb, re);
      std::vector<AccStore<T, KW>> accs(nthr);
      for (int tid = 0; tid < nthr; ++tid) {
        accs[tid].mem = accmem.data() + (size_t)tid * 2 * kMaxSg * N;
        bw2_build_meta<T, KW>(p, meta.data(), pbase, tid, nthr);
      }
      for (int tid = 0; tid < nthr; ++tid) bw2_init<T, KW>(p, accs[tid], meta.data(), stack, tid, nthr);
      for (int row0 = rb; row0 < re; row0 += kBw2Rows) {
        for (int tid = 0; tid < nthr; ++tid) {
          tile_load_v<T>(p.xin, p.xin_sB, p.xin_sS, p.xin_cols, bw_row_limit(p, re), stack, row0, kBw2Rows, p.panel, pbase, p.vec_x != 0, p.log_n, p.vr, smX.data(), tid, nthr);
          tile_load_v<T>(p.gin, p.gin_sB, p.gin_sS, bw_gin_cols(p, stack), bw_row_limit(p, re), stack, row0, kBw2Rows, p.panel, pbase, p.vec_g != 0, p.log_n, p.vr, smG.data(), tid, nthr);
        }
        for (int j = 0; j + 1 < p.nsg; ++j)
          for (int tid = 0; tid < nthr; ++tid)
            bw2_fw_step<T, KW, 0>(p, accs[tid], meta.data(), j, smX.data(), smG.data(), tid, nthr);
        for (int j = p.nsg - 1; j >= 0; --j)
          for (int tid = 0; tid < nthr; ++tid)
            bw2_bw_step<T, KW, 0>(p, accs[tid], meta.data(), j, smX.data(), smG.data(), tid, nthr);
        for (int tid = 0; tid < nthr; ++tid)
          tile_store_v<T>(p.gout, p.gout_sB, p.gout_sS, p.gout_cols, bw_row_limit(p, re), stack, row0, kBw2Rows, p.panel, pbase, p.vec_o != 0, p.log_n, p.vr, smG.data(), tid, nthr);
      }
      auto mask = [&](int j) { return sizeof(T) == 4 ? bw_row_threads(p, p.sg[j].ubit, p.sg[j].nubits) : 0; };
      const std::vector<T> folded = fold_rows<N, T>(p.nsg, nthr, mask, [&](int j, int tid, T* w) { accs[tid].ld(j, w); });
      for (int tid = 0; tid < nthr; ++tid)
        bw2_flush<T, KW>(p, accs[tid], meta.data(), stack, tid, nthr, [&](int j, T* w) {
          std::copy_n(&folded[(size_t)(j * nthr + tid) * N], N, w);
          return !(tid & mask(j));
        });
    }
    return BFLY_OK;
  }

  template <typename T, int KW> int run_bw_kw(const BwParams<T>& p) {
    if (p.v2) return run_bw2<T, KW>(p);
    constexpr int NSG = kMaxSg;
    const int C = 1 << p.panel.logC;
    // the device kernel uses exactly one thread per unit (or a power-of-two multiple)
    int nthr = threads_;
    const int U = C >> KW;
    if (U > nthr) nthr = U;
    std::vector<T> smX((size_t)p.nsg * p.Rb * C), smG((size_t)p.Rb * C);
    std::vector<BwState<T, KW, NSG>> st(nthr);
    const int nctas = bw_num_ctas(p);
    for (int cta = 0; cta < nctas; ++cta) {
      int pbase, stack, rb, re;
      bw_cta_coords(p, cta, pbase, stack, rb, re);
      for (int tid = 0; tid < nthr; ++tid) bw_load_state<T, KW, NSG>(p, st[tid], stack, pbase, tid, nthr);
      for (int row0 = rb; row0 < re; row0 += p.Rb) {
        const int R = p.Rb;
        for (int tid = 0; tid < nthr; ++tid) {
          tile_load_v<T>(p.xin, p.xin_sB, p.xin_sS, p.xin_cols, bw_row_limit(p, re), stack, row0, R, p.panel, pbase, p.vec_x != 0, p.log_n, p.vr, smX.data(), tid, nthr);
          tile_load_v<T>(p.gin, p.gin_sB, p.gin_sS, bw_gin_cols(p, stack), bw_row_limit(p, re), stack, row0, R, p.panel, pbase, p.vec_g != 0, p.log_n, p.vr, smG.data(), tid, nthr);
        }
        for (int j = 0; j + 1 < p.nsg; ++j)
          for (int tid = 0; tid < nthr; ++tid) bw_sg_step<T, KW, NSG, 0, 0, true>(p, st[tid], j, stack, smX.data(), smG.data(), R, tid, nthr);
        for (int j = p.nsg - 1; j >= 0; --j)
          for (int tid = 0; tid < nthr; ++tid) bw_sg_step<T, KW, NSG, 0, 0, false>(p, st[tid], j, stack, smX.data(), smG.data(), R, tid, nthr);
        for (int tid = 0; tid < nthr; ++tid)
          tile_store_v<T>(p.gout, p.gout_sB, p.gout_sS, p.gout_cols, bw_row_limit(p, re), stack, row0, R, p.panel, pbase, p.vec_o != 0, p.log_n, p.vr, smG.data(), tid, nthr);
      }
      for (int tid = 0; tid < nthr; ++tid) bw_flush_state<T, KW, NSG>(p, st[tid], stack, pbase, tid, nthr);
    }
    return BFLY_OK;
  }
  template <typename T> int run_bw(const BwParams<T>& p, int KW) {
    return KW == 2 ? run_bw_kw<T, 2>(p) : run_bw_kw<T, 1>(p);
  }
  int add_bias(float* out, const float* bias, int64_t B, int len, int64_t pitch) {
    for (int64_t b = 0; b < B; ++b)
      for (int f = 0; f < len; ++f) out[b * pitch + f] += bias[f];
    return BFLY_OK;
  }
  static constexpr bool kFusedBias = true;  // run_fw adds FwParams::bias
  // layers: the sums of the small kernels
  template <typename T> int column_sums(const T* g, int64_t pitch, int64_t B, int cols, T* out, float* partial) {
    constexpr int F = (int)(sizeof(T) / 4);
    auto sums = [](const float* src, int64_t p, int64_t rows, int n, float* dst) {
      for (int c = 0; c < n; ++c) {
        dst[c] = 0.f;
        for (int64_t r = 0; r < rows; ++r) dst[c] += src[r * p + c];
      }
    };
    const SumSlices s = column_sum_slices(B, cols * F);
    const float* gf = reinterpret_cast<const float*>(g);
    float* of = reinterpret_cast<float*>(out);
    if (s.count == 1) { sums(gf, pitch * F, B, cols * F, of); return BFLY_OK; }
    for (int64_t y = 0; y < s.count; ++y)
      sums(gf + y * s.rows * pitch * F, pitch * F, std::min(s.rows, B - y * s.rows), cols * F, partial + y * cols * F);
    sums(partial, cols * F, s.count, cols * F, of);
    return BFLY_OK;
  }
  template <typename T> int stack_sums(const T* g, int64_t B, int S, int64_t n, int cols, T* out) {
    for (int64_t b = 0; b < B; ++b)
      for (int c = 0; c < cols; ++c) {
        T acc = Ops<T>::zero();
        for (int s = 0; s < S; ++s) acc = add1(acc, g[(b * S + s) * n + c]);
        out[b * cols + c] = acc;
      }
    return BFLY_OK;
  }
  int zero(void* ptr, size_t bytes) { std::memset(ptr, 0, bytes); return BFLY_OK; }
  int zero2d(void* ptr, size_t pitch, size_t width, size_t rows) {
    for (size_t r = 0; r < rows; ++r) std::memset(static_cast<char*>(ptr) + r * pitch, 0, width);
    return BFLY_OK;
  }
};

template <typename T>
int emul_fw(const void* tw2, const void* tw4, const void* x, int64_t x_sB, int64_t x_sS, void* out, Problem q, int threads) {
  EmulExec ex; ex.threads_ = threads;
  std::vector<char> ws(fw_workspace_bytes<T>(q) + 256);
  void* wsp = (void*)(((uintptr_t)ws.data() + 255) / 256 * 256);
  return drive_fw<T>(ex, q, (const T*)tw2, (const T*)tw4, (const T*)x, x_sB, x_sS, (T*)out, wsp, fw_workspace_bytes<T>(q));
}
template <typename T>
int emul_bw(const void* tw2, const void* tw4, const void* x, int64_t x_sB, int64_t x_sS, const void* g, int64_t g_sB, int64_t g_sS,
            void* d2, void* d4, void* dx, Problem q, int threads, int sms) {
  EmulExec ex; ex.threads_ = threads; ex.sms = sms;
  BwLayout<T> lay;
  int rc = check_problem(q);
  if (rc) return rc;
  rc = plan_bw<T>(q, lay);
  if (rc) return rc;
  std::vector<char> ws(lay.ws_bytes + 256);
  void* wsp = (void*)(((uintptr_t)ws.data() + 255) / 256 * 256);
  return drive_bw<T>(ex, q, (const T*)tw2, (const T*)tw4, (const T*)x, x_sB, x_sS, (const T*)g, g_sB, g_sS, (T*)d2, (T*)d4, (T*)dx, wsp, lay.ws_bytes);
}

// forward that saves the phase-boundary activations, then the backward that starts from them
template <typename T>
int emul_fw_bw_saved(const void* tw2, const void* x, int64_t x_sB, int64_t x_sS, void* out, const void* g, int64_t g_sB,
                     int64_t g_sS, void* d2, void* dx, Problem q, int threads, int sms) {
  EmulExec ex; ex.threads_ = threads; ex.sms = sms;
  BwLayout<T> lay;
  int rc = check_problem(q);
  if (rc) return rc;
  rc = plan_bw<T>(q, lay);
  if (rc) return rc;
  std::vector<char> ws(lay.ws_bytes + 256);
  void* wsp = (void*)(((uintptr_t)ws.data() + 255) / 256 * 256);
  rc = drive_fw_saving<T>(ex, q, (const T*)tw2, (const T*)nullptr, (const T*)x, x_sB, x_sS, (T*)out, wsp, lay.ws_bytes);
  if (rc) return rc;
  return drive_bw<T>(ex, q, (const T*)tw2, (const T*)nullptr, (const T*)x, x_sB, x_sS, (const T*)g, g_sB, g_sS, (T*)d2,
                     (T*)nullptr, (T*)dx, wsp, lay.ws_bytes, true);
}

}  // namespace

// Worst shared-memory bank-conflict degree (1 = conflict-free) of the accesses a 256-thread CTA
// makes to one tile row: per group / sub-group, per warp, per element of the unit.  An access of
// `bytes` per lane is served in phases of 128/bytes lanes; the degree of a phase is the largest
// number of distinct 4-byte words that fall into one of the 32 banks.
static int conflict_degree(const std::vector<long>& byte_addr, int bytes) {
  const int lanes_per_phase = 128 / bytes;
  int worst = 1;
  for (size_t p0 = 0; p0 < byte_addr.size(); p0 += lanes_per_phase) {
    std::vector<std::vector<long>> bank(32);
    for (size_t i = p0; i < p0 + lanes_per_phase && i < byte_addr.size(); ++i)
      for (int w = 0; w < bytes / 4; ++w) {
        const long word = byte_addr[i] / 4 + w;
        auto& b = bank[word % 32];
        if (std::find(b.begin(), b.end(), word) == b.end()) b.push_back(word);
      }
    for (auto& b : bank) worst = std::max<int>(worst, (int)b.size());
  }
  return worst;
}

template <typename T>
static int window_conflicts(int logC, int lbit, int K, bool vec, const uint8_t* ubit, int nubits, const uint16_t* d) {
  const int nthr = 256, C = 1 << logC, U = C >> K;
  if (U < 32) return 1;  // tiny rows: several rows share a warp, not analysed
  int worst = 1;
  const int V = Vec16<T>::N, E = 1 << K;
  for (int warp = 0; warp < std::min(nthr, U) / 32; ++warp)
    for (int m = 0; m < (vec ? E / V : E); ++m) {
      std::vector<long> addr;
      for (int lane = 0; lane < 32; ++lane) {
        const int u = warp * 32 + lane;
        const int a0 = swzT<T>(deposit_unit(u, ubit, nubits));
        addr.push_back((long)(a0 ^ d[vec ? m * V : m]) * (long)sizeof(T));
      }
      worst = std::max(worst, conflict_degree(addr, vec ? 16 : (int)sizeof(T)));
    }
  return worst;
}

template <typename T>
static int max_conflicts(const Problem& q, int kmax) {
  const std::vector<Stage> st = problem_stages(q);
  int worst = 1;
  std::vector<FwGroup> groups;
  const Panel pn = full_row_panel(q.log_n);
  if (!plan_fw_groups(st, 0, (int)st.size(), {}, pn, Vec16<T>::LOG, kmax, groups)) return -1;
  for (auto& g : groups) worst = std::max(worst, window_conflicts<T>(pn.logC, g.lbit, g.K, g.vec != 0, g.ubit, g.nubits, g.d));
  BwLayout<T> lay;
  if (plan_bw<T>(q, lay) != BFLY_OK) return -1;
  for (auto& ph : lay.phases)
    for (int j = 0; j < ph.nsg; ++j) {
      const BwSg& sg = ph.sg[j];
      const int width = sg.radix == 4 ? 2 : lay.kw;
      worst = std::max(worst, window_conflicts<T>(ph.panel.logC, sg.lbit, width, sg.vec != 0, sg.ubit, sg.nubits, sg.d));
    }
  return worst;
}

extern "C" {
// the per-block arithmetic of the unitary twiddle kernels (bfly_glue.h), looped on the host
void bfly_emul_unitary_fw(const float* angles, float* tw, int64_t blocks) {
  for (int64_t i = 0; i < blocks; ++i) unitary_block_fw(angles + 4 * i, tw + 8 * i);
}
void bfly_emul_unitary_bw(const float* angles, const float* g, float* d, int64_t blocks) {
  for (int64_t i = 0; i < blocks; ++i) unitary_block_bw(angles + 4 * i, g + 8 * i, d + 4 * i);
}
long bfly_emul_fw2_calls(void) { return g_fw2_calls; }
long bfly_emul_bw3_calls(void) { return g_bw3_calls; }
// the library's development switches (bfly_driver.h) for this emulator instance
int bfly_emul_set_option(const char* name, int value) { return set_option(name, value); }
int bfly_emul_get_option(const char* name) { int v = -1; get_option(name, &v); return v; }
int bfly_emul_max_conflicts(int dtype, int base4, int log_n, int nblocks, int inc, int kmax) {
  Problem q{4, 1, log_n, nblocks, 1 << log_n, 1 << log_n, inc != 0, base4 != 0};
  return dtype == 0 ? max_conflicts<float>(q, kmax) : max_conflicts<cf>(q, kmax);
}
// dtype: 0 float32, 1 complex64.  base4: tw2 = twiddle2, tw4 = twiddle4; else tw2 = twiddle.
int bfly_emul_fw(int dtype, int base4, const void* tw2, const void* tw4, const void* x, int64_t x_sB, int64_t x_sS, void* out,
                 int B, int S, int log_n, int nblocks, int in_size, int out_size, int inc, int threads) {
  Problem q{B, S, log_n, nblocks, in_size, out_size, inc != 0, base4 != 0};
  return dtype == 0 ? emul_fw<float>(tw2, tw4, x, x_sB, x_sS, out, q, threads) : emul_fw<cf>(tw2, tw4, x, x_sB, x_sS, out, q, threads);
}
int bfly_emul_bw(int dtype, int base4, const void* tw2, const void* tw4, const void* x, int64_t x_sB, int64_t x_sS, const void* g,
                 int64_t g_sB, int64_t g_sS, void* d2, void* d4, void* dx, int B, int S, int log_n, int nblocks, int in_size,
                 int out_size, int inc, int threads, int sms) {
  Problem q{B, S, log_n, nblocks, in_size, out_size, inc != 0, base4 != 0};
  return dtype == 0 ? emul_bw<float>(tw2, tw4, x, x_sB, x_sS, g, g_sB, g_sS, d2, d4, dx, q, threads, sms)
                    : emul_bw<cf>(tw2, tw4, x, x_sB, x_sS, g, g_sB, g_sS, d2, d4, dx, q, threads, sms);
}
int bfly_emul_fw_bw_saved(int dtype, const void* tw, const void* x, int64_t x_sB, int64_t x_sS, void* out, const void* g,
                          int64_t g_sB, int64_t g_sS, void* d_tw, void* dx, int B, int S, int log_n, int nblocks, int in_size,
                          int out_size, int inc, int threads, int sms) {
  Problem q{B, S, log_n, nblocks, in_size, out_size, inc != 0, false};
  return dtype == 0 ? emul_fw_bw_saved<float>(tw, x, x_sB, x_sS, out, g, g_sB, g_sS, d_tw, dx, q, threads, sms)
                    : emul_fw_bw_saved<cf>(tw, x, x_sB, x_sS, out, g, g_sB, g_sS, d_tw, dx, q, threads, sms);
}
// fused linear layer: forward into out (B, S * n), backward with d_input summed over the stacks and d_bias
int bfly_emul_linear_fw(const void* tw, const void* x, int64_t x_sB, void* out, const void* bias, int B, int S, int log_n,
                        int nblocks, int in_size, int out_total, int inc) {
  EmulExec ex; ex.threads_ = 256;
  Problem q{B, S, log_n, nblocks, in_size, 1 << log_n, inc != 0, false};
  std::vector<char> ws(fw_workspace_bytes<float>(q) + 256);
  void* wsp = (void*)(((uintptr_t)ws.data() + 255) / 256 * 256);
  return drive_linear_fw(ex, q, (const float*)tw, (const float*)x, x_sB, (float*)out, (const float*)bias, out_total, wsp,
                         fw_workspace_bytes<float>(q));
}
int bfly_emul_linear_bw(const void* tw, const void* x, int64_t x_sB, const void* g, int64_t g_sB, void* d_tw, void* d_in,
                        int64_t din_sB, void* d_bias, int B, int S, int log_n, int nblocks, int in_size, int out_total, int inc,
                        int sms) {
  EmulExec ex; ex.threads_ = 256; ex.sms = sms;
  Problem q{B, S, log_n, nblocks, in_size, 1 << log_n, inc != 0, false};
  LinearBwLayout L;
  int rc = check_problem(q);
  if (rc) return rc;
  rc = plan_linear_bw(q, L);
  if (rc) return rc;
  std::vector<char> ws(L.ws_bytes + 256);
  void* wsp = (void*)(((uintptr_t)ws.data() + 255) / 256 * 256);
  return drive_linear_bw(ex, q, (const float*)tw, (const float*)x, x_sB, (const float*)g, g_sB, (float*)d_tw, (float*)d_in,
                         din_sB, (float*)d_bias, out_total, wsp, L.ws_bytes);
}
// the forward with glue operators (drive_fw_glue); dtype 0 float32, 1 complex64
int bfly_emul_fw_glue(int dtype, const void* tw, const void* x, int x_is_real, int64_t x_sB, int64_t x_sS, void* out, int out_is_real,
                      const int32_t* in_perm, const void* out_diag, const int32_t* out_perm, int B, int S, int log_n, int nblocks,
                      int in_size, int out_size, int inc, int threads) {
  EmulExec ex; ex.threads_ = threads;
  Problem q{B, S, log_n, nblocks, in_size, out_size, inc != 0, false};
  if (dtype == 0) {
    FwGlue<float> g{};
    g.in_perm = in_perm; g.out_perm = out_perm; g.out_diag = (const float*)out_diag;
    return drive_fw_glue<float>(ex, q, (const float*)tw, (const float*)x, x_sB, x_sS, (float*)out, g);
  }
  FwGlue<cf> g{};
  g.in_perm = in_perm; g.out_perm = out_perm; g.out_diag = (const cf*)out_diag;
  if (x_is_real) g.x_real = (const float*)x;
  if (out_is_real) g.out_real = (float*)out;
  return drive_fw_glue<cf>(ex, q, (const cf*)tw, x_is_real ? nullptr : (const cf*)x, x_sB, x_sS, out_is_real ? nullptr : (cf*)out, g);
}
// A whole layer: the forward (with the snapshots of the backward when `save`), then the backward that starts from them
// or recomputes.  dtype 0 float32, 1 complex64; tw2 / tw4 and their gradients as in bfly_emul_fw.
}
template <typename T>
static int emul_layer(const void* tw2, const void* tw4, const void* x, int64_t x_sB, const void* bias, void* out, const void* g, int64_t g_sB,
                      void* d2, void* d4, void* d_in, void* d_bias, Problem q, int out_total, int save, int threads, int sms) {
  EmulExec ex; ex.threads_ = threads; ex.sms = sms;
  BwLayout<T> lay;
  int rc = check_problem(q);
  if (rc) return rc;
  rc = plan_bw<T>(q, lay);
  if (rc) return rc;
  auto aligned = [](std::vector<char>& v) { return (void*)(((uintptr_t)v.data() + 255) / 256 * 256); };
  const size_t keep = save && !lay.chunked ? lay.ws_bytes : 0;
  std::vector<char> snaps(keep + 256), fws(fw_workspace_bytes<T>(q) + 256);
  void* sp = keep ? aligned(snaps) : nullptr;
  rc = drive_layer_fw<T>(ex, q, (const T*)tw2, (const T*)tw4, (const T*)x, x_sB, (T*)out, (const T*)bias, out_total, sp, keep,
                         sp ? nullptr : aligned(fws), sp ? 0 : fw_workspace_bytes<T>(q));
  if (rc) return rc;
  LayerBwLayout L;
  rc = plan_layer_bw<T>(q, out_total, sp != nullptr, L);
  if (rc) return rc;
  std::vector<char> ws(L.ws_bytes + 256);
  return drive_layer_bw<T>(ex, q, (const T*)tw2, (const T*)tw4, (const T*)x, x_sB, (const T*)g, g_sB, (T*)d2, (T*)d4, (T*)d_in, (T*)d_bias,
                           out_total, sp, keep, L.ws_bytes ? aligned(ws) : nullptr, L.ws_bytes);
}
extern "C" {
int bfly_emul_layer(int dtype, int base4, const void* tw2, const void* tw4, const void* x, int64_t x_sB, const void* bias, void* out,
                    const void* g, int64_t g_sB, void* d2, void* d4, void* d_in, void* d_bias, int B, int S, int log_n, int nblocks,
                    int in_size, int out_total, int inc, int save, int threads, int sms) {
  Problem q{B, S, log_n, nblocks, in_size, 1 << (log_n & 31), inc != 0, base4 != 0};
  return dtype == 0 ? emul_layer<float>(tw2, tw4, x, x_sB, bias, out, g, g_sB, d2, d4, d_in, d_bias, q, out_total, save, threads, sms)
                    : emul_layer<cf>(tw2, tw4, x, x_sB, bias, out, g, g_sB, d2, d4, d_in, d_bias, q, out_total, save, threads, sms);
}
// number of backward phases and workspace bytes the planner chooses (for tests of the planner)
int bfly_emul_bw_plan(int dtype, int base4, int B, int S, int log_n, int nblocks, int inc, int64_t* ws_bytes) {
  Problem q{B, S, log_n, nblocks, 1 << log_n, 1 << log_n, inc != 0, base4 != 0};
  int rc = check_problem(q);
  if (rc) return rc;
  size_t ws = 0; int nph = 0;
  if (dtype == 0) { BwLayout<float> l; rc = plan_bw<float>(q, l); ws = l.ws_bytes; nph = (int)l.phases.size(); }
  else { BwLayout<cf> l; rc = plan_bw<cf>(q, l); ws = l.ws_bytes; nph = (int)l.phases.size(); }
  if (rc) return rc;
  *ws_bytes = (int64_t)ws;
  return nph;
}
}

// ------------------------------------------------------------------ dry runs of whole training steps
//
// The drivers with an executor that launches nothing: every call gets buffers of exactly the queried sizes, at made-up
// addresses, and each launch's tensors are checked to lie inside them.
namespace {
struct DryExec {
  static constexpr bool kMma = true, kFusedBias = true;
  const int* guard = nullptr;
  struct Range { uintptr_t at; size_t bytes; };
  std::vector<Range> ranges;
  int outside = 0, passes = 0;  // tensors that left their buffer; tensor-core passes
  // a buffer of `bytes` bytes, `skew` past a 256-byte boundary
  template <typename T> T* buffer(size_t bytes, size_t skew = 0) {
    if (!bytes) return nullptr;
    ranges.push_back({((uintptr_t)(ranges.size() + 1) << 44) + skew, bytes});
    return reinterpret_cast<T*>(ranges.back().at);
  }
  void in(const void* p, size_t bytes) {
    const uintptr_t a = (uintptr_t)p;
    for (auto& r : ranges)
      if (a >= r.at && a + bytes <= r.at + r.bytes) return;
    ++outside;
  }
  template <typename T> void rows(const T* p, int64_t B, int64_t S, int64_t sB, int64_t sS, int64_t cols) {
    if (p && B > 0 && cols > 0) in(p, ((B - 1) * sB + (S - 1) * sS + cols) * sizeof(T));
  }
  int num_sms() const { return 148; }
  int threads() const { return 256; }
  bool has_bw2(size_t, int kw) const { return kw == 2; }
  int run_fw2(const Fw2Params& p, int) {
    const int64_t S = p.view ? 1 : p.S, n = p.view ? p.view_row : (int64_t)1 << p.log_n;
    for (const float* s : p.snap)
      if (s) in(s, (size_t)p.B * S * n * sizeof(float));
    in(p.packed, (size_t)p.packed_stack * p.S * 16);
    rows(p.x, p.B, S, p.x_sB, p.x_sS, p.view ? n : std::min<int64_t>(p.x_cols, n));
    rows(p.out, p.B, S, p.out_sB, p.out_sS, p.view ? n : p.out_cols);
    return BFLY_OK;
  }
  template <typename T> int run_fw(const FwParams<T>& p) {
    const int64_t n = (int64_t)1 << p.log_n;
    for (const T* s : p.snap)
      if (s) in(s, ((size_t)p.B_rows * p.S << p.log_n) * sizeof(T));
    rows(p.x, p.B_rows, p.S, p.x_sB, p.x_sS, std::min<int64_t>(p.x_cols, n));
    rows(p.out, p.B_rows, p.S, p.out_sB, p.out_sS, std::min<int64_t>(p.out_cols, n));
    return BFLY_OK;
  }
  template <typename T> int run_bw(const BwParams<T>& p, int) {
    const int64_t n = (int64_t)1 << p.log_n;
    rows(p.xin, p.B_rows, p.S, p.xin_sB, p.xin_sS, std::min<int64_t>(p.xin_cols, n));
    rows(p.gin, p.B_rows, p.gin_flat > 0 ? 1 : p.S, p.gin_sB, p.gin_sS, p.gin_flat > 0 ? p.gin_flat : std::min<int64_t>(p.gin_cols, n));
    rows(p.gout, p.B_rows, p.S, p.gout_sB, p.gout_sS, p.gout_cols);
    return BFLY_OK;
  }
  bool can_run_bw3(const Bw3Params&) { return true; }
  int run_bw3(const Bw3Params& p) { return run_bw(p.b, 2); }
  int add_bias(float* out, const float* bias, int64_t B, int len, int64_t pitch) { rows(out, B, 1, pitch, 0, len); in(bias, len * 4); return BFLY_OK; }
  template <typename T> int column_sums(const T* g, int64_t pitch, int64_t B, int cols, T* out, float* partial) {
    rows(g, B, 1, pitch, 0, cols);
    in(out, cols * sizeof(T));
    if (const size_t f = column_sum_slices(B, cols * (int)(sizeof(T) / 4)).floats) in(partial, f * 4);
    return BFLY_OK;
  }
  template <typename T> int stack_sums(const T* g, int64_t B, int S, int64_t n, int cols, T* out) {
    in(g, B * S * n * sizeof(T));
    in(out, B * cols * sizeof(T));
    return BFLY_OK;
  }
  int zero(void* p, size_t bytes) { in(p, bytes); return BFLY_OK; }
  int zero2d(void* p, size_t pitch, size_t width, size_t n) { if (n) in(p, (n - 1) * pitch + width); return BFLY_OK; }
  void io(const MmaRowsIO& r, const MmaPass& p) {
    if (r.flat > 0) rows(r.p, p.B, 1, r.sB, 0, r.flat);
    else rows(r.p, p.B, p.S, r.sB, r.sS, std::min(r.cols, 1 << p.geo.log_nf));
  }
  void plane(const float* t, const MmaPass& p) { in(t, ((size_t)p.S * p.nt * kMmaRows << p.geo.log_nf) * sizeof(float)); }
  int mma_prep(const MmaPrep& p, bool) { in(p.images, (size_t)p.ng * p.S * p.nq * kMmaImageBytes); return BFLY_OK; }
  int mma_fw(const MmaPass& p) {
    ++passes;
    in(p.images, (size_t)p.S * p.nq * kMmaImageBytes);
    if (p.in_t) plane(p.in_t, p); else io(p.in, p);
    if (p.out_t) plane(p.out_t, p); else io(p.out, p);
    return BFLY_OK;
  }
  int mma_bw(const MmaPass& p, int ctas) {
    ++passes;
    in(p.images, (size_t)p.S * p.nq * kMmaImageBytes);
    if (p.in_t) plane(p.in_t, p); else io(p.in, p);
    if (p.x_t) plane(p.x_t, p); else io(p.x, p);
    if (p.out_t) plane(p.out_t, p); else io(p.out, p);
    // the last slot that a CTA can leave (mma_slot)
    const int used = mma_ctas(p.geo, (int64_t)p.S * p.nq * p.nt, ctas);
    const int64_t last = mma_slot(p.geo, p.parts, (int64_t)p.S * p.nq - 1, p.parts.of(p.nt - 1), (used >> p.geo.sib) - 1) + 1;
    in(p.slots, (size_t)last * kMmaSlotFloats * sizeof(float));
    if (p.bias_slots) in(p.bias_slots, (size_t)last * kMmaCols * sizeof(float));
    return BFLY_OK;
  }
  int mma_post(const MmaPost&, bool) { return BFLY_OK; }
};

// A layer: bias, gradients of everything.
template <typename T> int dry_layer(const Problem& q, int out_total, bool save, size_t skew, int* passes) {
  DryExec ex;
  const int64_t n = (int64_t)1 << q.log_n, DX = std::max<int64_t>(q.in_size, n);
  int64_t stk[2];
  twiddle_stack_sizes(q, stk);
  T* tw2 = ex.buffer<T>(q.S * stk[0] * sizeof(T)), *tw4 = ex.buffer<T>(q.S * stk[1] * sizeof(T));
  T* d2 = ex.buffer<T>(q.S * stk[0] * sizeof(T)), *d4 = ex.buffer<T>(q.S * stk[1] * sizeof(T));
  T* x = ex.buffer<T>((size_t)q.B * q.in_size * sizeof(T)), *out = ex.buffer<T>((size_t)q.B * q.S * n * sizeof(T));
  T* g = ex.buffer<T>((size_t)q.B * out_total * sizeof(T)), *dx = ex.buffer<T>((size_t)q.B * (q.S > 1 ? q.in_size : DX) * sizeof(T));
  T* bias = ex.buffer<T>(out_total * sizeof(T)), *db = ex.buffer<T>(out_total * sizeof(T));
  const int64_t kept = save ? layer_snapshot_need<T>(q, out_total) : 0;
  if (kept < 0) return (int)kept;
  const int64_t own = layer_bw_need<T>(q, out_total, kept > 0);
  if (own < 0) return (int)own;
  const size_t fws = kept > 0 || q.base4 ? 0 : fw_workspace_bytes<T>(q);
  char* k = ex.buffer<char>(kept, skew), *f = ex.buffer<char>(fws, skew), *w = ex.buffer<char>(own, skew);
  int rc = drive_layer_fw<T>(ex, q, tw2, tw4, x, q.in_size, out, bias, out_total, k, kept, f, fws);
  if (rc == BFLY_OK) rc = drive_layer_bw<T>(ex, q, tw2, tw4, x, q.in_size, g, out_total, d2, d4, dx, db, out_total, k, kept, w, own);
  *passes = ex.passes;
  return rc ? rc : (ex.outside ? 1 : 0);
}

// Is the plan of the passes one?  Groups that hold all stages in order, windows that hold their bits, blocks that tile the
// row, CTAs that take every tile once and leave no two sums in one slot.  0, or the number of what is wrong.
template <typename T> int check_mma_plan(const Problem& q, int most) {
  MmaLayout L;
  if (!mma_layout<T>(q, L)) return 0;
  const std::vector<Stage> st = problem_stages(q);
  const int cols = 1 << L.log_nf;
  int next = 0;
  if (L.g.size() > (size_t)kMmaMaxGroups) return 1;
  for (const MmaGroup& g : L.g) {
    if (g.t0 != next || g.t1 <= g.t0 || g.nst != g.t1 - g.t0) return 2;
    next = g.t1;
    int weight = 0, active = 0;
    for (int k = 0; k < g.nst; ++k) {
      const MmaStage& m = g.st[k];
      const Stage& s = st[g.t0 + k];
      weight += m.radix == 4 ? 2 : 1;
      for (int b = 0; b < (m.radix == 4 ? 2 : 1); ++b) {
        active |= 1 << (m.lbit + b);
        if (g.geo.col(1 << (m.lbit + b + L.F)) != 1 << (s.bit + b + L.F)) return 3;  // the window's bit is the row's
      }
      if (m.gbit != s.bit || m.tw_off != s.tw_off || m.which != s.which || m.radix != s.radix) return 4;
    }
    if (weight > kMmaMaxStages || (active & g.passive) || (active | g.passive) != (kMmaCols >> L.F) - 1) return 5;
    std::vector<char> seen(cols, 0);
    for (int b = 0; b < L.nq; ++b)
      for (int j = 0; j < kMmaCols; ++j) {
        const int c = g.geo.base(b) + g.geo.col(j);
        if (c < 0 || c >= cols || seen[c]++) return 6;
      }
    // the work, as Walk takes it
    const int64_t blocks = (int64_t)q.S * L.nq, nt = L.nt;
    const int ctas = mma_ctas(g.geo, blocks * nt, most), sib = g.geo.sib, G = ctas >> sib;
    if (ctas < 1 || blocks % (1 << sib)) return 7;
    const int64_t W = (blocks >> sib) * nt;
    std::vector<char> tile(blocks * nt, 0), slot(L.slots_per_group(q.S), 0);
    std::vector<int64_t> owner(slot.size(), -1);
    for (int cta = 0; cta < ctas; ++cta) {
      const int c = cta >> sib;
      const int64_t begin = mma_first_tile(W, G, c), end = mma_first_tile(W, G, c + 1);
      for (int64_t w = begin; w < end; ++w) {
        if (mma_cta_of(W, G, w) != c) return 8;
        const int64_t block = ((w / nt) << sib) + (cta & ((1 << sib) - 1));
        if (tile[block * nt + w % nt]++) return 9;
        const int t = (int)(w % nt), part = L.parts.of(t);
        auto leave = [&](int64_t at) {
          if (at < 0 || at >= (int64_t)slot.size() || slot[at]++) return false;
          owner[at] = block;
          return true;
        };
        if (w == begin && L.parts.begins(t) && !leave(mma_slot(g.geo, L.parts, block, part - 1, c))) return 10;
        if ((t + 1 == nt || w + 1 == end || L.parts.ends(t)) && !leave(mma_slot(g.geo, L.parts, block, part, c))) return 10;
      }
    }
    // what is added up for a block: slots that were left for it, all of them
    int64_t left = 0, added = 0;
    for (char s : slot) left += s;
    for (int64_t block = 0; block < blocks; ++block) {
      const int64_t first = (block >> sib) * nt;
      const int64_t s0 = mma_slot(g.geo, L.parts, block, 0, mma_cta_of(W, G, first));
      const int64_t s1 = mma_slot(g.geo, L.parts, block, L.parts.of((int)nt - 1), mma_cta_of(W, G, first + nt - 1));
      for (int64_t s = s0; s <= s1; s += 1 << sib, ++added)
        if (owner[s] != block) return 13;
    }
    if (left != added) return 14;
    for (char t : tile)
      if (!t) return 11;
  }
  return next == (int)st.size() ? -(int)L.g.size() : 12;
}

// how: 0 the operator with saved activations and a work space of its own, 1 the backward that makes them itself.
template <typename T> int dry_step(Problem q, int how, size_t skew, int* passes) {
  DryExec ex;
  const int64_t n = (int64_t)1 << q.log_n, DX = std::max<int64_t>(q.in_size, n);
  int64_t stk[2];
  twiddle_stack_sizes(q, stk);
  T* tw2 = ex.buffer<T>(q.S * stk[0] * sizeof(T)), *tw4 = ex.buffer<T>(q.S * stk[1] * sizeof(T));
  T* d2 = ex.buffer<T>(q.S * stk[0] * sizeof(T)), *d4 = ex.buffer<T>(q.S * stk[1] * sizeof(T));
  const size_t BS = (size_t)q.B * q.S;
  T* x = ex.buffer<T>(BS * q.in_size * sizeof(T)), *out = ex.buffer<T>(BS * n * sizeof(T));
  T* g = ex.buffer<T>(BS * q.out_size * sizeof(T)), *dx = ex.buffer<T>(BS * DX * sizeof(T));
  const int64_t x_sB = (int64_t)q.S * q.in_size, g_sB = (int64_t)q.S * q.out_size;
  int rc = BFLY_OK;
  if (how == 0) {
    const int64_t kept = bw_snapshot_need<T>(q), own = mma_either<T>(q, [](const Problem& d, const MmaLayout& L) { return mma_bw_need<T>(d, L, true) + kMmaSpare; });
    if (kept < 0) return (int)kept;
    char* k = ex.buffer<char>(kept, skew), *w = ex.buffer<char>(own, skew);
    rc = drive_fw_saving<T>(ex, q, tw2, tw4, x, x_sB, q.in_size, out, k, kept);
    if (rc == BFLY_OK)
      rc = drive_bw<T>(ex, q, tw2, tw4, x, x_sB, q.in_size, g, g_sB, q.out_size, d2, d4, dx, k, kept, true, 0, w, own);
  } else {
    const int64_t need = bw_workspace_need<T>(q);
    if (need < 0) return (int)need;
    rc = drive_bw<T>(ex, q, tw2, tw4, x, x_sB, q.in_size, g, g_sB, q.out_size, d2, d4, dx, ex.buffer<char>(need, skew), need);
  }
  *passes = ex.passes;
  return rc ? rc : (ex.outside ? 1 : 0);
}
}  // namespace
extern "C" {
// 0, a status of the library, or 1: a launch left the buffers it was given
int bfly_emul_dry_step(int dtype, int base4, int how, int64_t skew, int B, int S, int log_n, int nblocks, int in_size, int out_size, int inc, int* passes) {
  Problem q{B, S, log_n, nblocks, in_size, out_size, inc != 0, base4 != 0};
  if (const int rc = check_problem(q)) return rc;
  return dtype == 0 ? dry_step<float>(q, how, (size_t)skew, passes) : dry_step<cf>(q, how, (size_t)skew, passes);
}
int bfly_emul_dry_layer(int dtype, int base4, int save, int64_t skew, int B, int S, int log_n, int nblocks, int in_size, int out_total, int inc, int* passes) {
  Problem q{B, S, log_n, nblocks, in_size, 1 << log_n, inc != 0, base4 != 0};
  if (const int rc = check_problem(q)) return rc;
  return dtype == 0 ? dry_layer<float>(q, out_total, save != 0, (size_t)skew, passes) : dry_layer<cf>(q, out_total, save != 0, (size_t)skew, passes);
}
// minus the number of groups, 0 where the passes do not run, or what is wrong
int bfly_emul_check_mma_plan(int dtype, int base4, int B, int S, int log_n, int nblocks, int inc, int ctas) {
  Problem q{B, S, log_n, nblocks, 1 << log_n, 1 << log_n, inc != 0, base4 != 0};
  if (const int rc = check_problem(q)) return rc;
  return dtype == 0 ? check_mma_plan<float>(q, ctas) : check_mma_plan<cf>(q, ctas);
}
}
