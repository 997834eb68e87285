// Score form of float32 attention on the tcgen05 tensor cores: the forward and grad_q (rows = queries).  Operands, products
// and rounding as in fm_dense_split.cu; here a CTA walks row tiles.
//
// A row tile used to be a CTA.  At 512 heads x 1000 causal tokens (d = 32) its column tiles took 12 300 (forward) and 14 500
// (grad_q) of the 20 800 and 25 400 cycles it held the SM; the rest went to its start (launch, tensor memory, first loads,
// row operands, first scores: 2 700 to 3 900), its end and the gap to the next one (1 700).  Now the loads, the scores and
// the products run on from one row tile to the next: its operands are loaded while the last one's columns are walked and
// copied to tensor memory when the last one's scores are done, and a row tile's result is stored after the first column tile
// of the next one is on its way.
//
// 352 threads: warps 0-7 compute (warp % 4 = TMEM lane quarter = 32 rows, warp / 4 = half of the tile's 64 columns, and half of
// the features when accumulators are read), warp 8 loads tiles by TMA, warp 9 issues X Y^T and U Z^T, warp 10 the accumulating
// products.  S and W are refilled as soon as they are in registers.  The forward at d = 32 needs so little that two CTAs
// share an SM, and one's chain from scores to sums runs under the other's.  All waits are bounded.
//
// Measured (B200, us, a CTA per row tile / now): 512 heads x 1000 causal, d = 32: forward 303 / 220 (after the
// operands' preparation, as in a step, 304 / 241), grad_q 370 / 290; 60 heads x
// 4000 unmasked, d = 32: 687 / 605, 815 / 735; 64 heads x 1000 causal, d = 64: 60 / 54, 97 / 89.  What bounds it: tensor pipe
// and CUDA cores (ALU) are each busy for half of the time (forward at d = 32: 780 and 620 of 1 400 cycles a tile).
#include "fm_dense_split.cuh"

namespace fm {

__device__ int g_split_rows_status = 0;

namespace {
using namespace sm100;
using namespace split;

constexpr int kProducerWarp = 8, kIssuerWarp = 9, kAccIssuerWarp = 10;

// CTAS: per SM.  Two have 256 TMEM columns and 112 KB each, and the warps that load and issue give registers to those that
// compute.
template <int D, int MODE, int CTAS>
struct SR {
  static constexpr bool HAS_U = MODE != MODE_FWD;
  static constexpr int THREADS = CTAS == 2 ? 384 : 352, REGS = CTAS == 2 ? 80 : 168, REGS_COMPUTE = 96, REGS_OTHER = 48;
  static_assert(32 * kComputeWarps * REGS_COMPUTE + (384 - 32 * kComputeWarps) * REGS_OTHER <= 384 * 80,
                "the shares of the warpgroups add up to what the block is launched with");
  static constexpr int ROW_SUB = BM * D * 2, ROW_TILE = 3 * ROW_SUB, ROWS = (HAS_U ? 2 : 1) * ROW_TILE;
  static constexpr int COL_SUB = BN * D * 2, COL_TILE = 3 * COL_SUB, STAGE = 2 * COL_TILE;
  static constexpr int NXB = D == 32 && HAS_U ? 2 : 1;     // buffers of row operands
  static constexpr int OFF_U = ROW_TILE, OFF_ST = NXB * ROWS;
  static constexpr int NS = HAS_U ? (D == 64 ? 2 : 4) : 3;  // (two stages leave the next scores waiting for their tile)
  static constexpr int OFF_VEC = OFF_ST + NS * STAGE;       // row-sum exchange
  static constexpr int OFF_BAR = OFF_VEC + 2 * 2 * BM * 4;
  static constexpr int NBAR = 2 * NXB + 1 + 2 * NS + 5;
  static constexpr int OFF_TMEM = OFF_BAR + NBAR * 8;
  static constexpr int SMEM = OFF_TMEM + 16 + 1024;
  static_assert(CTAS * (SMEM + 1024) <= 228 * 1024, "shared memory of an SM");
  // the row operands are copied to tensor memory where there is room (3 d / 2 columns each)
  static constexpr bool IN_T = CTAS == 1;
  // TMEM columns: S 64 | W 64 (DQ) | three parts of 32 packed columns | accumulator of 64 columns (d = 32: leading terms 32,
  // cross terms with ym or yl 32) | row operands
  enum : int {
    T_S = 0, T_W = BN, T_E = HAS_U ? 2 * BN : BN, T_A = T_E + 96, T_X = T_A + 64, T_U = T_X + 3 * D / 2, T_COLS = 512 / CTAS
  };
  static constexpr int CH = CTAS == 2 ? 8 : 16;             // pairs of columns whose parts a thread holds at once
  // Whether a pair is formed and split in one go.  us, d = 64: forward 269 instead of 277 (448 row tiles of 4000 columns), grad_q 483
  // instead of 495; but grad_q of d = 32 198 instead of 190 (2400 of 1000)
  static constexpr bool AT_ONCE = CTAS == 1 && D == 64;
};

__device__ __forceinline__ void put(uint32_t taddr, const uint32_t (&r)[8]) { tmem_st8(taddr, r); }
__device__ __forceinline__ void put(uint32_t taddr, const uint32_t (&r)[16]) { tmem_st16(taddr, r); }

__device__ __forceinline__ void report(int code) { atomicCAS(&g_split_rows_status, 0, code); }

template <int D, int MODE, int CTAS>
__global__ void __launch_bounds__(SR<D, MODE, CTAS>::THREADS, CTAS)
split_rows_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmU,
             const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmZ, const SplitArgs a) {
  using C = SR<D, MODE, CTAS>;
  constexpr int NS = C::NS, NXB = C::NXB;
  constexpr bool HAS_U = C::HAS_U;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + C::OFF_BAR;
  // barrier map: x[NXB] | x free[NXB] | x in tensor memory | full[NS] | empty[NS] | s_full | s_free | p_full | pv_done | row sums
  auto BAR_X = [&](int b) { return bar0 + 8u * b; };
  auto BAR_XE = [&](int b) { return bar0 + 8u * (NXB + b); };
  const uint32_t BAR_XT = bar0 + 8u * (2 * NXB);
  auto BAR_FULL = [&](int s) { return bar0 + 8u * (2 * NXB + 1 + s); };
  auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (2 * NXB + 1 + NS + s); };
  const uint32_t BAR_S = bar0 + 8u * (2 * NXB + 1 + 2 * NS), BAR_SFREE = BAR_S + 8, BAR_P = BAR_S + 16, BAR_PV = BAR_S + 24, BAR_RS = BAR_S + 32;
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + C::OFF_TMEM);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int b = 0; b < NXB; ++b) {
      mbar_init(BAR_X(b), 1);
      mbar_init(BAR_XE(b), C::IN_T ? kComputeWarps : 1);
    }
    mbar_init(BAR_XT, kComputeWarps);
    for (int s = 0; s < NS; ++s) {
      mbar_init(BAR_FULL(s), 1);
      mbar_init(BAR_EMPTY(s), 1);
    }
    mbar_init(BAR_S, 1);
    mbar_init(BAR_SFREE, kComputeWarps);
    mbar_init(BAR_P, kComputeWarps);
    mbar_init(BAR_PV, 1);
    mbar_init(BAR_RS, kComputeWarps);
    mbar_fence_init();
  }
  if (warp == kIssuerWarp) tmem_alloc(smem_u32((const void*)tmem_slot), C::T_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // every role walks the same row tiles and counts their column tiles in g
  Rows w;
  w.open(a);
  int g = 0;
  bool ok = true;
  if (warp >= kComputeWarps) {
    if constexpr (CTAS == 2) regs_down<C::REGS_OTHER>();
    if (warp == kProducerWarp) {
      // ================= TMA producer =================
      if (lane == 0) {
        tma_prefetch_desc(&tmX);
        if (HAS_U) tma_prefetch_desc(&tmU);
        tma_prefetch_desc(&tmY);
        tma_prefetch_desc(&tmZ);
      }
      for (; ok && w.live(a); w.next(a)) {
        const int b = w.m % NXB;
        if (!mbar_wait(BAR_XE(b), (uint32_t)(((w.m / NXB) & 1) ^ 1))) { report(1); break; }
        if (lane == 0) {
          mbar_expect_tx(BAR_X(b), C::ROWS);
          const uint32_t dst = sbase + b * C::ROWS;
          for (int p = 0; p < 3; ++p) {
            tma_load_3d(dst + p * C::ROW_SUB, &tmX, BAR_X(b), p * D, w.r0, w.head);
            if (HAS_U) tma_load_3d(dst + C::OFF_U + p * C::ROW_SUB, &tmU, BAR_X(b), p * D, w.r0, w.head);
          }
        }
        const int h = w.head / a.ratio;
        for (int i = 0; i < w.j; ++i, ++g) {
          const int s = g % NS;
          if (!mbar_wait(BAR_EMPTY(s), (uint32_t)(((g / NS) & 1) ^ 1))) { report(1); ok = false; break; }
          if (lane == 0) {
            mbar_expect_tx(BAR_FULL(s), C::STAGE);
            const uint32_t dst = sbase + C::OFF_ST + s * C::STAGE;
            for (int p = 0; p < 3; ++p) {
              tma_load_3d(dst + p * C::COL_SUB, &tmY, BAR_FULL(s), p * D, (w.tb + i) * BN, h);
              tma_load_3d(dst + C::COL_TILE + p * C::COL_SUB, &tmZ, BAR_FULL(s), p * D, (w.tb + i) * BN, h);
            }
          }
        }
      }
    } else if (warp == kIssuerWarp) {
      // ================= MMA issuer of the S / W products (whole warp, one elected lane issues) ============
      for (; ok && w.live(a); w.next(a)) {
        const int b = w.m % NXB;
        if (!C::IN_T) ok = mbar_wait_warp(BAR_X(b), (uint32_t)((w.m / NXB) & 1));
        if (ok && C::IN_T) ok = mbar_wait_warp(BAR_XT, (uint32_t)(w.m & 1));
        if (!ok) { report(2); break; }
        const uint32_t x_lo = desc_lo(sbase + b * C::ROWS, 16);
        for (int i = 0; i < w.j; ++i, ++g) {
          const int s = g % NS;
          if (!mbar_wait_warp(BAR_FULL(s), (uint32_t)((g / NS) & 1))) { report(3); ok = false; break; }
          if (g >= 1 && !mbar_wait_warp(BAR_SFREE, (uint32_t)((g - 1) & 1))) { report(4); ok = false; break; }
          tc_fence_after();
          const uint32_t y_lo = desc_lo(sbase + C::OFF_ST + s * C::STAGE, 16);
          if (elect_one()) {
            issue_scores<D, C::IN_T>(tmem + C::T_S, C::IN_T ? tmem + C::T_X : x_lo, y_lo);
            if constexpr (HAS_U) issue_scores<D, true>(tmem + C::T_W, tmem + C::T_U, y_lo + (C::COL_TILE >> 4));
            umma_commit(BAR_S);
            if (!C::IN_T && i + 1 == w.j) umma_commit(BAR_XE(b));
          }
          __syncwarp();
        }
      }
      __syncwarp();
    } else if (warp == kAccIssuerWarp) {
      // ================= MMA issuer of the accumulating products =================
      for (; ok && w.live(a); w.next(a)) {
        for (int i = 0; i < w.j; ++i, ++g) {
          const int s = g % NS;
          if (!mbar_wait_warp(BAR_FULL(s), (uint32_t)((g / NS) & 1)) || !mbar_wait_warp(BAR_P, (uint32_t)(g & 1))) {
            report(5);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t y_mn = desc_mn(sbase + C::OFF_ST + s * C::STAGE, D);
          if (elect_one()) {
            issue_acc<D>(tmem + C::T_A, tmem + C::T_E, HAS_U ? y_mn : y_mn + (C::COL_TILE >> 4));
            umma_commit(BAR_PV);
            umma_commit(BAR_EMPTY(s));
          }
          __syncwarp();
        }
      }
      __syncwarp();
    }
  } else {
    // ================= compute warps =================
    if constexpr (CTAS == 2) regs_up<C::REGS_COMPUTE>();
    const int cpart = warp >> 2, qd = warp & 3, rl = qd * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)(qd * 32) << 16);
    const uint64_t A0v = pack2(a.a0, a.a0);
    // statistics of the next row tile's heads and dvec of its row, asked for early
    stat_t st_q = 0, st_k = 0;
    float dl_next = 0.f;
    auto ask = [&](const Rows& x) {
      if (a.stat_q) {
        st_q = __ldg(a.stat_q + x.head);
        st_k = __ldg(a.stat_k + x.head / a.ratio);
      }
      if (MODE == MODE_DQ) dl_next = x.r0 + rl < a.nrows ? __ldg(a.dvec + (size_t)x.head * a.nrows + x.r0 + rl) : 0.f;
    };
    // copies the row operands to tensor memory: column c of a part holds elements 2c and 2c+1 of the row; the two warps of
    // a lane quarter take alternate parts.  (16-byte pieces, XOR-swizzled by the row's place in its swizzle atom)
    auto copy_rows = [&](int m) -> bool {
      if constexpr (C::IN_T) {
        const int b = m % NXB, sw = D == 64 ? (rl & 7) : ((rl >> 1) & 3);
        if (!mbar_wait(BAR_X(b), (uint32_t)((m / NXB) & 1))) { report(6); return false; }
        for (int it = cpart; it < (HAS_U ? 6 : 3); it += 2) {
          const uint32_t src = sbase + b * C::ROWS + it * C::ROW_SUB + rl * (D * 2), dst = tl + C::T_X + it * (D / 2);
#pragma unroll
          for (int h = 0; h < D / 32; ++h) {
            uint32_t x[16];
#pragma unroll
            for (int pc = 0; pc < 4; ++pc) {
              const ulonglong2 v = lds_v2(src + (((4 * h + pc) ^ sw) << 4));
              x[4 * pc] = (uint32_t)v.x; x[4 * pc + 1] = (uint32_t)(v.x >> 32);
              x[4 * pc + 2] = (uint32_t)v.y; x[4 * pc + 3] = (uint32_t)(v.y >> 32);
            }
            tmem_st16(dst + 16 * h, x);
          }
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(BAR_XT);
          if (C::IN_T) mbar_arrive(BAR_XE(b));
        }
      }
      return true;
    };
    uint64_t run[D / 4];
    auto clear = [&]() {
#pragma unroll
      for (int e = 0; e < D / 4; ++e) run[e] = 0ull;
    };
    clear();
    // a finished row tile: each compute thread owns half of the features of one row
    auto finish = [&](int m, int head, int r0, uint64_t sums) -> bool {
      const int row = r0 + rl;
      const bool row_ok = row < a.nrows;
      const size_t grow = (size_t)head * a.nrows + (row_ok ? row : 0), at = grow * D + cpart * (D / 2);
      if constexpr (MODE == MODE_FWD) {
        float* const rows_sum = (float*)(smem + C::OFF_VEC) + (m & 1) * 2 * BM;
        float lo, hi;
        unpack2(sums, lo, hi);
        rows_sum[cpart * BM + rl] = lo + hi;
        // (a warp that gave up is not waited for without a limit; the next sums go to the other buffer)
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR_RS);
        if (!mbar_wait(BAR_RS, (uint32_t)(m & 1))) { report(11); return false; }
        if (row_ok)
          store_forward<D>(a, run, grow, cpart, rows_sum[rl] + rows_sum[BM + rl] + (a.den_add ? a.den_add[grow] : 0.f));
      } else {
        float part = 0.f;
        if (row_ok) part = store_half<D>(run, a.o1 + at, a.o1_add ? a.o1_add + at : nullptr, a.dots ? a.x + at : nullptr, 1.f);
        if (a.dots) {
#pragma unroll
          for (int k = 16; k >= 1; k >>= 1) part += __shfl_xor_sync(0xffffffffu, part, k);
          if (lane == 0) atomicAdd(a.dots + head, part);
        }
      }
      clear();
      return true;
    };
    // the row tile whose last products are still under way: its head, first row and row sums
    int last_head = -1, last_r0 = 0;
    uint64_t last_sums = 0ull;
    ask(w);
    ok = copy_rows(0);
    while (ok && w.live(a)) {
      const float c = a.stat_q ? stat_scale(&st_q, 0, a.lim) * stat_scale(&st_k, 0, a.lim) : 1.f;
      const float A1 = a.a1 * c, A2 = a.a2 * c * c, A2f = HAS_U ? 2.f * A2 : A2;      // DQ: of the derivative
      const uint64_t A1v = pack2(A1, A1), A2v = pack2(A2f, A2f);
      const int limcol = a.mask ? min(a.ncols - 1, w.r0 + rl + a.off) : a.ncols - 1;   // last column kept
      const uint64_t ndl_row = pack2(-dl_next, -dl_next);
      uint64_t rs2 = 0ull;
      for (int i = 0; i < w.j; ++i, ++g) {
        if (!mbar_wait(BAR_S, (uint32_t)(g & 1))) { report(7); ok = false; break; }
        tc_fence_after();
        uint32_t sv[32], wv[HAS_U ? 32 : 1];
        tmem_ld32(tl + C::T_S + cpart * 32, sv);
        if constexpr (HAS_U) {
          tmem_ld32(tl + C::T_W + cpart * 32, wv);
          tmem_wait_ld(sv, wv);
        } else {
          tmem_wait_ld(sv);
        }
        // S and W of this tile are in registers: the next tile's may be issued
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR_SFREE);
        if (i + 1 == w.j) {          // the row tile's score products are done: the next one's operands take their place
          Rows n = w;
          n.next(a);
          if (n.live(a)) {
            ask(n);
            if (!(ok = copy_rows(n.m))) break;
          }
        }
        const int c0 = (w.tb + i) * BN + cpart * 32;          // first of this warp's 32 columns
        const bool need_mask = c0 + 32 > a.ncols || (a.mask && c0 + 31 > w.r0 + qd * 32 + a.off);
        // P or E of a pair of columns.  The mask test stays outside the loops so that each is one basic block of independent
        // pairs
        auto value = [&](int e) {
          const uint64_t s2 = pack2u(sv[2 * e], sv[2 * e + 1]), f = fma2(A2v, s2, A1v);
          if constexpr (HAS_U) return mul2(f, add2(pack2u(wv[2 * e], wv[2 * e + 1]), ndl_row));
          else return fma2(f, s2, A0v);
        };
        auto zero = [&](int e) { return c0 + e > limcol; };
        uint64_t ts2 = 0ull;                                  // row sums of this tile
        if constexpr (C::AT_ONCE) {
          uint32_t e3[3][16];
          auto split = [&](int e, uint64_t v) {
            if constexpr (!HAS_U) ts2 = add2(ts2, v);
            split3(v, e3[0][e], e3[1][e], e3[2][e]);
          };
          if (!need_mask) {
#pragma unroll
            for (int e = 0; e < 16; ++e) split(e, value(e));
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              float lo, hi;
              unpack2(value(e), lo, hi);
              split(e, pack2(zero(2 * e) ? 0.f : lo, zero(2 * e + 1) ? 0.f : hi));
            }
          }
          // the previous tile's products must be done before their operands are overwritten
          if (g > 0) {
            if (!mbar_wait(BAR_PV, (uint32_t)((g - 1) & 1))) { report(9); ok = false; break; }
            tc_fence_after();
          }
#pragma unroll
          for (int p = 0; p < 3; ++p) tmem_st16(tl + C::T_E + 32 * p + cpart * 16, e3[p]);
        } else {
          // in the place of the scores first
          auto keep = [&](int e, float lo, float hi) { sv[2 * e] = __float_as_uint(lo); sv[2 * e + 1] = __float_as_uint(hi); };
          float lo, hi;
          if (!need_mask) {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              unpack2(value(e), lo, hi);
              keep(e, lo, hi);
            }
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              unpack2(value(e), lo, hi);
              keep(e, zero(2 * e) ? 0.f : lo, zero(2 * e + 1) ? 0.f : hi);
            }
          }
#pragma unroll
          for (int k = 0; k < 16 / C::CH; ++k) {
            uint32_t e3[3][C::CH];                            // three packed parts each of CH pairs
#pragma unroll
            for (int e = 0; e < C::CH; ++e) {
              const int x = 2 * (C::CH * k + e);
              const uint64_t v = pack2u(sv[x], sv[x + 1]);
              if constexpr (!HAS_U) ts2 = add2(ts2, v);
              split3(v, e3[0][e], e3[1][e], e3[2][e]);
            }
            if (k == 0 && g > 0) {                            // (as above)
              if (!mbar_wait(BAR_PV, (uint32_t)((g - 1) & 1))) { report(9); ok = false; break; }
              tc_fence_after();
            }
#pragma unroll
            for (int p = 0; p < 3; ++p) put(tl + C::T_E + 32 * p + cpart * 16 + C::CH * k, e3[p]);
          }
          if (!ok) break;
        }
        if (MODE == MODE_FWD) rs2 = add2(rs2, ts2);
        // its sums are taken over before the arrival below lets this tile's products replace them
        if (g > 0) promote<D>(run, tl + C::T_A, cpart);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR_P);
        if (i == 0 && last_head >= 0 && !(ok = finish(w.m - 1, last_head, last_r0, last_sums))) break;
      }
      last_head = w.head;
      last_r0 = w.r0;
      last_sums = rs2;
      w.next(a);
    }
    if (ok && last_head >= 0) {
      if (!mbar_wait(BAR_PV, (uint32_t)((g - 1) & 1))) report(10);
      else {
        tc_fence_after();
        promote<D>(run, tl + C::T_A, cpart);
        finish(w.m - 1, last_head, last_r0, last_sums);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kIssuerWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, C::T_COLS);
  }
}

template <int D, int MODE, int CTAS>
int launch_rows(const Ctx& c, const char* name, const void* x, const void* u, const void* y, const void* z, SplitArgs a) {
  using C = SR<D, MODE, CTAS>;
  const fastmax_problem& p = c.p;
  if (p.bh == 0 || p.nq == 0) return FASTMAX_OK;
  CUtensorMap tx, tu, ty, tz;
  int rc;
  if ((rc = split_map<D>(&tx, x, p.bh, p.nq, BM))) return rc;
  if ((rc = split_map<D>(&tu, u, p.bh, p.nq, BM))) return rc;
  if ((rc = split_map<D>(&ty, y, p.bhkv, p.nk, BN))) return rc;
  if ((rc = split_map<D>(&tz, z, p.bhkv, p.nk, BN))) return rc;
  long long blocks;
  if ((rc = set_sizes(p, p.bh, p.nq, p.nk, &a, &blocks))) return rc;
  a.order = row_order(p, a.heads, a.ntr, CTAS, a.chunk);
  const auto kernel = split_rows_kernel<D, MODE, CTAS>;
  FM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
  const unsigned grid = (unsigned)(blocks < 148 * CTAS ? blocks : 148 * CTAS);
  FM_LAUNCH(name, c.stream, (kernel<<<grid, C::THREADS, C::SMEM, c.stream>>>(tx, tu, ty, tz, a)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

}  // namespace

// Which problems' forward (MODE_FWD) and grad_q (MODE_DQ) walk row tiles; fm_dense_split.cu has a CTA per row tile for the others.
// Measured, walk as part of that:
//   d = 32  forward (two CTAs per SM; one walking is 0 to 10 % slower than none): up to 148 row tiles 1.10 to 1.26.  Causal, up to 296: 0.76
//           to 0.99 of 128 to 300 columns, 1.03 to 1.16 of 384, 1.06 to 1.33 of 474, 1.1 to 1.7 above.  From 300 on 0.78 to 0.93 of up
//           to 1000 columns, but with 2100 to 4000 1.08 to 1.12 at 310 row tiles, 1.00 to 1.04 at 340, 0.92 to 0.98 from 370 on.
//           Unmasked 0.75 to 1.00, but 1.03 to 1.04 for 350 to 380 row tiles of 4000.
//           grad_q: up to 148 1.06 to 1.14 of 128 to 384 columns, 1.01 to 1.04 of 474 to 1000, 0.95 of 2000; above 0.77 to 1.03
//   d = 64  up to 148 row tiles 1.03 to 1.07.  Up to 296, causal: forward 0.88 to 0.98, grad_q 0.89 to 0.99 at 200 to 296 row tiles of 212
//           and 474 columns; of 1000 columns 1.03 at 200, 0.95 to 0.97 from 224 on; of 2000 1.05 and 1.03 at 224, 0.99 to 1.00 from 256
//           on; 160 row tiles 0.88 and 0.93 of 212 columns, 1.00 and 1.04 of 474, 1.07 and 1.04 of 1000.  Unmasked: forward 0.90 to
//           0.96 of 212 and 474, 0.97 to 0.98 of 1000, 1.00 to 1.02 of 2000; grad_q 0.92 to 0.99, 0.99 to 1.01, 1.02 to 1.05.  Above 296
//           0.84 to 1.01, but grad_q 1.00 to 1.04 unmasked, 3000 columns and more
bool split_rows_serve(const fastmax_problem& p, int mode, int chunk) {
  const long long tiles = (long long)p.bh * ((p.nq + BM - 1) / BM);
  const int most = chunk > 0 ? chunk : p.nk;         // columns of the longest row
  if (p.d == 32 && mode == MODE_DQ) return tiles > 148 || most > 1000;
  if (p.d == 64) {
    const int seen = p.mask ? most / 2 : most;       // mean columns of a row tile
    if (tiles > 2 * 148) return mode == MODE_FWD || seen <= 2000;
    return tiles > 148 && (p.mask ? 8 * (tiles - 148) >= seen : seen <= (mode == MODE_FWD ? 1000 : 500));
  }
  // the compute warps of two CTAs wait for registers that the block must have been launched with
  static std::atomic<int> regs{0};
  const bool second = tiles <= 2 * 148;
  const bool few = p.mask ? (second ? most > 320 : most > 1400 && tiles <= 370) : !second && most > 2800 && tiles <= 400;
  return tiles > 148 && !few &&
         launch_registers(split_rows_kernel<32, MODE_FWD, 2>, &regs) >= SR<32, MODE_FWD, 2>::REGS;
}
int split_rows_forward(const Ctx& c, const void* q, const void* k, const void* v, const SplitArgs& a) {
  if (c.p.d == 32) return launch_rows<32, MODE_FWD, 2>(c, "fm_dense_split_fwd", q, q, k, v, a);
  return launch_rows<64, MODE_FWD, 1>(c, "fm_dense_split_fwd", q, q, k, v, a);
}
int split_rows_dq(const Ctx& c, const void* q, const void* gs, const void* k, const void* v, const SplitArgs& a) {
  if (c.p.d == 32) return launch_rows<32, MODE_DQ, 1>(c, "fm_dense_split_dq", q, gs, k, v, a);
  return launch_rows<64, MODE_DQ, 1>(c, "fm_dense_split_dq", q, gs, k, v, a);
}

int split_rows_status(int* out, cudaStream_t stream) {
  FM_CUDA_TRY(cudaMemcpyFromSymbolAsync(out, g_split_rows_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
int split_rows_status_reset(cudaStream_t stream) {
  const int zero = 0;
  FM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_split_rows_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}

}  // namespace fm
