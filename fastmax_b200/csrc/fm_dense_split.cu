// Score form of float32 attention on the tcgen05 tensor cores, head dimension 32 or 64.
//
// Every float32 operand is the exact sum of three bf16 numbers, x = xh + xm + xl (8 significand bits each,
// rounded to nearest twice, the rest is exact), so a float32 product sum is six bf16 product sums
//   x.y = xh.yh + (xh.ym + xm.yh) + (xh.yl + xl.yh + xm.ym)  + terms below 2^-26 of the product,
// each exact per product and accumulated in float32.  The same holds for the score polynomial, which the
// compute warps split again before it becomes the operand of the accumulating products.
//
//   FWD   rows = queries, columns = keys:   P = f(X Y^T),              out  = (P Z) / row sum of P
//   DQ    rows = queries, columns = keys:   E = f'(X Y^T) (U Z^T - dvec_row),        grad_q = E Y
//   DKDV  rows = keys, columns = queries:   E = f'(X Y^T) (U Z^T - dvec_col),        grad_k = E Y,
//                                           P = f(X Y^T),                            grad_v = P Z
// with z (FWD, DQ) = v, u (DQ) = z (DKDV) = gs = grad_out / den and dvec = gs . out -- the sums of
// fm_dense_ffma.cu (reference fastmax_cuda_forward.cu:25-197, fastmax_cuda_backward.cu:26-871 and the
// second-order terms in `old stuff/*_quad.cu`).
//
// Rounding.  The tensor core adds sixteen products to a float32 accumulator and truncates, so a long chain of
// additions into one accumulator would drift by about half an ulp per step.  The chain is kept short: the
// small cross terms are added before the leading ones, and the TMEM accumulators hold ONE 64-column tile; the
// compute warps add every tile to float32 registers, rounded to nearest.
//
// Here are the preparation of the operands and the kernels of one CTA per 128-row tile: grad_k + grad_v, and the forward and
// grad_q of grids that those of fm_dense_split_rows.cu, whose CTAs go on from row tile to row tile, do not serve
// (split_rows_serve).  352 threads: warps 0-7 compute (warp % 4 = TMEM lane quarter = 32 rows, warp / 4 = half of the tile's 64
// columns, and half of the features when accumulators are read), warp 8 loads tiles by TMA, warp 9 issues X Y^T and U Z^T,
// warp 10 the accumulating products.  S and W are single buffers that are refilled as soon as they are in registers, so the
// tensor core works on the next tile's scores while the polynomial and the split of this one run on the CUDA cores.  All
// waits are bounded.
//
// Measured (B200, forward / grad_q / grad_k + grad_v, ms; the CUDA-core family on the same inputs in brackets):
//   512 heads x 1000 causal, d = 32:   0.22 / 0.29 / 0.53  (1.40 / 2.00 / 2.45); one after another in a step 0.24 / 0.29 / 0.54
//    64 heads x 4000 unmasked, d = 64: 1.07 / 1.81 / 3.05  (7.96 / 11.7 / 15.6)
// Error against float64 (2-norm, outputs and gradients): 0.8-3.7e-7 for 64 to 10 000 tokens where the CUDA-core
// family has 0.9e-7 to 2.4e-6.  What bounds grad_k + grad_v: the chain of hand-offs per 64-column tile (scores -> registers ->
// operand parts -> products -> sums), 2 950 cycles at d = 32 of which the polynomial and the splits take 1 550 and the tensor
// pipe 1 740, and a row tile's ends, a quarter of its time at 8 column tiles.  It does not gain from what serves the others:
// walking row tiles in one CTA costs it as much in registers as it saves (533 -> 528 us), sixteen compute warps instead of
// eight 558, two CTAs per SM with the parts in the place of the scores 607.  32 columns of S and W and six arrays of parts are
// held at once, and it spills at 168 registers (246 bytes of stores at d = 64, 28 at d = 32).
//
// Operands: split3_kernel writes each tensor once as rows of [h | m | l] (3 d bf16); each part of a tile is a tile of its own
// in shared memory, with rows of d bf16 swizzled over their whole length (128 or 64 bytes).
#include "fm_dense_split.cuh"

namespace fm {

__device__ int g_split_status = 0;

namespace {
using namespace sm100;
using namespace split;

constexpr int kThreads = 352, kProducerWarp = 8, kIssuerWarp = 9, kAccIssuerWarp = 10;

template <int D, int MODE>
struct SC {
  static constexpr bool rev = MODE == MODE_DKDV, HAS_U = MODE != MODE_FWD;
  static constexpr int ROW_SUB = BM * D * 2, ROW_TILE = 3 * ROW_SUB;
  static constexpr int COL_SUB = BN * D * 2, COL_TILE = 3 * COL_SUB, STAGE = 2 * COL_TILE;
  static constexpr int OFF_U = ROW_TILE, OFF_ST = (HAS_U ? 2 : 1) * ROW_TILE;
  static constexpr int NS = HAS_U ? (D == 64 ? 2 : 4) : 3;
  static constexpr int OFF_VEC = OFF_ST + NS * STAGE;       // per compute warp 2 x 32 floats; row-sum exchange
  static constexpr int OFF_BAR = OFF_VEC + kComputeWarps * 2 * 32 * 4;
  static constexpr int NBAR = 3 + 2 * NS + 4;
  static constexpr int OFF_TMEM = OFF_BAR + NBAR * 8;
  static constexpr int SMEM = OFF_TMEM + 16 + 1024;
  // TMEM columns: S 64 | W 64 | three parts of 32 packed columns (P, or E and P) | accumulators of 64 columns (d = 32: leading
  // terms 32, cross terms with ym or yl 32) | row operands as far as there is room (3 d / 2 columns each)
  enum : int {
    T_S = 0, T_W = BN, T_E = HAS_U ? 2 * BN : BN, T_P = T_E + 96, T_A1 = rev ? T_P + 96 : T_E + 96, T_A2 = T_A1 + 64,
    T_X = rev ? T_A2 + 64 : T_A1 + 64, T_U = T_X + 3 * D / 2, T_COLS = 512
  };
  static constexpr bool X_IN_T = !rev || D == 32, U_IN_T = MODE == MODE_DQ;
};

__device__ __forceinline__ void report(int code) { atomicCAS(&g_split_status, 0, code); }

template <int D, int MODE>
__global__ void __launch_bounds__(kThreads, 1)
split_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmU,
             const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmZ, const SplitArgs a) {
  using C = SC<D, MODE>;
  constexpr int NS = C::NS;
  constexpr bool rev = C::rev, HAS_U = C::HAS_U;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + C::OFF_BAR;
  // barrier map: x | done | x in tensor memory | full[NS] | empty[NS] | s_full | s_free | p_full | pv_done
  const uint32_t BAR_X = bar0, BAR_DONE = bar0 + 8, BAR_XT = bar0 + 16;
  auto BAR_FULL = [&](int s) { return bar0 + 8u * (3 + s); };
  auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (3 + NS + s); };
  const uint32_t BAR_S = bar0 + 8u * (3 + 2 * NS), BAR_SFREE = BAR_S + 8, BAR_P = BAR_S + 16, BAR_PV = BAR_S + 24;
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + C::OFF_TMEM);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // longest rows first (row_tile_of)
  int head, pidx;
  row_tile_of(blockIdx.x, a.order, a.ntr, head, pidx);
  const int r0 = (rev ? pidx : a.ntr - 1 - pidx) * BM;

  int tb = 0, te = (a.ncols + BN - 1) / BN;
  if (a.mask) {
    if (rev) tb = max(0, r0 - a.off) / BN;
    else te = min(te, (min(r0 + BM - 1, a.nrows - 1) + a.off) / BN + 1);
  }
  if (a.chunk > 0) {        // the row tile lies in one chunk (chunk % 256 == 0)
    const int cb = (r0 / a.chunk) * (a.chunk / BN);
    if (rev) te = min(te, cb + a.chunk / BN);
    else tb = cb;
  }
  // grouped heads: a key/value head walks its tile range once per query head of the group
  const int Jh = max(te - tb, 0), J = rev ? Jh * a.ratio : Jh;
  struct ColPos { int t, h; };
  const ColPos pos0 = {tb, rev ? head * a.ratio : head / a.ratio};
  auto advance = [&](ColPos& cp) {
    if (++cp.t >= tb + Jh && rev) { cp.t = tb; ++cp.h; }
  };

  if (tid == 0) {
    mbar_init(BAR_X, 1);
    mbar_init(BAR_DONE, 1);
    mbar_init(BAR_XT, kComputeWarps);
    for (int s = 0; s < NS; ++s) {
      mbar_init(BAR_FULL(s), 1);
      mbar_init(BAR_EMPTY(s), 1);
    }
    mbar_init(BAR_S, 1);
    mbar_init(BAR_SFREE, kComputeWarps);
    mbar_init(BAR_P, kComputeWarps);
    mbar_init(BAR_PV, 1);
    mbar_fence_init();
  }
  if (warp == kIssuerWarp) tmem_alloc(smem_u32((const void*)tmem_slot), C::T_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // where the two column halves of a row exchange their row sums (FWD)
  float* const rows_sum = (float*)(smem + C::OFF_VEC);
  bool ok_compute = true;
  uint64_t run1[D / 4], run2[rev ? D / 4 : 1];
  if (warp == kProducerWarp) {
    // ================= TMA producer =================
    if (lane == 0 && J > 0) {
      tma_prefetch_desc(&tmX);
      if (HAS_U) tma_prefetch_desc(&tmU);
      tma_prefetch_desc(&tmY);
      tma_prefetch_desc(&tmZ);
      mbar_expect_tx(BAR_X, (HAS_U ? 2 : 1) * C::ROW_TILE);
      for (int p = 0; p < 3; ++p) {
        tma_load_3d(sbase + p * C::ROW_SUB, &tmX, BAR_X, p * D, r0, head);
        if (HAS_U) tma_load_3d(sbase + C::OFF_U + p * C::ROW_SUB, &tmU, BAR_X, p * D, r0, head);
      }
    }
    ColPos pc = pos0;
    for (int j = 0; j < J; ++j, advance(pc)) {
      const int s = j % NS;
      if (!mbar_wait(BAR_EMPTY(s), (((j / NS) & 1) ^ 1))) { report(1); break; }
      if (lane == 0) {
        mbar_expect_tx(BAR_FULL(s), C::STAGE);
        const uint32_t dst = sbase + C::OFF_ST + s * C::STAGE;
        for (int p = 0; p < 3; ++p) {
          tma_load_3d(dst + p * C::COL_SUB, &tmY, BAR_FULL(s), p * D, pc.t * BN, pc.h);
          tma_load_3d(dst + C::COL_TILE + p * C::COL_SUB, &tmZ, BAR_FULL(s), p * D, pc.t * BN, pc.h);
        }
      }
    }
  } else if (warp == kIssuerWarp) {
    // ================= MMA issuer of the S / W products (whole warp, one elected lane issues) ============
    if (J > 0) {
      const uint32_t x_lo = desc_lo(sbase, 16), u_lo = desc_lo(sbase + C::OFF_U, 16);
      const uint32_t st_k = desc_lo(sbase + C::OFF_ST, 16);   // stage 0, K-major view
      bool ok = mbar_wait_warp(BAR_X, 0);
      if (ok && C::X_IN_T) ok = mbar_wait_warp(BAR_XT, 0);
      if (!ok) report(2);
      tc_fence_after();
      for (int j = 0; ok && j < J; ++j) {
        const int s = j % NS;
        if (!mbar_wait_warp(BAR_FULL(s), (uint32_t)((j / NS) & 1))) { report(3); break; }
        if (j >= 1 && !mbar_wait_warp(BAR_SFREE, (uint32_t)((j - 1) & 1))) { report(4); break; }
        tc_fence_after();
        const uint32_t y_lo = st_k + (uint32_t)s * (C::STAGE >> 4);
        if (elect_one()) {
          issue_scores<D, C::X_IN_T>(tmem + C::T_S, C::X_IN_T ? tmem + C::T_X : x_lo, y_lo);
          if constexpr (HAS_U)
            issue_scores<D, C::U_IN_T>(tmem + C::T_W, C::U_IN_T ? tmem + C::T_U : u_lo, y_lo + (C::COL_TILE >> 4));
          umma_commit(BAR_S);
        }
        __syncwarp();
      }
    }
    __syncwarp();
  } else if (warp == kAccIssuerWarp) {
    // ================= MMA issuer of the accumulating products =================
    if (J > 0) {
      const uint32_t st_mn = desc_mn(sbase + C::OFF_ST, D);   // stage 0, MN-major view
      for (int j = 0; j < J; ++j) {
        const int s = j % NS;
        if (!mbar_wait_warp(BAR_P, (uint32_t)(j & 1))) { report(5); break; }
        tc_fence_after();
        const uint32_t y_mn = st_mn + (uint32_t)s * (C::STAGE >> 4), z_mn = y_mn + (C::COL_TILE >> 4);
        if (elect_one()) {
          issue_acc<D>(tmem + C::T_A1, tmem + C::T_E, HAS_U ? y_mn : z_mn);
          if (rev) issue_acc<D>(tmem + C::T_A2, tmem + C::T_P, z_mn);
          umma_commit(BAR_PV);
          umma_commit(BAR_EMPTY(s));
          if (j + 1 == J) umma_commit(BAR_DONE);
        }
        __syncwarp();
      }
    }
    __syncwarp();
  } else {
    // ================= compute warps =================
    const int cpart = warp >> 2, qd = warp & 3;
    const int row = r0 + qd * 32 + lane;
    const bool row_ok = row < a.nrows;
    const float ck = stat_scale(a.stat_k, rev ? head : head / a.ratio, a.lim);
    const uint64_t A0v = pack2(a.a0, a.a0);
    uint64_t A1v, A2v, A2d;
    auto set_coefficients = [&](int hq) {
      const float c = stat_scale(a.stat_q, hq, a.lim) * ck;
      const float A1 = a.a1 * c, A2 = a.a2 * c * c;
      A1v = pack2(A1, A1);
      A2v = pack2(A2, A2);
      A2d = pack2(2.f * A2, 2.f * A2);
    };
    int hq_now = rev ? head * a.ratio : head;
    set_coefficients(hq_now);
    int limcol = a.ncols - 1, lowcol = 0;                   // columns kept: lowcol <= col <= limcol
    if (a.mask) {
      if (rev) lowcol = row - a.off;
      else limcol = min(limcol, row + a.off);
    }
    const int wrow_lo = r0 + qd * 32, wrow_hi = wrow_lo + 31;
    const float dl_row = MODE == MODE_DQ && row_ok ? __ldg(a.dvec + (size_t)head * a.nrows + row) : 0.f;
    const uint64_t ndl_row = pack2(-dl_row, -dl_row);
    const uint32_t tl = tmem + ((uint32_t)(qd * 32) << 16);
    float* myvec = (float*)(smem + C::OFF_VEC) + warp * 64;
    const uint32_t myvec_s = sbase + C::OFF_VEC + warp * 256;
    // negated dvec of this lane's column in the next tile, fetched one tile ahead
    auto fetch_vec = [&](int j, const ColPos& cp) -> float {
      if (j >= J) return 0.f;
      const int col = cp.t * BN + cpart * 32 + lane;
      return (col < a.ncols) ? -__ldg(a.dvec + (size_t)cp.h * a.ncols + col) : 0.f;
    };
#pragma unroll
    for (int e = 0; e < D / 4; ++e) {
      run1[e] = 0ull;
      if constexpr (rev) run2[e] = 0ull;
    }
    bool ok = true;
    if (C::X_IN_T && J > 0) {
      // copy the row operands to tensor memory: column c of a part holds elements 2c and 2c+1 of the row; the two warps of a
      // lane quarter take alternate parts.  (16-byte pieces, XOR-swizzled by the row's place in its swizzle atom)
      if (!mbar_wait(BAR_X, 0)) { report(6); ok = false; }
      if (ok) {
        const int r = qd * 32 + lane, sw = D == 64 ? (r & 7) : ((r >> 1) & 3);
        for (int it = cpart; it < (C::U_IN_T ? 6 : 3); it += 2) {
          const uint32_t src = sbase + it * C::ROW_SUB + r * (D * 2), dst = tl + C::T_X + it * (D / 2);
          uint32_t w[D / 2];
#pragma unroll
          for (int pc = 0; pc < D / 8; ++pc) {
            const ulonglong2 v = lds_v2(src + ((pc ^ sw) << 4));
            w[4 * pc] = (uint32_t)v.x; w[4 * pc + 1] = (uint32_t)(v.x >> 32);
            w[4 * pc + 2] = (uint32_t)v.y; w[4 * pc + 3] = (uint32_t)(v.y >> 32);
          }
          if constexpr (D == 64) tmem_st32(dst, w);
          else tmem_st16(dst, w);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR_XT);
      }
    }
    uint64_t rs2 = 0ull;
    ColPos pc = pos0;
    float nxt = rev ? fetch_vec(0, pc) : 0.f;
    for (int j = 0; ok && j < J; ++j, advance(pc)) {
      const float cur = nxt;
      if (rev) {
        ColPos pn = pc;
        advance(pn);
        nxt = fetch_vec(j + 1, pn);
        if (pc.h != hq_now) {
          hq_now = pc.h;
          set_coefficients(pc.h);
        }
      }
      if (!mbar_wait(BAR_S, (uint32_t)(j & 1))) { report(7); ok = false; break; }
      tc_fence_after();
      const uint32_t vec_s = myvec_s + (j & 1) * 128;
      if (rev) {
        myvec[(j & 1) * 32 + lane] = cur;
        __syncwarp();
      }
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
      const int c0 = pc.t * BN + cpart * 32;                // first of this warp's 32 columns
      bool need_mask = c0 + 32 > a.ncols;
      if (a.mask) need_mask = need_mask || (rev ? c0 < wrow_hi - a.off : c0 + 31 > wrow_lo + a.off);
      // E (or P of the forward) and P of the tile as three packed parts each
      uint32_t e3[3][16], p3[3][rev ? 16 : 1];
      ulonglong2 nd2 = make_ulonglong2(0ull, 0ull);
      uint64_t ts2 = 0ull;                                  // row sums of this tile
      auto element = [&](int e, bool masked) {
        const uint64_t s2 = pack2u(sv[2 * e], sv[2 * e + 1]);
        bool z0 = false, z1 = false;
        if (masked) {
          const int col = c0 + 2 * e;
          z0 = col > limcol || col < lowcol;
          z1 = col + 1 > limcol || col + 1 < lowcol;
        }
        auto keep = [&](uint64_t v) -> uint64_t {
          if (!masked) return v;
          float v0, v1;
          unpack2(v, v0, v1);
          return pack2(z0 ? 0.f : v0, z1 ? 0.f : v1);
        };
        if constexpr (!HAS_U) {
          const uint64_t pv = keep(fma2(fma2(A2v, s2, A1v), s2, A0v));
          ts2 = add2(ts2, pv);
          split3(pv, e3[0][e], e3[1][e], e3[2][e]);
        } else {
          if (rev && (e & 1) == 0) nd2 = lds_v2(vec_s + (e >> 1) * 16);   // four column values per load
          const uint64_t ndl = rev ? ((e & 1) ? nd2.y : nd2.x) : ndl_row;
          split3(keep(mul2(fma2(A2d, s2, A1v), add2(pack2u(wv[2 * e], wv[2 * e + 1]), ndl))), e3[0][e], e3[1][e], e3[2][e]);
          if constexpr (rev) split3(keep(fma2(fma2(A2v, s2, A1v), s2, A0v)), p3[0][e], p3[1][e], p3[2][e]);
        }
      };
      // the mask test stays outside the element loops so that each is one basic block of independent pairs
      if (!need_mask) {
#pragma unroll
        for (int e = 0; e < 16; ++e) element(e, false);
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) element(e, true);
      }
      if (!HAS_U) rs2 = add2(rs2, ts2);
      // the previous tile's products must be done before their operands are overwritten; their sums are
      // taken over before the arrival below lets this tile's products replace them
      if (j > 0) {
        if (!mbar_wait(BAR_PV, (uint32_t)((j - 1) & 1))) { report(9); ok = false; break; }
        tc_fence_after();
      }
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        tmem_st16(tl + C::T_E + 32 * t + cpart * 16, e3[t]);
        if constexpr (rev) tmem_st16(tl + C::T_P + 32 * t + cpart * 16, p3[t]);
      }
      if (j > 0) {
        promote<D>(run1, tl + C::T_A1, cpart);
        if constexpr (rev) promote<D>(run2, tl + C::T_A2, cpart);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_P);
    }
    if (ok && J > 0) {
      if (!mbar_wait(BAR_DONE, 0)) { report(10); ok = false; }
      else {
        tc_fence_after();
        promote<D>(run1, tl + C::T_A1, cpart);
        if constexpr (rev) promote<D>(run2, tl + C::T_A2, cpart);
      }
    }
    ok_compute = ok;
    if (!HAS_U) {
      float lo, hi;
      unpack2(rs2, lo, hi);
      rows_sum[cpart * BM + qd * 32 + lane] = lo + hi;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kIssuerWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, C::T_COLS);
  }
  // ---- epilogue: each compute thread owns half of the features of one row ----
  if (warp < kComputeWarps && ok_compute) {
    const int cpart = warp >> 2, rl = (warp & 3) * 32 + lane, row = r0 + rl;
    const bool row_ok = row < a.nrows;
    const size_t grow = (size_t)head * a.nrows + (row_ok ? row : 0), at = grow * D + cpart * (D / 2);
    if constexpr (!HAS_U) {
      if (row_ok)
        store_forward<D>(a, run1, grow, cpart, rows_sum[rl] + rows_sum[BM + rl] + (a.den_add ? a.den_add[grow] : 0.f));
    } else {
      float part = 0.f;
      if (row_ok) {
        part = store_half<D>(run1, a.o1 + at, a.o1_add ? a.o1_add + at : nullptr, a.dots ? a.x + at : nullptr, 1.f);
        if constexpr (rev) store_half<D>(run2, a.o2 + at, a.o2_add ? a.o2_add + at : nullptr, nullptr, 1.f);
      }
      if (a.dots) {
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) part += __shfl_xor_sync(0xffffffffu, part, m);
        if (lane == 0) atomicAdd(a.dots + head, part);
      }
    }
  }
}

// ---------------------------------------------------------------------------------------------------------
// Rows of float32 -> rows of [h | m | l] bf16, up to four tensors in one launch (blockIdx.y).  With `den` the
// row is first divided by its denominator and dvec = (that row) . out is written too.  8 elements per thread;
// HBM-bound: reads 4 and writes 6 bytes per element.
struct SplitJob {
  const float* src;
  __nv_bfloat16* dst;
  size_t rows;
  const float* den;
  const float* out;
  float* dvec;
  const stat_t* stat;     // rows are taken times pow2_of the scale of their head, `n` rows each, or null
  int n;
  float lim;
};
struct SplitJobs {
  SplitJob j[4];
  float* zero;      // `zeros` floats set to zero (the per-head dots of the kernels that follow)
  int zeros;
};

template <int D>
__global__ void __launch_bounds__(256) split3_kernel(const SplitJobs jobs) {
  constexpr int TPR = D / 8;                    // threads per row
  const SplitJob& jb = jobs.j[blockIdx.y];
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (int i = threadIdx.x; i < jobs.zeros; i += 256) jobs.zero[i] = 0.f;
  const size_t idx = (size_t)blockIdx.x * 256 + threadIdx.x, row = idx / TPR;
  const int part = (int)(idx % TPR);
  if (row - (size_t)(threadIdx.x & 31) / TPR >= jb.rows) return;      // whole warps leave together
  const bool ok = row < jb.rows;
  // (rows stay below 2^32: their parts take at most 48 GiB)
  const stat_t st = jb.stat && ok ? __ldg((const unsigned long long*)jb.stat + (unsigned)row / (unsigned)jb.n) : 0;
  float f[8];
  if (ok) {
    const float4 u = __ldg((const float4*)(jb.src + row * D + part * 8)), w = __ldg((const float4*)(jb.src + row * D + part * 8) + 1);
    f[0] = u.x; f[1] = u.y; f[2] = u.z; f[3] = u.w; f[4] = w.x; f[5] = w.y; f[6] = w.z; f[7] = w.w;
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] = 0.f;
  }
  if (jb.den) {
    const float inv = ok ? 1.0f / __ldg(jb.den + row) : 0.f;
    float s = 0.f;
    if (ok) {
      const float4 u = __ldg((const float4*)(jb.out + row * D + part * 8)), w = __ldg((const float4*)(jb.out + row * D + part * 8) + 1);
      const float o[8] = {u.x, u.y, u.z, u.w, w.x, w.y, w.z, w.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) s = fmaf(f[e], o[e], s);
    }
#pragma unroll
    for (int m = TPR / 2; m >= 1; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
    if (ok && part == 0) jb.dvec[row] = s * inv;
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= inv;
  }
  if (!ok) return;
  if (jb.stat) {
    const float s = pow2_of(stat_scale(&st, 0, jb.lim));
#pragma unroll
    for (int e = 0; e < 8; ++e) f[e] *= s;
  }
  uint32_t h[4], m[4], l[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) split3(pack2(f[2 * e], f[2 * e + 1]), h[e], m[e], l[e]);
  uint4* dst = (uint4*)(jb.dst + row * 3 * D) + part;
  dst[0] = make_uint4(h[0], h[1], h[2], h[3]);
  dst[TPR] = make_uint4(m[0], m[1], m[2], m[3]);
  dst[2 * TPR] = make_uint4(l[0], l[1], l[2], l[3]);
}

int launch_split3(const Ctx& c, const SplitJobs& jobs, int count) {
  size_t rows = 0;
  for (int i = 0; i < count; ++i) rows = jobs.j[i].rows > rows ? jobs.j[i].rows : rows;
  const size_t per_block = 256 / (c.p.d / 8);
  dim3 grid((unsigned)((rows + per_block - 1) / per_block), count);
  if (c.p.d == 32) FM_LAUNCH("fm_split3", c.stream, (split3_kernel<32><<<grid, 256, 0, c.stream>>>(jobs)));
  else FM_LAUNCH("fm_split3", c.stream, (split3_kernel<64><<<grid, 256, 0, c.stream>>>(jobs)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

template <int D, int MODE>
int launch_tiles(const Ctx& c, const char* name, const void* x, const void* u, const void* y, const void* z, SplitArgs a) {
  using C = SC<D, MODE>;
  const fastmax_problem& p = c.p;
  const int heads = C::rev ? p.bhkv : p.bh, col_heads = C::rev ? p.bh : p.bhkv;
  const int nrows = C::rev ? p.nk : p.nq, ncols = C::rev ? p.nq : p.nk;
  if (heads == 0 || nrows == 0) return FASTMAX_OK;
  CUtensorMap tx, tu, ty, tz;
  int rc;
  if ((rc = split_map<D>(&tx, x, heads, nrows, BM))) return rc;
  if ((rc = split_map<D>(&tu, u, heads, nrows, BM))) return rc;
  if ((rc = split_map<D>(&ty, y, col_heads, ncols, BN))) return rc;
  if ((rc = split_map<D>(&tz, z, col_heads, ncols, BN))) return rc;
  long long blocks;
  if ((rc = set_sizes(p, heads, nrows, ncols, &a, &blocks))) return rc;
  a.order = rows_by_tile(p.mask && a.chunk == 0, a.heads, a.ntr, 1);
  const auto kernel = split_kernel<D, MODE>;
  FM_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
  FM_LAUNCH(name, c.stream, (kernel<<<(unsigned)blocks, kThreads, C::SMEM, c.stream>>>(tx, tu, ty, tz, a)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

size_t up256(size_t x) { return (x + 255) / 256 * 256; }
size_t parts_bytes(const fastmax_problem& p, int heads, int n) { return up256((size_t)6 * heads * n * p.d); }

}  // namespace

// float32, d 32 or 64, as the default of the float32 score family and of the chunks of the float32 moment family (the
// families that name the CUDA cores, FASTMAX_IMPL_DENSE_FFMA and _MOMENTS_FFMA, stay on them).  The parts take one and a
// half times the memory of the tensors they are made of.  Problems whose parts would need more than 48 GiB -- tensors of
// 8 GB each, eight of which autograd and the caller hold -- stay on the CUDA cores, so that what fitted a device without
// a workspace still does.
bool dense_split_supports(const fastmax_problem& p) {
  return (p.impl == FASTMAX_IMPL_AUTO || p.impl == FASTMAX_IMPL_MOMENTS) && p.dtype == FASTMAX_F32 &&
         (p.d == 32 || p.d == 64) && p.bhkv > 0 && p.nq > 0 && p.nk > 0 && dense_split_bwd_bytes(p) <= (size_t)48 << 30;
}

// Workspace: forward [q | k | v], backward [q | k | v | gs | dvec], parts of 3 d bf16 per row.
size_t dense_split_fwd_bytes(const fastmax_problem& p) {
  return parts_bytes(p, p.bh, p.nq) + 2 * parts_bytes(p, p.bhkv, p.nk);
}
size_t dense_split_bwd_bytes(const fastmax_problem& p) {
  return dense_split_fwd_bytes(p) + parts_bytes(p, p.bh, p.nq) + up256(sizeof(float) * (size_t)p.bh * p.nq);
}

int dense_split_forward(const Ctx& c, const void* q, const void* k, const void* v, const stat_t* stats, const FwdOut& o,
                        void* workspace, const ChunkAdd* ca) {
  const fastmax_problem& p = c.p;
  char* ws = (char*)workspace;
  const size_t bq = parts_bytes(p, p.bh, p.nq), bk = parts_bytes(p, p.bhkv, p.nk);
  __nv_bfloat16 *q3 = (__nv_bfloat16*)ws, *k3 = (__nv_bfloat16*)(ws + bq), *v3 = (__nv_bfloat16*)(ws + bq + bk);
  SplitJobs jobs = {};
  jobs.j[0] = {(const float*)q, q3, (size_t)p.bh * p.nq, nullptr, nullptr, nullptr};
  jobs.j[1] = {(const float*)k, k3, (size_t)p.bhkv * p.nk, nullptr, nullptr, nullptr};
  jobs.j[2] = {(const float*)v, v3, (size_t)p.bhkv * p.nk, nullptr, nullptr, nullptr};
  int rc;
  if ((rc = launch_split3(c, jobs, 3))) return rc;
  SplitArgs a = {};
  a.stat_q = p.normalize ? stats : nullptr;
  a.stat_k = p.normalize ? stats + p.bh : nullptr;
  a.o1 = (float*)o.out;
  a.den_out = o.den;
  a.o_stride = o.o_stride;
  a.den_stride = o.den_stride;
  if (ca) { a.chunk = ca->chunk; a.o1_add = ca->out_add; a.den_add = ca->den_add; }
  if (split_rows_serve(p, MODE_FWD, a.chunk)) return split_rows_forward(c, q3, k3, v3, a);
  if (p.d == 32) return launch_tiles<32, MODE_FWD>(c, "fm_dense_split_fwd", q3, q3, k3, v3, a);
  return launch_tiles<64, MODE_FWD>(c, "fm_dense_split_fwd", q3, q3, k3, v3, a);
}

int dense_split_backward(const Ctx& c, const void* q, const void* k, const void* v, const void* out, const float* den,
                         const stat_t* stats, const void* grad_out, float* dots, void* grad_q, void* grad_k,
                         void* grad_v, void* workspace, const ChunkAdd* ca) {
  const fastmax_problem& p = c.p;
  char* ws = (char*)workspace;
  const size_t bq = parts_bytes(p, p.bh, p.nq), bk = parts_bytes(p, p.bhkv, p.nk);
  __nv_bfloat16 *q3 = (__nv_bfloat16*)ws, *k3 = (__nv_bfloat16*)(ws + bq), *v3 = (__nv_bfloat16*)(ws + bq + bk),
                *g3 = (__nv_bfloat16*)(ws + bq + 2 * bk);
  float* dvec = (float*)(ws + 2 * bq + 2 * bk);
  SplitJobs jobs = {};
  jobs.j[0] = {(const float*)q, q3, (size_t)p.bh * p.nq, nullptr, nullptr, nullptr};
  jobs.j[1] = {(const float*)k, k3, (size_t)p.bhkv * p.nk, nullptr, nullptr, nullptr};
  jobs.j[2] = {(const float*)v, v3, (size_t)p.bhkv * p.nk, nullptr, nullptr, nullptr};
  jobs.j[3] = {(const float*)grad_out, g3, (size_t)p.bh * p.nq, den, (const float*)out, dvec};
  if (p.normalize && !ca) {      // with `ca` other kernels have added to the dots already
    jobs.zero = dots;
    jobs.zeros = p.bh + p.bhkv;
  }
  int rc;
  if ((rc = launch_split3(c, jobs, 4))) return rc;
  SplitArgs a = {};
  a.stat_q = p.normalize ? stats : nullptr;
  a.stat_k = p.normalize ? stats + p.bh : nullptr;
  a.dvec = dvec;
  a.chunk = ca ? ca->chunk : 0;
  a.o1 = (float*)grad_q;
  a.o1_add = ca ? ca->gq_add : nullptr;
  a.x = (const float*)q;
  a.dots = p.normalize ? dots : nullptr;
  if (split_rows_serve(p, MODE_DQ, a.chunk)) rc = split_rows_dq(c, q3, g3, k3, v3, a);
  else if (p.d == 32) rc = launch_tiles<32, MODE_DQ>(c, "fm_dense_split_dq", q3, g3, k3, v3, a);
  else rc = launch_tiles<64, MODE_DQ>(c, "fm_dense_split_dq", q3, g3, k3, v3, a);
  if (rc) return rc;
  a.o1 = (float*)grad_k;
  a.o2 = (float*)grad_v;
  a.o1_add = ca ? ca->gk_add : nullptr;
  a.o2_add = ca ? ca->gv_add : nullptr;
  a.x = (const float*)k;
  a.dots = p.normalize ? dots + p.bh : nullptr;
  if (p.d == 32) return launch_tiles<32, MODE_DKDV>(c, "fm_dense_split_dkdv", k3, v3, q3, g3, a);
  return launch_tiles<64, MODE_DKDV>(c, "fm_dense_split_dkdv", k3, v3, q3, g3, a);
}

int split3_scaled_q(const Ctx& c, const void* q, void* q3, const void* v, void* v3, const stat_t* stats) {
  const fastmax_problem& p = c.p;
  SplitJobs jobs = {};
  jobs.j[0] = {(const float*)q, (__nv_bfloat16*)q3, (size_t)p.bh * p.nq, nullptr, nullptr, nullptr, stats, p.nq, p.lim};
  jobs.j[1] = {(const float*)v, (__nv_bfloat16*)v3, (size_t)p.bhkv * p.nk, nullptr, nullptr, nullptr};
  return launch_split3(c, jobs, 2);
}

int split_status(int* out, cudaStream_t stream) {
  FM_CUDA_TRY(cudaMemcpyFromSymbolAsync(out, g_split_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
int split_status_reset(cudaStream_t stream) {
  const int zero = 0;
  FM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_split_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}

}  // namespace fm
