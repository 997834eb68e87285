// Score form on the tcgen05 tensor cores for SHORT rows (bf16, d = 64): the same sums as fm_dense_tc_wide.cu for
// problems, or chunks of the moment family, whose rows see a few hundred columns.
//
// A row tile of fm_dense_tc_wide.cu takes a whole SM (640 threads, all 512 TMEM columns) and spends several
// microseconds outside its column loop -- barriers, TMEM, the first tiles from HBM, the fp32 rows the epilogue adds,
// the stores -- which two compute groups and two score buffers cannot hide when the loop itself runs two to eight
// times.  Here a CTA needs half an SM (352 threads at 80 registers, 256 TMEM columns, at most 82 KB of shared memory),
// so two row tiles run on each SM and one's loop covers the other's ends; inside a CTA there is a single score buffer.
//
// Warps 0-7 compute (warp % 4 = TMEM lane quarter = 32 rows, warp / 4 = half of the 64 columns of a tile, taken 16 at
// a time), warp 8 loads tiles by TMA, warp 9 issues S = X Y^T and W = U Z^T, warp 10 the accumulating products.
// TMEM columns:  FWD  S 64 | P 32 | out 64        DQ  S 64 | W 64 | E 32 | grad_q 64
//                DKDV S 64 | W 64 | grad_k 64 | grad_v 64, with E over S and P over W: the 16 columns a warp has just
//                read hold its 8 packed columns, so the next tile's scores wait for this tile's products
// All waits are bounded.
//
// FIRST: the first-order moment family's chunks.  What a token takes from everything before its chunk (or, DKDV, after
// it) is one more product per row tile with the d x d state S1 -- FWD x S1, DQ gs S1^T, DKDV v S1^T and k S1 -- so it
// goes into the same accumulators before the chunk's own products, from a bf16 copy of S1 already scaled by the
// first-order coefficient; the state's vectors (constant row, normaliser column) are added in the epilogue.  No fp32
// rows travel between a read-out kernel and this one.
#include "fm_common.cuh"
#include "fm_sm100.cuh"

namespace fm {

__device__ int g_short_status = 0;

namespace {
using namespace sm100;

enum { MODE_FWD = 0, MODE_DQ = 1, MODE_DKDV = 2 };

struct ShortArgs {
  void* o1;              // out, grad_q or grad_k
  void* o2;              // grad_v
  float* den_out;
  const float* o1_add;   // fp32 rows added before the division / rounding (may be null)
  const float* o2_add;
  const float* den_add;
  const void* x;         // row operand in global memory (normalisation dot)
  const float* dvec;
  float* dots;
  const stat_t* stat_q;
  const stat_t* stat_k;
  int nrows, ncols, off, mask, ntr, chunk, ratio, o_heads, by_tile;
  float a0, a1, a2, lim;
  // FIRST: running sums of the states, rows [y_a | 1] of `dvp` floats, d + 1 rows per (head, chunk)
  const float* st;
  int dvp, nchunk, zero_chunk;    // zero_chunk: the chunk whose running sum is empty (-1: none)
};

constexpr int BM = 128, BN = 64, D = 64;
constexpr int kThreads = 352, kComputeWarps = 8, kProducerWarp = 8, kIssuerWarp = 9, kAccIssuerWarp = 10;
constexpr int ROW_TILE = BM * 128, COL_TILE = BN * 128, STAGE = 2 * COL_TILE;

template <int MODE, bool FIRST>
struct SH {
  static constexpr int NS = 3;
  static constexpr int OFF_U = ROW_TILE, OFF_ST = (MODE == MODE_FWD ? 1 : 2) * ROW_TILE;
  static constexpr int OFF_S1 = OFF_ST + NS * STAGE;       // FIRST: the chunk's 64 x 64 state copy
  static constexpr int OFF_STV = OFF_S1 + (FIRST ? 8192 : 0);   // FIRST: normaliser column 64, constant row 65 (+ 3)
  static constexpr int OFF_VEC = OFF_STV + (FIRST ? 132 * 4 : 0);   // per compute warp 2 x 32 floats; row sums (FWD)
  static constexpr int OFF_BAR = OFF_VEC + kComputeWarps * 2 * 32 * 4;
  static constexpr int NBAR = 2 + 2 * NS + 4;
  static constexpr int OFF_TMEM = OFF_BAR + NBAR * 8;
  static constexpr int SMEM = OFF_TMEM + 16 + 1024;
  static constexpr int T_S = 0, T_W = 64;
  static constexpr bool INPLACE = MODE == MODE_DKDV;
  static constexpr int T_E = MODE == MODE_FWD ? 64 : (MODE == MODE_DQ ? 128 : T_S), T_P = T_W;
  static constexpr int T_A1 = MODE == MODE_FWD ? 96 : (MODE == MODE_DQ ? 160 : 128), T_A2 = 192;
  static constexpr int T_COLS = 256;
};

__device__ __forceinline__ void report(int code) { atomicCAS(&g_short_status, 0, code); }

// acc (+)= (128 x 64 operand in TMEM, `step` columns per 16 keys) x (column tile, MN-major)
__device__ __forceinline__ void issue_acc(uint32_t acc, uint32_t a_tmem, int step, uint32_t b_mn, uint32_t accumulate) {
  constexpr uint32_t idesc = idesc_bf16(BM, D, 0, 1);
#pragma unroll
  for (int ks = 0; ks < BN / 16; ++ks) umma_ts_1(acc, a_tmem + ks * step, b_mn + ks * 128, idesc, ks > 0 ? 1u : accumulate);
}

// One thread's row segment: (accumulator + mul * vec) * scale -> bf16, vec NC floats of shared memory; returns its
// dot product with the x row when wanted (store_row of fm_sm100.cuh with a vector in place of fp32 rows).
template <int NC>
__device__ __forceinline__ float store_row_vec(uint32_t taddr, bool row_ok, __nv_bfloat16* dst, uint32_t vec_s, float mul,
                                               const __nv_bfloat16* xr, float scale) {
  float part = 0.f;
  const bool wide = (((uintptr_t)dst | (uintptr_t)xr) & 31) == 0;
  uint32_t xw[NC / 16][8];                 // asked for together
  if (xr && row_ok) {
#pragma unroll
    for (int i = 0; i < NC / 16; ++i) ldg32(xr + 16 * i, xw[i], wide);
  }
#pragma unroll
  for (int c0 = 0; c0 < NC; c0 += 16) {
    uint32_t ov[16];
    tmem_ld16(taddr + c0, ov);
    tmem_wait_ld(ov);
    if (row_ok) {
      float f[16];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const ulonglong2 v = lds_v2(vec_s + (c0 + 4 * e) * 4);
        float w[4];
        unpack2(v.x, w[0], w[1]);
        unpack2(v.y, w[2], w[3]);
#pragma unroll
        for (int i = 0; i < 4; ++i) f[4 * e + i] = fmaf(mul, w[i], __uint_as_float(ov[4 * e + i])) * scale;
      }
      uint32_t w[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) w[e] = pack_bf16(f[2 * e], f[2 * e + 1]);
      stg32(dst + c0, w, wide);
      if (xr) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          part = fmaf(f[2 * e], __uint_as_float(xw[c0 / 16][e] << 16), part);
          part = fmaf(f[2 * e + 1], __uint_as_float(xw[c0 / 16][e] & 0xFFFF0000u), part);
        }
      }
    }
  }
  return part;
}

template <int MODE, bool FIRST>
__global__ void __launch_bounds__(kThreads, 2)
short_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmU,
             const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmZ,
             const __grid_constant__ CUtensorMap tmS, const ShortArgs a) {
  using C = SH<MODE, FIRST>;
  constexpr int NS = C::NS;
  constexpr bool rev = MODE == MODE_DKDV, FWD = MODE == MODE_FWD, HAS_U = !FWD;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + C::OFF_BAR;
  // barrier map: x | done | full[NS] | empty[NS] | s_full | s_free | p_full | pv_done
  const uint32_t BAR_X = bar0, BAR_DONE = bar0 + 8;
  auto BAR_FULL = [&](int s) { return bar0 + 8u * (2 + s); };
  auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (2 + NS + s); };
  const uint32_t BAR_S = bar0 + 8u * (2 + 2 * NS), BAR_SFREE = BAR_S + 8, BAR_P = BAR_S + 16, BAR_PV = BAR_S + 24;
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + C::OFF_TMEM);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // longest rows first (row_tile_of)
  int head, pidx;
  row_tile_of(blockIdx.x, a.by_tile, a.ntr, head, pidx);
  const int r0 = (rev ? pidx : a.ntr - 1 - pidx) * BM;
  const int ntile = (a.ncols + BN - 1) / BN;
  int tb = 0, te = ntile;
  if (a.mask) {
    if (rev) tb = max(0, r0 - a.off) / BN;
    else te = min(ntile, (min(r0 + BM - 1, a.nrows - 1) + a.off) / BN + 1);
  }
  if (a.chunk > 0) {  // the row tile lies in one chunk (chunk % 256 == 0)
    const int cbeg = (r0 / a.chunk) * (a.chunk / BN), cend = cbeg + a.chunk / BN;
    if (rev) te = min(te, cend);
    else tb = cbeg;
  }
  // grouped heads: a key/value head (DKDV rows) walks its tile range once per query head of the group
  const int Jh = max(te - tb, 0), J = rev ? Jh * a.ratio : Jh;
  struct ColPos { int t, h; };
  const ColPos pos0 = {tb, rev ? head * a.ratio : head / a.ratio};
  auto advance = [&](ColPos& cp) {
    if (++cp.t >= tb + Jh && rev) { cp.t = tb; ++cp.h; }
  };

  const int chunk = FIRST ? r0 / a.chunk : 0;
  const bool has_state = FIRST && chunk != a.zero_chunk;
  if (tid == 0) {
    mbar_init(BAR_X, 1);
    mbar_init(BAR_DONE, 1);
    for (int s = 0; s < NS; ++s) { mbar_init(BAR_FULL(s), 1); mbar_init(BAR_EMPTY(s), 1); }
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
  float* const rows_sum = (float*)(smem + C::OFF_VEC);

  if (warp == kProducerWarp) {
    // ================= TMA producer =================
    if (lane == 0 && J > 0) {
      mbar_expect_tx(BAR_X, (HAS_U ? 2 : 1) * ROW_TILE + (has_state ? 8192 : 0));
      tma_load_3d(sbase, &tmX, BAR_X, 0, r0, head);
      if (HAS_U) tma_load_3d(sbase + C::OFF_U, &tmU, BAR_X, 0, r0, head);
      if (has_state) tma_load_3d(sbase + C::OFF_S1, &tmS, BAR_X, 0, 0, head * a.nchunk + chunk);
    }
    ColPos pc = pos0;
    for (int j = 0; j < J; ++j, advance(pc)) {
      const int s = j % NS;
      if (!mbar_wait(BAR_EMPTY(s), (uint32_t)(((j / NS) & 1) ^ 1))) { report(71); break; }
      if (lane == 0) {
        mbar_expect_tx(BAR_FULL(s), STAGE);
        const uint32_t dst = sbase + C::OFF_ST + s * STAGE;
        tma_load_3d(dst, &tmY, BAR_FULL(s), 0, pc.t * BN, pc.h);
        tma_load_3d(dst + COL_TILE, &tmZ, BAR_FULL(s), 0, pc.t * BN, pc.h);
      }
    }
  } else if (warp == kIssuerWarp) {
    // ================= issuer of the S / W products (whole warp, one elected lane issues) ============
    if (J > 0) {
      constexpr uint32_t idescS = idesc_bf16(BM, BN, 0, 0);
      const uint32_t x_lo = desc_lo(sbase, 16), u_lo = desc_lo(sbase + C::OFF_U, 16);
      const uint32_t st_k = desc_lo(sbase + C::OFF_ST, 16);   // stage 0, K-major view
      bool ok = mbar_wait_warp(BAR_X, 0);
      if (!ok) report(72);
      for (int j = 0; ok && j < J; ++j) {
        const int s = j % NS;
        if (!mbar_wait_warp(BAR_FULL(s), (uint32_t)((j / NS) & 1))) { report(73); break; }
        // the score region is free once it is in registers, or (INPLACE) once the products that read it are done
        if (j >= 1 && !mbar_wait_warp(C::INPLACE ? BAR_PV : BAR_SFREE, (uint32_t)((j - 1) & 1))) { report(74); break; }
        tc_fence_after();
        const uint32_t y_lo = st_k + (uint32_t)s * (STAGE >> 4);
        if (elect_one()) {
          umma_ss_k64(tmem + C::T_S, x_lo, y_lo, idescS);
          if (HAS_U) umma_ss_k64(tmem + C::T_W, u_lo, y_lo + (COL_TILE >> 4), idescS);
          umma_commit(BAR_S);
        }
        __syncwarp();
      }
    }
    __syncwarp();
  } else if (warp == kAccIssuerWarp) {
    // ================= issuer of the accumulating products =================
    if (J > 0) {
      const uint32_t st_mn = desc_lo(sbase + C::OFF_ST, COL_TILE);   // stage 0, MN-major view
      bool ok = true;
      if (has_state) {
        ok = mbar_wait_warp(BAR_X, 0);
        if (!ok) report(76);
        tc_fence_after();
        const uint32_t x_lo = desc_lo(sbase, 16), u_lo = desc_lo(sbase + C::OFF_U, 16);
        const uint32_t s_k = desc_lo(sbase + C::OFF_S1, 16), s_mn = desc_lo(sbase + C::OFF_S1, 8192);
        if (ok && elect_one()) {
          if (!FWD) umma_ss_k64(tmem + C::T_A1, u_lo, s_k, idesc_bf16(BM, D, 0, 0));
          if (FWD || rev) umma_ss_kmn_steps<4>(tmem + (FWD ? C::T_A1 : C::T_A2), x_lo, s_mn, idesc_bf16(BM, D, 0, 1), 0u);
        }
        __syncwarp();
      }
      for (int j = 0; ok && j < J; ++j) {
        const int s = j % NS;
        if (!mbar_wait_warp(BAR_P, (uint32_t)(j & 1))) { report(75); break; }
        tc_fence_after();
        const uint32_t y_mn = st_mn + (uint32_t)s * (STAGE >> 4), z_mn = y_mn + (COL_TILE >> 4);
        if (elect_one()) {
          issue_acc(tmem + C::T_A1, tmem + C::T_E, C::INPLACE ? 16 : 8, FWD ? z_mn : y_mn, j > 0 || has_state ? 1u : 0u);
          if (rev) issue_acc(tmem + C::T_A2, tmem + C::T_P, 16, z_mn, j > 0 || has_state ? 1u : 0u);
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
    float dl_row = 0.f;
    if (MODE == MODE_DQ && row_ok) dl_row = __ldg(a.dvec + (size_t)head * a.nrows + row);
    const uint64_t ndl_row = pack2(-dl_row, -dl_row);
    const uint32_t tl = tmem + ((uint32_t)(qd * 32) << 16);
    float* myvec = (float*)(smem + C::OFF_VEC) + warp * 64;
    const uint32_t myvec_s = sbase + C::OFF_VEC + warp * 256;
    auto fetch_vec = [&](int j, const ColPos& cp) -> float {   // negated dvec of this lane's column, one tile ahead
      if (j >= J) return 0.f;
      const int col = cp.t * BN + cpart * 32 + lane;
      return (col < a.ncols) ? -__ldg(a.dvec + (size_t)cp.h * a.ncols + col) : 0.f;
    };
    float* const stv = (float*)(smem + C::OFF_STV);
    if (FIRST) {    // read after the barrier in the epilogue
      const float* st = a.st + (size_t)(head * a.nchunk + chunk) * (D + 1) * a.dvp;
      for (int i = tid; i < 129; i += 256)
        stv[i] = !has_state ? 0.f : (i < 64 ? __ldg(st + (size_t)i * a.dvp + D) : __ldg(st + (size_t)D * a.dvp + (i - 64)));
    }
    uint64_t rs2 = 0ull;
    ColPos pc = pos0;
    float nxt = rev ? fetch_vec(0, pc) : 0.f;
    bool ok = true;
    for (int j = 0; j < J; ++j, advance(pc)) {
      const float cur = nxt;
      if (rev) {
        ColPos pn = pc;
        advance(pn);
        nxt = fetch_vec(j + 1, pn);
        if (pc.h != hq_now) {
          hq_now = pc.h;
          set_coefficients(pc.h);
        }
        myvec[(j & 1) * 32 + lane] = cur;
        __syncwarp();
      }
      const uint32_t vec_s = myvec_s + (j & 1) * 128;
      if (!mbar_wait(BAR_S, (uint32_t)(j & 1))) { report(77); ok = false; break; }
      tc_fence_after();
#pragma unroll
      for (int ps = 0; ps < 2; ++ps) {
        uint32_t sv[16], wv[HAS_U ? 16 : 1];
        tmem_ld16(tl + C::T_S + cpart * 32 + ps * 16, sv);
        if constexpr (HAS_U) {
          tmem_ld16(tl + C::T_W + cpart * 32 + ps * 16, wv);
          tmem_wait_ld(sv, wv);
        } else {
          tmem_wait_ld(sv);
        }
        if (!C::INPLACE && ps == 1) {   // S and W of this tile are in registers: the next tile's may be issued
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(BAR_SFREE);
        }
        const int c0 = pc.t * BN + cpart * 32 + ps * 16;      // first of these 16 columns
        bool need_mask = (c0 + 16 > a.ncols);
        if (a.mask) need_mask = need_mask || (rev ? (c0 < wrow_hi - a.off) : (c0 + 15 > wrow_lo + a.off));
        uint32_t pe[8], pp[rev ? 8 : 1];
        ulonglong2 nd2 = make_ulonglong2(0ull, 0ull);
        auto element = [&](int e, bool masked) {
          const uint64_t s2 = pack2u(sv[2 * e], sv[2 * e + 1]);
          bool z0 = false, z1 = false;
          if (masked) {
            const int col = c0 + 2 * e;
            z0 = col > limcol || col < lowcol;
            z1 = col + 1 > limcol || col + 1 < lowcol;
          }
          auto round2 = [&](uint64_t v) -> uint32_t {
            float v0, v1;
            unpack2(v, v0, v1);
            return pack_bf16(z0 ? 0.f : v0, z1 ? 0.f : v1);
          };
          if constexpr (FWD) {
            const uint64_t pv = fma2(fma2(A2v, s2, A1v), s2, A0v);
            pe[e] = round2(pv);
            // a row with few columns sums what the tensor core will multiply (the rounded values): its rounding
            // then cancels between numerator and denominator; full tiles keep the fp32 sum
            rs2 = add2(rs2, masked ? pack2u(pe[e] << 16, pe[e] & 0xFFFF0000u) : pv);
          } else {
            if (rev && (e & 1) == 0) nd2 = lds_v2(vec_s + ps * 64 + (e >> 1) * 16);   // four column values per load
            const uint64_t ndl = rev ? ((e & 1) ? nd2.y : nd2.x) : ndl_row;
            pe[e] = round2(mul2(fma2(A2d, s2, A1v), add2(pack2u(wv[2 * e], wv[2 * e + 1]), ndl)));
            if constexpr (rev) pp[e] = round2(fma2(fma2(A2v, s2, A1v), s2, A0v));
          }
        };
        if (!need_mask) {
#pragma unroll
          for (int e = 0; e < 8; ++e) element(e, false);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) element(e, true);
        }
        if (C::INPLACE) {
          tmem_st8(tl + C::T_E + cpart * 32 + ps * 16, pe);
          if constexpr (rev) tmem_st8(tl + C::T_P + cpart * 32 + ps * 16, pp);
        } else {
          // the previous tile's products must have consumed E (P) before it is overwritten
          if (ps == 0 && j > 0) {
            if (!mbar_wait(BAR_PV, (uint32_t)((j - 1) & 1))) { report(79); ok = false; break; }
            tc_fence_after();
          }
          tmem_st8(tl + C::T_E + cpart * 16 + ps * 8, pe);
        }
      }
      if (!ok) break;
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_P);
    }
    if (ok && J > 0) {
      if (!mbar_wait(BAR_DONE, 0)) { report(80); ok = false; }
    }
    tc_fence_after();
    // ---- epilogue: FWD and DQ 32 of the 64 columns per warp; DKDV grad_k by warps 0-3, grad_v by warps 4-7 ----
    float scale = 1.f, rowsum = 0.f;
    const uint32_t stv_s = sbase + C::OFF_STV;
    float A1 = 0.f;
    if (FIRST) {
      float unused;
      unpack2(A1v, A1, unused);
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    if (FWD) {
      float lo, hi;
      unpack2(rs2, lo, hi);
      lo += hi;
      if (FIRST && has_state && ok && J > 0) {
        // the state's share of the row sum: x . (normaliser column), half of the row per warp, read from its tile
        if (!mbar_wait(BAR_X, 0)) report(78);
        const int r = qd * 32 + lane;
        float dot = 0.f;
#pragma unroll
        for (int pc = 0; pc < 4; ++pc) {
          const ulonglong2 xv = lds_v2(sbase + r * 128 + (((cpart * 4 + pc) ^ (r & 7)) << 4));
          const uint32_t xw[4] = {(uint32_t)xv.x, (uint32_t)(xv.x >> 32), (uint32_t)xv.y, (uint32_t)(xv.y >> 32)};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float* nc = stv + cpart * 32 + 8 * pc + 2 * e;
            dot = fmaf(__uint_as_float(xw[e] << 16), nc[0], dot);
            dot = fmaf(__uint_as_float(xw[e] & 0xFFFF0000u), nc[1], dot);
          }
        }
        lo += A1 * dot + (cpart == 0 ? a.a0 * stv[128] : 0.f);
      }
      rows_sum[cpart * BM + qd * 32 + lane] = lo;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      rowsum = rows_sum[qd * 32 + lane] + rows_sum[BM + qd * 32 + lane];
      if (a.den_add && row_ok) rowsum += a.den_add[(size_t)head * a.nrows + row];
      scale = 1.0f / rowsum;
    }
    if (ok && J > 0) {
      const size_t grow = (size_t)head * a.nrows + (row_ok ? row : 0);
      float part = 0.f;
      const bool dots_here = !FWD && a.dots != nullptr && !(rev && cpart == 1);
      if constexpr (FIRST && rev) {
        const bool second = cpart == 1;
        part = store_row_vec<64>(tl + (second ? C::T_A2 : C::T_A1), row_ok,
                                 (__nv_bfloat16*)(second ? a.o2 : a.o1) + grow * D, second ? stv_s + 256 : stv_s,
                                 second ? a.a0 : A1, dots_here ? (const __nv_bfloat16*)a.x + grow * D : nullptr, 1.f);
      } else if constexpr (FIRST) {
        const int cc = cpart * 32;
        const size_t orow = FWD ? out_row(head, row_ok ? row : 0, a.nrows, a.o_heads) : grow;
        part = store_row_vec<32>(tl + C::T_A1 + cc, row_ok, (__nv_bfloat16*)a.o1 + orow * D + cc,
                                 stv_s + (FWD ? 256 : 0) + cc * 4, FWD ? a.a0 : -A1 * dl_row,
                                 dots_here ? (const __nv_bfloat16*)a.x + grow * D + cc : nullptr, scale);
        if (FWD && cpart == 0 && row_ok) a.den_out[grow] = rowsum;
      } else if constexpr (rev) {
        const bool second = cpart == 1;
        const float* add = second ? a.o2_add : a.o1_add;
        part = store_row<64, 16>(tl + (second ? C::T_A2 : C::T_A1), row_ok, (__nv_bfloat16*)(second ? a.o2 : a.o1) + grow * D,
                             add ? add + grow * D : nullptr, dots_here ? (const __nv_bfloat16*)a.x + grow * D : nullptr, 1.f);
      } else {
        const int cc = cpart * 32;
        const size_t orow = FWD ? out_row(head, row_ok ? row : 0, a.nrows, a.o_heads) : grow;
        part = store_row<32, 16>(tl + C::T_A1 + cc, row_ok, (__nv_bfloat16*)a.o1 + orow * D + cc,
                             a.o1_add ? a.o1_add + grow * D + cc : nullptr,
                             dots_here ? (const __nv_bfloat16*)a.x + grow * D + cc : nullptr, scale);
        if (FWD && cpart == 0 && row_ok) a.den_out[grow] = rowsum;
      }
      if (dots_here) {
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) part += __shfl_xor_sync(0xffffffffu, part, m);
        if (lane == 0) atomicAdd(a.dots + head, part);
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

// Whether the forward, whose registers and shared memory leave room for a third CTA on an SM, is to run with two.  The third
// one waits for the tensor memory of a CTA of its own SM, so its start is covered, but it is bound to that SM, which evens
// out over many row tiles only.  us, two / three: 322 row tiles of 800 causal columns 13.4 / 15.4, 357 14.9 / 16.6, 600 of 3000 8 %
// slower, 720 1 % faster, 2048 of 450 52.4 / 49.4; causal rows of 300 columns and unmasked ones of 300 5 %
// faster at 300 to 600.
constexpr int kTwoFit = 80 * 1024;
bool two_ctas(long long tiles, int ncols, const ShortArgs& a) {
  const int seen = a.chunk > 0 ? a.chunk / 2 : (a.mask ? ncols / 2 : ncols);
  return tiles <= 666 && seen > (a.mask ? 160 : 320);
}

template <int MODE>
int launch(const Ctx& c, const char* name, const void* x, const void* u, const void* y, const void* z, int nrows,
           int ncols, ShortArgs a, const FirstState* fs = nullptr) {
  constexpr bool rev = MODE == MODE_DKDV;
  const fastmax_problem& p = c.p;
  const int heads = rev ? p.bhkv : p.bh, col_heads = rev ? p.bh : p.bhkv;
  if (heads == 0 || nrows == 0) return FASTMAX_OK;
  // the first-order chunks come here without passing dense_tc_forward / _backward, which check this for the others:
  // TMA reads the operands, rows are stored and read back 16 bytes at a time
  const uintptr_t bases = (uintptr_t)x | (uintptr_t)u | (uintptr_t)y | (uintptr_t)z | (uintptr_t)a.o1 | (uintptr_t)a.o2;
  if (bases & 15) return fail(FASTMAX_E_ARG, "the tensor-core family needs 16-byte aligned tensors");
  CUtensorMap tx, tu, ty, tz, ts;
  int rc;
  if ((rc = tma_map_bf16(&tx, x, heads, nrows, D, BM))) return rc;
  if ((rc = tma_map_bf16(&tu, u ? u : x, heads, nrows, D, BM))) return rc;
  if ((rc = tma_map_bf16(&ty, y, col_heads, ncols, D, BN))) return rc;
  if ((rc = tma_map_bf16(&tz, z, col_heads, ncols, D, BN))) return rc;
  a.x = x;
  a.nrows = nrows;
  a.ncols = ncols;
  a.ntr = (nrows + BM - 1) / BM;
  a.by_tile = rows_by_tile(p.mask && a.chunk == 0, heads, a.ntr, 2);
  a.ratio = p.bh / p.bhkv;
  a.off = p.nk - p.nq;
  a.mask = p.mask;
  a.a0 = p.a0;
  a.a1 = p.a1;
  a.a2 = (p.p == 2) ? p.a2 : 0.f;
  a.lim = p.lim;
  dim3 grid((unsigned)((size_t)heads * a.ntr));
  if (fs) {
    a.nchunk = (nrows + a.chunk - 1) / a.chunk;
    a.st = fs->states;
    a.dvp = moment_dims(D, 1).dvp;
    a.zero_chunk = fs->zero_chunk;
    if ((rc = tma_map_bf16(&ts, fs->s1b, (size_t)heads * a.nchunk, D, D, D))) return rc;
    using C = SH<MODE, true>;
    FM_CUDA_TRY(cudaFuncSetAttribute(short_kernel<MODE, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    FM_LAUNCH(name, c.stream, (short_kernel<MODE, true><<<grid, kThreads, C::SMEM, c.stream>>>(tx, tu, ty, tz, ts, a)));
  } else {
    using C = SH<MODE, false>;
    // (the limit is the same for all calls: another thread may be between these two lines)
    constexpr int most = MODE == MODE_FWD && C::SMEM < kTwoFit ? kTwoFit : C::SMEM;
    const int smem = MODE == MODE_FWD && two_ctas(grid.x, ncols, a) ? most : C::SMEM;
    FM_CUDA_TRY(cudaFuncSetAttribute(short_kernel<MODE, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    FM_LAUNCH(name, c.stream, (short_kernel<MODE, false><<<grid, kThreads, smem, c.stream>>>(tx, tu, ty, tz, tx, a)));
  }
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

}  // namespace

int dense_tc_short_forward(const Ctx& c, const void* q, const void* k, const void* v, const stat_t* stats, void* out,
                           float* den, const ChunkAdd* ca, const FirstState* fs) {
  const fastmax_problem& p = c.p;
  ShortArgs a = {};
  a.stat_q = p.normalize ? stats : nullptr;
  a.stat_k = p.normalize ? stats + p.bh : nullptr;
  a.o1 = out;
  a.den_out = den;
  a.o_heads = c.out_heads;
  if (ca) { a.chunk = ca->chunk; a.o1_add = ca->out_add; a.den_add = ca->den_add; }
  return launch<MODE_FWD>(c, "fm_dense_tc_fwd", q, nullptr, k, v, p.nq, p.nk, a, fs);
}

static ShortArgs backward_args(const fastmax_problem& p, const float* dvec, const stat_t* stats, const ChunkAdd* ca) {
  ShortArgs a = {};
  a.stat_q = p.normalize ? stats : nullptr;
  a.stat_k = p.normalize ? stats + p.bh : nullptr;
  a.dvec = dvec;
  a.chunk = ca ? ca->chunk : 0;
  return a;
}

int dense_tc_short_dq(const Ctx& c, const void* q, const void* k, const void* v, const void* gs, const float* dvec,
                      const stat_t* stats, float* dots, void* grad_q, const ChunkAdd* ca, const FirstState* fs) {
  ShortArgs a = backward_args(c.p, dvec, stats, ca);
  a.o1 = grad_q;
  a.dots = c.p.normalize ? dots : nullptr;
  a.o1_add = ca ? ca->gq_add : nullptr;
  return launch<MODE_DQ>(c, "fm_dense_tc_dq", q, gs, k, v, c.p.nq, c.p.nk, a, fs);
}

int dense_tc_short_dkdv(const Ctx& c, const void* q, const void* k, const void* v, const void* gs, const float* dvec,
                        const stat_t* stats, float* dots, void* grad_k, void* grad_v, const ChunkAdd* ca, const FirstState* fs) {
  ShortArgs a = backward_args(c.p, dvec, stats, ca);
  a.o1 = grad_k;
  a.o2 = grad_v;
  a.dots = c.p.normalize ? dots + c.p.bh : nullptr;
  a.o1_add = ca ? ca->gk_add : nullptr;
  a.o2_add = ca ? ca->gv_add : nullptr;
  return launch<MODE_DKDV>(c, "fm_dense_tc_dkdv", k, v, q, gs, c.p.nk, c.p.nq, a, fs);
}

int tc_short_status(int* out, cudaStream_t stream) {
  FM_CUDA_TRY(cudaMemcpyFromSymbolAsync(out, g_short_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
int tc_short_status_reset(cudaStream_t stream) {
  const int zero = 0;
  FM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_short_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}

}  // namespace fm
