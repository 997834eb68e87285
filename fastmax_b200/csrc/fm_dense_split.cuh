// What the float32 score kernels on the tensor cores share (fm_dense_split.cu, fm_dense_split_rows.cu).
#pragma once

#include "fm_row_walk.cuh"
#include "fm_sm100.cuh"

namespace fm {
// Tensor map like tma_map_bf16 with boxes of 32 elements and 64-byte swizzle (fm_dense_tc.cu)
int tma_map_bf16_half(CUtensorMap* m, const void* base, size_t mats, size_t rows, int d, int box_rows);

namespace split {

enum { MODE_FWD = 0, MODE_DQ = 1, MODE_DKDV = 2 };

struct SplitArgs {
  float* o1;              // out, grad_q or grad_k
  float* o2;              // grad_v (DKDV)
  float* den_out;         // FWD
  const float* o1_add;    // fp32 rows added before the result is divided / stored (may be null)
  const float* o2_add;
  const float* den_add;   // FWD
  const float* x;         // row operand as given (normalisation dot)
  const float* dvec;      // (query heads, nq)
  float* dots;            // per row head: sum of o1 . x, or null
  const stat_t* stat_q;
  const stat_t* stat_k;
  int heads, nrows, ncols, off, mask, ntr, chunk, ratio;   // heads: row heads
  int order;              // row walks: see RowWalk; a CTA per row tile: see rows_by_tile
  int o_stride, den_stride;   // FWD: floats per row of out and den (the packed layout interleaves them)
  float a0, a1, a2, lim;
};

constexpr int BM = 128, BN = 64, kComputeWarps = 8;

using Rows = RowWalk<SplitArgs, BN, false>;   // of the forward's and grad_q's walks

// ---- operands and products ----
// A tile's part p (0 h, 1 m, 2 l) lies at p * SUB: rows of D bf16, 128 or 64 bytes, swizzled over their whole length.
// High descriptor word: groups of eight rows, version 1, swizzle code.
template <int D>
__device__ __forceinline__ constexpr uint32_t desc_hi() {
  return (uint32_t)(D * 16 >> 4) | (1u << 14) | ((D == 64 ? 2u : 4u) << 29);
}
// One K = 16 step of D[tmem] (+)= A B, A in shared or in tensor memory.
template <int D>
__device__ __forceinline__ void mma_ss(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .b64 da, db;\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %5, 0;\n"
      "mov.b64 da, {%1, %3};\n"
      "mov.b64 db, {%2, %3};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n"
      "}\n" ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(desc_hi<D>()), "r"(idesc), "r"(accumulate)
      : "memory");
}
template <int D>
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .b64 db;\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %5, 0;\n"
      "mov.b64 db, {%2, %3};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n"
      "}\n" ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(desc_hi<D>()), "r"(idesc), "r"(accumulate)
      : "memory");
}

// 128 x 64 scores of a row tile against a column tile: the six part products, small terms first.  The row operand lies in
// tensor memory (TS; D / 2 columns a part) or in shared memory: a K step then also reads it from there, 49 instead of 32
// cycles.
template <int D, bool TS>
__device__ __forceinline__ void issue_scores(uint32_t d_tmem, uint32_t a, uint32_t b_lo) {
  constexpr uint32_t idesc = sm100::idesc_bf16(BM, BN, 0, 0), row_sub = BM * D * 2 >> 4, col_sub = BN * D * 2 >> 4;
  constexpr int PA[6] = {1, 0, 2, 0, 1, 0}, PB[6] = {1, 2, 0, 1, 0, 0};
#pragma unroll
  for (int t = 0; t < 6; ++t)
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
      const uint32_t b = b_lo + PB[t] * col_sub + 2 * ks, acc = (t | ks) ? 1u : 0u;
      if constexpr (TS) mma_ts<D>(d_tmem, a + PA[t] * (D / 2) + 8 * ks, b, idesc, acc);
      else mma_ss<D>(d_tmem, a + PA[t] * row_sub + 2 * ks, b, idesc, acc);
    }
}

// acc = (parts of a 128 x 64 operand in TMEM, 32 packed columns each) x (column tile, MN-major), small terms first.
template <int D>
__device__ __forceinline__ void issue_acc(uint32_t acc, uint32_t parts, uint32_t b_mn) {
  auto run = [&](uint32_t d, int pa, int pb, uint32_t idesc, uint32_t accumulate) {
#pragma unroll
    for (int ks = 0; ks < BN / 16; ++ks)
      mma_ts<D>(d, parts + 32 * pa + 8 * ks, b_mn + pb * (BN * D * 2 >> 4) + ks * (D * 2), idesc, ks ? 1u : accumulate);
  };
  if constexpr (D == 32) {
    // 64 columns: 0..31 against the h part, 32..63 against the m part; the l part is added to the latter
    constexpr uint32_t i64 = sm100::idesc_bf16(BM, 64, 0, 1), i32 = sm100::idesc_bf16(BM, 32, 0, 1);
    run(acc, 1, 0, i64, 0u);
    run(acc + 32, 0, 2, i32, 1u);
    run(acc, 2, 0, i32, 1u);
    run(acc, 0, 0, i64, 1u);
  } else {
    constexpr uint32_t id = sm100::idesc_bf16(BM, D, 0, 1);
    run(acc, 1, 1, id, 0u);
    run(acc, 0, 2, id, 1u);
    run(acc, 2, 0, id, 1u);
    run(acc, 0, 1, id, 1u);
    run(acc, 1, 0, id, 1u);
    run(acc, 0, 0, id, 1u);
  }
}
// descriptor word of a column tile as such an operand (D = 32: a step from the h to the m part)
__device__ __forceinline__ uint32_t desc_mn(uint32_t saddr, int D) { return sm100::desc_lo(saddr, BN * D * 2); }

// Adds this warp's half of the features of one tile's accumulator to the running sums (packed pairs).
template <int D>
__device__ __forceinline__ void promote(uint64_t (&run)[D / 4], uint32_t taddr, int cpart) {
  using namespace sm100;
  if constexpr (D == 64) {
    uint32_t a[32];
    tmem_ld32(taddr + cpart * 32, a);
    tmem_wait_ld(a);
#pragma unroll
    for (int e = 0; e < 16; ++e) run[e] = add2(run[e], pack2u(a[2 * e], a[2 * e + 1]));
  } else {
    uint32_t a[16], b[16];
    tmem_ld16(taddr + cpart * 16, a);
    tmem_ld16(taddr + 32 + cpart * 16, b);
    tmem_wait_ld(a, b);
#pragma unroll
    for (int e = 0; e < 8; ++e)
      run[e] = add2(run[e], add2(pack2u(a[2 * e], a[2 * e + 1]), pack2u(b[2 * e], b[2 * e + 1])));
  }
}

// (sum + add) * scale -> one row's half of the features; returns its dot product with x when wanted.
template <int D>
__device__ __forceinline__ float store_half(const uint64_t (&run)[D / 4], float* dst, const float* add, const float* xr,
                                            float scale) {
  using namespace sm100;
  float part = 0.f;
  const bool wide = (((uintptr_t)dst | (uintptr_t)add | (uintptr_t)xr) & 31) == 0;
#pragma unroll
  for (int b = 0; b < D / 16; ++b) {
    float f[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) unpack2(run[4 * b + e], f[2 * e], f[2 * e + 1]);
    if (add) {
      uint32_t aw[8];
      ldg32(add + 8 * b, aw, wide);
#pragma unroll
      for (int e = 0; e < 8; ++e) f[e] += __uint_as_float(aw[e]);
    }
    uint32_t w[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      f[e] *= scale;
      w[e] = __float_as_uint(f[e]);
    }
    stg32(dst + 8 * b, w, wide);
    if (xr) {
      uint32_t xw[8];
      ldg32(xr + 8 * b, xw, wide);
#pragma unroll
      for (int e = 0; e < 8; ++e) part = fmaf(f[e], __uint_as_float(xw[e]), part);
    }
  }
  return part;
}

// One row's half of the features of every kind of result; `row` < nrows.
template <int D>
__device__ __forceinline__ void store_forward(const SplitArgs& a, const uint64_t (&run)[D / 4], size_t grow, int cpart,
                                              float dsum) {
  if (cpart == 0) a.den_out[grow * a.den_stride] = dsum;
  const size_t at = grow * D + cpart * (D / 2);
  if (a.o_stride == D) {
    store_half<D>(run, a.o1 + at, a.o1_add ? a.o1_add + at : nullptr, nullptr, 1.0f / dsum);
  } else {             // rows of d + 1 floats: no alignment to use
    const float inv = 1.0f / dsum;
    float* dst = a.o1 + grow * a.o_stride + cpart * (D / 2);
#pragma unroll
    for (int e = 0; e < D / 4; ++e) {
      float lo, hi;
      sm100::unpack2(run[e], lo, hi);
      dst[2 * e] = lo * inv;
      dst[2 * e + 1] = hi * inv;
    }
  }
}

// ---- host ----
// Tensor map of rows of [h | m | l] whose boxes are `rows` rows of one part.
template <int D>
int split_map(CUtensorMap* m, const void* base, int heads, int n, int rows) {
  return D == 64 ? tma_map_bf16(m, base, heads, n, 3 * D, rows) : tma_map_bf16_half(m, base, heads, n, 3 * D, rows);
}
inline int set_sizes(const fastmax_problem& p, int heads, int nrows, int ncols, SplitArgs* a, long long* blocks) {
  a->heads = heads;
  a->nrows = nrows;
  a->ncols = ncols;
  a->ntr = (nrows + BM - 1) / BM;
  a->ratio = p.bh / p.bhkv;
  a->off = p.nk - p.nq;
  a->mask = p.mask;
  a->a0 = p.a0;
  a->a1 = p.a1;
  a->a2 = p.p == 2 ? p.a2 : 0.f;
  a->lim = p.lim;
  *blocks = (long long)heads * a->ntr;
  if (*blocks > 0x7FFF0000LL) return fail(FASTMAX_E_ARG, "heads x row tiles = %lld exceeds the grid limit", *blocks);
  return FASTMAX_OK;
}

}  // namespace split

// fm_dense_split_rows.cu; q, gs, k, v: parts
bool split_rows_serve(const fastmax_problem& p, int mode, int chunk);
int split_rows_forward(const Ctx& c, const void* q, const void* k, const void* v, const split::SplitArgs& a);
int split_rows_dq(const Ctx& c, const void* q, const void* gs, const void* k, const void* v, const split::SplitArgs& a);

}  // namespace fm
