// What the read-outs of second-order states share (fm_readout.cu, fm_split_moments.cu), head dimension 64: the layout of the
// type A operand copies, the walk of a persistent CTA over the token groups, and small access helpers.
#pragma once
#include "fm_common.cuh"
#include "fm_sm100.cuh"

namespace fm {
namespace rdo {
using namespace sm100;

constexpr int D = 64;
constexpr int TILE = 128 * D * 2;         // 128 rows of 64 bf16

// Type A: 17 steps, streamed in this order.  Step 0 (16 KB, 128-byte swizzle): rows 0..63 S1 transposed (row c, a along
// K), rows 64..127 E (row b, a along K).  Step 1 + 4 g + j holds two slices, the sixteen value columns of group g against
// the features b of octet j, then of octet 7 - j, so that every step has five K steps in all.  The 128 rows of a slice are
// (c / 8 % 2) * 64 + b % 8 * 8 + c % 8.  A slice is unswizzled K-major: per K step of 16 features two halves of 2048
// bytes, in them 128-byte groups of eight rows.  One feature b and eight value columns are one such group, which is what
// the CTA that owns b writes.
constexpr int A_STEPS = 17;
constexpr int A_STAGE = 5 * 4096;
constexpr int A_BYTES = TILE + 16 * A_STAGE;
__device__ __forceinline__ int a_slice(int g, int oct) {
  const int j = oct < 4 ? oct : 7 - oct;
  return TILE + (g * 4 + j) * A_STAGE + (oct < 4 ? 0 : ((j >> 1) + 1) * 4096);
}
__device__ __forceinline__ int swz(int row, int byte) { return row * 128 + (byte ^ ((row & 7) << 4)); }

constexpr int BLK_LD = 68;

struct RdArgs {
  const char* copies;     // A_BYTES or B_BYTES per state
  const float* state;     // fp32 states, for the constant row and S1's normaliser column
  const float* uvec;      // type B: (heads, n) dvec, whose negative is e; null: e = 1
  float* out;             // (heads, n, 64) fp32
  float* den;             // type A: (heads, n), may be null
  const stat_t* stat_q;
  const stat_t* stat_k;
  float a0, a1, a2, lim;
  size_t per_state;
  int dvp, heads, n;
  int items;              // heads * groups
  int chunk, nchunk;      // chunk 0: one state per head
  int per_chunk;          // groups of a chunk
  int first, groups;      // groups of 256 tokens of a head that are read out: first .. first + groups - 1
  int zero_first, zero_groups;   // groups whose state is empty: zeros are written
  int wide_io;            // out is 32-byte aligned
};
// A CTA's walk over the items blockIdx.x, blockIdx.x + gridDim.x, ...: head, first token and state of the present one.
struct Walk {
  int left, head, grp, dhead, dgrp;
  __device__ __forceinline__ explicit Walk(const RdArgs& a) {
    left = (a.items - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    head = blockIdx.x / a.groups;
    grp = blockIdx.x % a.groups;
    dhead = gridDim.x / a.groups;
    dgrp = gridDim.x % a.groups;
  }
  __device__ __forceinline__ bool more() const { return left > 0; }
  __device__ __forceinline__ void next(const RdArgs& a) {
    --left;
    head += dhead;
    grp += dgrp;
    if (grp >= a.groups) { grp -= a.groups; ++head; }
  }
  __device__ __forceinline__ int tok0(const RdArgs& a) const { return (a.first + grp) * 256; }
  __device__ __forceinline__ int state(const RdArgs& a) const {
    return a.chunk > 0 ? head * a.nchunk + (a.first + grp) / a.per_chunk : head;
  }
};
__device__ __forceinline__ uint4 lds128(uint32_t saddr) {
  uint4 r;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(saddr));
  return r;
}
__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
// K steps of D[tmem] = A[smem] B[smem]^T, A in the 128-byte swizzle (32 bytes per step), B unswizzled in the layout of
// the type A slices (4096 bytes per step, K halves 2048 bytes apart, groups of eight rows 128 bytes apart)
constexpr uint32_t kDescHiFlat = (128u >> 4) | (1u << 14);
__device__ __forceinline__ void mma_steps(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, int steps,
                                          bool accumulate = false) {
  for (int ks = 0; ks < steps; ++ks)
    asm volatile(
        "{\n"
        ".reg .b64 da, db;\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %6, 0;\n"
        "mov.b64 da, {%1, %3};\n"
        "mov.b64 db, {%2, %4};\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n"
        "}\n"
        ::"r"(d_tmem), "r"(a_lo + ks * 2), "r"(b_lo + ks * (4096 >> 4)), "r"(kDescHi), "r"(kDescHiFlat), "r"(idesc),
          "r"(ks > 0 || accumulate ? 1u : 0u)
        : "memory");
}

}  // namespace rdo
}  // namespace fm
