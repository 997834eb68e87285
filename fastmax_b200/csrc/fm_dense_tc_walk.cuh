// Arguments of the score kernels that walk row tiles (fm_dense_tc_walk.cu).
#pragma once

#include <cuda.h>

#include "fm_square.cuh"

namespace fm {
namespace walk {

enum { MODE_FWD = 0, MODE_DKDV = 1 };

struct WalkArgs {
  void* o;               // (heads, nrows, 64) bf16: out, or grad_k
  void* o2;              // DKDV: grad_v
  float* den_out;        // FWD: (heads, nrows) row sums
  const float* den_add;  // FWD: added to the row sum (may be null)
  const float* o_add;    // fp32 rows added before the division / rounding (may be null)
  const float* o2_add;
  const void* x;         // row operand in global memory (normalisation dots)
  const float* dvec;     // (heads, nq)
  float* dots;           // per head sum of o . x, or null
  const stat_t* stat_q;
  const stat_t* stat_k;
  int heads, nrows, ncols, off, mask, ntr, chunk, ratio, order;   // see RowWalk
  float a0, a1, a2, lim;
  Square sq;             // DKDV, where square_form() gives one
  // first-order chunks: running sums of the states, rows [y_a | 1] of `dvp` floats, d + 1 rows per (head, chunk)
  const float* st;
  int dvp, nchunk, zero_chunk;   // zero_chunk: the chunk whose running sum is empty (-1: none)
  int o_heads;           // FWD: > 0 writes out as (batch, nrows, o_heads, 64)
};

}  // namespace walk

// Boxes of 128 rows x 32 of a (mats, rows, 64) float32 array, 128-byte swizzle (fm_dense_tc.cu)
int tma_map_f32_rows(CUtensorMap* m, const float* base, size_t mats, size_t rows);

// Whether the kernels have the registers that their warpgroups exchange, which the compiler decides; where not, the short and wide
// kernels serve their rows.
bool dense_tc_walk_runs(bool forward);
int dense_tc_walk_forward(const Ctx& c, const void* q, const void* k, const void* v, const walk::WalkArgs& a);
int dense_tc_walk_dkdv(const Ctx& c, const void* k, const void* v, const void* q, const void* gs, const walk::WalkArgs& a,
                       const FirstState* fs = nullptr);

}  // namespace fm
