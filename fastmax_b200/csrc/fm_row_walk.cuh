// Persistent score kernels: the row tiles of 128 rows that a CTA takes one after the other, and their column tiles.
#pragma once

#include "fm_common.cuh"

namespace fm {

// In which order row tiles are dealt out to the CTAs of a grid:
//   ORDER_LINEAR   head by head (row tiles of the same length, or one to a CTA)
//   ORDER_TILES    causal: tile by tile over all chunks and heads, the longest first, every other round backwards
//   ORDER_PAIRS    causal: head by head, so that a head's column tiles stay in L2, the i-th longest row tile of a head together
//                  with the i-th shortest, so that every pair is the same work
// A grid of up to eight waves goes by tiles.  (Chunks head by head instead, float32 forward / grad_q, us: 8 heads of 8192 in
// chunks of 2048 111 / 187, so 94 / 150.)  Longer ones go in pairs where pairs fill their rounds, and in any case beyond
// forty waves.  bf16 forward, tiles / pairs, as parts of what a CTA per row tile takes: 1300 causal columns (pairs fill 86 % of
// theirs) 0.92 / 1.08 at 1188 row tiles, 0.90 / 1.05 at 2046, 0.85 / 1.01 at 3003; 2200 columns 0.88 / 0.97 at 1188 (80 %), 0.87 / 0.86 at
// 2052 (99 %), 0.82 / 0.81 at 4104; chunks of 2048 0.82 / 0.75 at 2048 row tiles of whole chunks, 0.81 / 0.93 (grad_k + grad_v 0.86 / 1.24) at
// 2106 where the last chunk is shorter.
enum { ORDER_LINEAR = 0, ORDER_TILES = 1, ORDER_PAIRS = 2 };
inline int row_order(const fastmax_problem& p, long long heads, long long ntr, int ctas_per_sm, int chunk) {
  const long long ctas = 148LL * ctas_per_sm, tiles = heads * ntr, units = heads * ((ntr + 1) / 2), rounds = (units + ctas - 1) / ctas;
  if (!p.mask || tiles <= ctas) return ORDER_LINEAR;
  if (tiles <= 8 * ctas) return ORDER_TILES;
  const bool even = chunk == 0 || ntr % (chunk / 128) == 0;
  return tiles > 40 * ctas || (even && 100 * tiles >= 93 * 2 * ctas * rounds) ? ORDER_PAIRS : ORDER_TILES;
}

// Args: heads (row heads), ntr (row tiles of a head), order, nrows, ncols, off, mask, chunk, ratio.  REV: rows are keys, whose
// columns (queries) begin at the row instead of ending there, for each of the `ratio` query heads in turn.
template <class Args, int BN, bool REV>
struct RowWalk {
  int turn = 0, second = 0, head, r0;   // position; row head and first row
  int tb, jh, j;                        // first column tile; column tiles per column head, and in all
  int m = 0;                            // row tiles before this one
  __device__ __forceinline__ static int units(const Args& a) {
    return a.heads * (a.order == ORDER_PAIRS ? (a.ntr + 1) / 2 : a.ntr);
  }
  __device__ __forceinline__ int unit(const Args& a) const {
    const int b = (int)blockIdx.x, g = (int)gridDim.x;
    return turn * g + (a.order == ORDER_TILES && (turn & 1) ? g - 1 - b : b);
  }
  __device__ __forceinline__ bool live(const Args& a) const { return unit(a) < units(a); }
  // the row tile with the t-th most column tiles: one place of all chunks (without chunks, of the one there is) after the
  // other.  FWD from a chunk's last place on; the places that the last, shorter chunk lacks come in one chunk less.
  __device__ __forceinline__ static int longest(const Args& a, int t) {
    const int places = a.chunk > 0 ? a.chunk / 128 : a.ntr, chunks = (a.ntr + places - 1) / places;
    const int last = a.ntr - (chunks - 1) * places;                   // row tiles of the last chunk
    const int first = REV ? last * chunks : (places - last) * (chunks - 1);
    const bool after = t >= first;
    if (after) t -= first;
    const int of = REV == after ? chunks - 1 : chunks, at = t / of;
    return (t - at * of) * places + (REV ? (after ? last : 0) + at : (after ? last : places) - 1 - at);
  }
  __device__ __forceinline__ void open(const Args& a) {
    const int u = unit(a), per = a.order == ORDER_PAIRS ? (a.ntr + 1) / 2 : a.ntr;
    if (a.order == ORDER_TILES) {
      head = u % a.heads;
      r0 = longest(a, u / a.heads) * 128;
    } else {
      head = u / per;
      const int t = second ? a.ntr - 1 - u % per : u % per;
      r0 = (REV ? t : a.ntr - 1 - t) * 128;
    }
    int te = (a.ncols + BN - 1) / BN;
    tb = 0;
    if (a.mask) {
      if (REV) tb = max(0, r0 - a.off) / BN;
      else te = min(te, (min(r0 + 127, a.nrows - 1) + a.off) / BN + 1);
    }
    if (a.chunk > 0) {        // the row tile lies in one chunk (chunk % 256 == 0)
      const int cb = (r0 / a.chunk) * (a.chunk / BN);
      if (REV) te = min(te, cb + a.chunk / BN);
      else tb = cb;
    }
    jh = te - tb;             // at least one: every row sees a column and every column a row
    j = REV ? jh * a.ratio : jh;
  }
  __device__ __forceinline__ void next(const Args& a) {
    ++m;
    const int t = unit(a) % ((a.ntr + 1) / 2);
    if (a.order == ORDER_PAIRS && !second && a.ntr - 1 - t != t) {
      second = 1;
    } else {
      second = 0;
      ++turn;
    }
    if (live(a)) open(a);
  }
};

}  // namespace fm
