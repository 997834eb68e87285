// Persistent score kernels: the row tiles of 128 rows that a CTA takes one after the other, and their column tiles.
#pragma once

#include "fm_common.cuh"

namespace fm {

// In which order row tiles are dealt out to the CTAs of a grid:
//   ORDER_LINEAR   head by head (row tiles of the same length, or one to a CTA)
//   ORDER_TILES    causal grids of a few waves: tile by tile over all chunks and heads, the longest first, every other round
//                  backwards.  (Chunks head by head instead, float32 forward / grad_q, us: 8 heads of 8192 in chunks of 2048
//                  111 / 187, so 94 / 150; 24 heads of 5000, d 32, in chunks of 1024 92 / 105, so 72 / 90)
//   ORDER_PAIRS    longer causal grids: head by head, so that a head's column tiles stay in L2, the i-th longest row tile
//                  together with the i-th shortest, so that every CTA gets the same work
enum { ORDER_LINEAR = 0, ORDER_TILES = 1, ORDER_PAIRS = 2 };
inline int row_order(const fastmax_problem& p, long long heads, long long ntr, int ctas_per_sm) {
  if (!p.mask || heads * ntr <= 148 * ctas_per_sm) return ORDER_LINEAR;
  return heads * ntr > 8LL * 148 * ctas_per_sm ? ORDER_PAIRS : ORDER_TILES;
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
