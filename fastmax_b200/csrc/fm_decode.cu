// Token-by-token (decode) Fastmax attention against a persistent moment state.
//
// The reference's model decodes with a key/value cache: every new token calls the
// attention with one query row and all cached keys (model.py:501-504, 828-852), so
// the cost per token grows with the length.  The factorised form needs no cache:
// per key/value head keep
//
//   S0[c]       = sum_j            vt_j[c]
//   S1[a][c]    = sum_j k_j[a]     vt_j[c]
//   S2[a][b][c] = sum_j k_j[a] k_j[b] vt_j[c]          (p = 2 only)
//
// with vt_j = (v_j, 1), over the RAW keys; the max-norm scaling lim / max_j |k_j|
// multiplies whole blocks (S1 by s, S2 by s^2), so it is applied when a query reads
// the state and the running maximum is one float in the state's header.  A query
// row is normalised by its own norm, as it is when the reference's attention is
// called with a single query row.  One step adds the new token to the state and
// reads it:  num[c] = a0 S0[c] + a1 s (q.S1)[c] + a2 s^2 (q(x)q . S2)[c],
// out = num[:d] / num[d]  -- the last row of causal attention over the tokens so far
// (fastmax_cuda_forward.cu:109, 132-150 with nq = 1).
//
// The state is fp32, F = (d^2 +) d + 1 rows of d+1 floats (second-order rows first, the
// constant row last) after a 4-word header {max |k|^2, token count (int32 bits), arrival count of a
// running step (0 between calls), 0} per key/value head.  S2 is symmetric in (a, b), so only its
// upper triangle of tiles is computed; every result is written to both of its rows.
//
// The kernels:
//   step_kernel    one token and its read-out: bound by the state's traffic with many heads, by a chain of latencies with
//                  few.  The lower triangle is written but never read: 4 F (d+1) x (1 + 0.56) bytes at d = 64.  Measured, us,
//                  p = 2: 1024 heads, d = 64: 312 for 1.73 GB = 5.5 TB/s (352 when every thread fenced and each CTA waited for its
//                  arrival, 330 with one thread's fence); 128 heads, d = 128: 271 (334).  Steps one after another in a graph: 8
//                  key/value heads of 4 query heads 8.9 (9.2 when every thread fenced), 4 heads, float32, 6.1 (6.3), 64 heads 22.8
//                  (24.3); p = 1, whose head is one CTA at d 32 and 64, 64 heads of d = 32 3.8 (5.6 with a fence and a counter).
//                  The same bytes in 2 KB runs, without the arithmetic: 258.  Other arrangements for 1024 heads:
//                  several groups of blocks to a CTA 397, five CTAs to an SM 377 (both before the above); tiles by bulk copies
//                  through shared memory, CTAs as here 366 / 291 (one kernel / without the sums; d = 128 319 / 264, kept),
//                  persistent with 1 to 4 CTAs an SM 338 to 403.
//   sum_kernel     the heads' sums, where step_kernel leaves them out (kSharesFrom).
//   few_kernel     the same update for a few tokens of a prompt.
//   append_kernel  many tokens (prompt), float32 or d = 32: bound by the FMA pipe; see there.  bf16 prompts of
//                  d 64 and 128 go to the tensor cores (fm_decode_tc.cu).
#include "fm_common.cuh"
#include "fm_sm100.cuh"

namespace fm {

__device__ int g_step_status = 0;

namespace {
using namespace sm100;

constexpr int kTile = 8;        // step_kernel: a thread's block is half (4 x 8) of an 8 x 8 tile of second-order rows ...
constexpr int kHalf = 4;
constexpr int kLinear = kHalf * kTile;   // ... or 32 first-order rows, or the constant row
constexpr int kTokBatch = 32;   // tokens staged in shared memory per pass
constexpr int kQueries = 4;     // query heads of a group that are read out together
constexpr int kHeader = 4;

struct DecArgs {
  int bh, bhkv, ratio, p, normalize;
  float a0, a1, a2, lim;
  long long n_new;       // tokens to add
  long long head_floats; // kHeader + F * (d + 1)
};

template <int D> struct DecCfg {
  static constexpr int DV = D + 1;
  static constexpr int RPB = (D == 128) ? 2 : 256 / DV;           // row blocks per CTA
  static constexpr int PER_SM = (D == 64) ? 4 : 3;                // CTAs per SM, a compromise with spills
  static constexpr int THREADS = RPB * DV;
  static constexpr int NT = D / kTile;
  static constexpr int NB2 = NT * (NT + 1);                       // second-order half tiles per head
  static constexpr int NB1 = (D + kLinear - 1) / kLinear;         // first-order blocks per head
  __host__ __device__ static constexpr int ctas(int p) { return ((p == 2 ? NB2 : 0) + NB1 + 1 + RPB - 1) / RPB; }
};

// A tile of step_kernel in shared memory: its rows are kTile runs of kTile * DV contiguous floats, each kept from the 16-byte
// boundary before it on; its mirror image's rows are kTile more.
template <int D> struct RunCfg {
  static constexpr int RUN = kTile * DecCfg<D>::DV, LD = RUN + 4, TILE = kTile * LD, SMEM = 2 * TILE * 4;
};

// Sum of squares of x[0..D) by one warp; the result is valid in every lane.
template <int D>
__device__ __forceinline__ float warp_norm2(const float* x, int lane) {
  float n2 = 0.0f;
#pragma unroll
  for (int e = lane; e < D; e += 32) n2 = fmaf(x[e], x[e], n2);
#pragma unroll
  for (int m = 16; m >= 1; m >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, m);
  return n2;
}

// 16 bytes of T from global memory as fp32 values.
__device__ __forceinline__ void load16_to_f32(const float* src, float* dst) {
  const float4 w = __ldg(reinterpret_cast<const float4*>(src));
  dst[0] = w.x; dst[1] = w.y; dst[2] = w.z; dst[3] = w.w;
}
__device__ __forceinline__ void load16_to_f32(const __nv_bfloat16* src, float* dst) {
  const uint4 w = __ldg(reinterpret_cast<const uint4*>(src));
  const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    dst[2 * e] = __uint_as_float(ww[e] << 16);
    dst[2 * e + 1] = __uint_as_float(ww[e] & 0xFFFF0000u);
  }
}

// 16 bytes of T held in registers to shared memory as fp32 values.
template <typename T>
__device__ __forceinline__ void store16_as_f32(const uint4& w, float* dst) {
  if constexpr (sizeof(T) == 4) {
    *reinterpret_cast<uint4*>(dst) = w;
  } else {
    *reinterpret_cast<uint4*>(dst) = make_uint4(w.x << 16, w.x & 0xFFFF0000u, w.y << 16, w.y & 0xFFFF0000u);
    *reinterpret_cast<uint4*>(dst + 4) = make_uint4(w.z << 16, w.z & 0xFFFF0000u, w.w << 16, w.w & 0xFFFF0000u);
  }
}

// A tile of the upper triangle, counted row by row: (ta, tb) with ta <= tb < nt.
__device__ __forceinline__ void upper_tile(int idx, int nt, int& ta, int& tb) {
  ta = 0;
  while (idx >= nt - ta) { idx -= nt - ta; ++ta; }
  tb = ta + idx;
}

// A thread owns one column c of one block of rows, so a CTA's accesses are runs of whole rows: half of an 8 x 8 tile of
// the second order on or above the diagonal, 32 first-order rows, or the constant row.
template <int D> struct Block {
  typedef DecCfg<D> C;
  int a0, b0, kind, live, ustride;        // kind 2, 1, 0: order of the block (-1: none); live: rows of it that exist
  bool diagonal;
  float *base, *base2;                    // row (u, i) at base[u * ustride + i * DV]; a tile's mirror image at base2
  float s[kHalf][kTile];

  // block sb of the head whose rows start at `rows`, column c
  __device__ __forceinline__ void place(int sb, int p, float* rows, int c) {
    const int nb2 = p == 2 ? C::NB2 : 0, n2rows = p == 2 ? D * D : 0;
    diagonal = false;
    a0 = b0 = 0;
    kind = -1;
    live = 0;
    if (sb < nb2) {
      upper_tile(sb >> 1, C::NT, a0, b0);
      diagonal = a0 == b0;
      a0 = a0 * kTile + (sb & 1) * kHalf;
      b0 *= kTile;
      kind = 2;
      live = kHalf * kTile;
    } else if (sb < nb2 + C::NB1) {
      a0 = (sb - nb2) * kLinear;
      kind = 1;
      live = D - a0 < kLinear ? D - a0 : kLinear;
    } else if (sb == nb2 + C::NB1) {
      kind = 0;
      live = 1;
    }
    base = rows + c + (long long)C::DV * (kind == 2 ? a0 * D + b0 : n2rows + (kind == 1 ? a0 : D));
    base2 = rows + c + (long long)C::DV * (b0 * D + a0);
    ustride = (kind == 2 ? D : kTile) * C::DV;
  }
  __device__ __forceinline__ void load() {
#pragma unroll
    for (int u = 0; u < kHalf; ++u)
#pragma unroll
      for (int i = 0; i < kTile; ++i) s[u][i] = (u * kTile + i < live) ? base[u * ustride + i * C::DV] : 0.0f;
  }
  // The same from and to shared memory (kind 2): the half tile's rows (half * kHalf + u, i) at column c of the tile's runs,
  // which start x floats behind a 16-byte boundary, and of its mirror image's.
  __device__ __forceinline__ void load_staged(const float* tile, int half, int x, int c) {
#pragma unroll
    for (int u = 0; u < kHalf; ++u)
#pragma unroll
      for (int i = 0; i < kTile; ++i) s[u][i] = tile[(half * kHalf + u) * RunCfg<D>::LD + x + i * C::DV + c];
  }
  __device__ __forceinline__ void store_staged(float* tile, int half, int x, int c) const {
    typedef RunCfg<D> S;
#pragma unroll
    for (int u = 0; u < kHalf; ++u)
#pragma unroll
      for (int i = 0; i < kTile; ++i) {
        tile[(half * kHalf + u) * S::LD + x + i * C::DV + c] = s[u][i];
        if (!diagonal) tile[S::TILE + i * S::LD + x + (half * kHalf + u) * C::DV + c] = s[u][i];
      }
  }
  // what bulk copies leave out: a run's first floats up to a 16-byte boundary and its last ones after one
  __device__ __forceinline__ void store_edges(int half, int x, int c) const {
    const bool head = x > 0 && c < 4 - x, tail = c >= C::DV - x;
#pragma unroll
    for (int u = 0; u < kHalf; ++u) {
      if (head) base[u * ustride] = s[u][0];
      if (tail) base[u * ustride + (kTile - 1) * C::DV] = s[u][kTile - 1];
    }
    if (diagonal) return;
#pragma unroll
    for (int i = 0; i < kTile; ++i) {
      if (head && half == 0) base2[i * D * C::DV] = s[0][i];
      if (tail && half == 1) base2[(i * D + kHalf - 1) * C::DV] = s[kHalf - 1][i];
    }
  }
  // one token: k, and this column's value
  __device__ __forceinline__ void add(const float* k, float vc) {
    if (kind == 2) {
      float kb[kTile];
#pragma unroll
      for (int i = 0; i < kTile; ++i) kb[i] = k[b0 + i];
#pragma unroll
      for (int u = 0; u < kHalf; ++u) {
        const float ka = k[a0 + u];
#pragma unroll
        for (int i = 0; i < kTile; ++i) s[u][i] = fmaf(ka * kb[i], vc, s[u][i]);
      }
    } else if (kind == 1) {
#pragma unroll
      for (int u = 0; u < kHalf; ++u)
#pragma unroll
        for (int i = 0; i < kTile; ++i)
          if (u * kTile + i < live) s[u][i] = fmaf(k[a0 + u * kTile + i], vc, s[u][i]);
    } else if (kind == 0) {
      s[0][0] += vc;
    }
  }
  // the block's share of a read-out: query row q, scale sc of its products with keys
  __device__ __forceinline__ float read(const DecArgs& a, const float* q, float sc) const {
    float part = 0.0f;
    if (kind == 2) {
      // a tile above the diagonal stands for its mirror image too
      const float coef = a.a2 * sc * sc * (diagonal ? 1.0f : 2.0f);
#pragma unroll
      for (int u = 0; u < kHalf; ++u) {
        float row = 0.0f;
#pragma unroll
        for (int i = 0; i < kTile; ++i) row = fmaf(q[b0 + i], s[u][i], row);
        part = fmaf(coef * q[a0 + u], row, part);
      }
    } else if (kind == 1) {
#pragma unroll
      for (int u = 0; u < kHalf; ++u)
#pragma unroll
        for (int i = 0; i < kTile; ++i)
          if (u * kTile + i < live) part = fmaf(a.a1 * sc * q[a0 + u * kTile + i], s[u][i], part);
    } else if (kind == 0) {
      part = a.a0 * s[0][0];
    }
    return part;
  }
  __device__ __forceinline__ void store() const {
#pragma unroll
    for (int u = 0; u < kHalf; ++u)
#pragma unroll
      for (int i = 0; i < kTile; ++i)
        if (u * kTile + i < live) base[u * ustride + i * C::DV] = s[u][i];
    if (kind == 2 && !diagonal) {
#pragma unroll
      for (int i = 0; i < kTile; ++i)
#pragma unroll
        for (int u = 0; u < kHalf; ++u) base2[(i * D + u) * C::DV] = s[u][i];
    }
  }
};

// One token per head and its read-out.  A CTA takes one group of RPB blocks of its head and leaves their share of the
// read-out in scratch[query head][CTA][column]; the CTA of a head that arrives last (a counter in the head's header) adds
// the shares in CTA order, divides and writes the output row.
// SUMS says how: the last CTA to arrive; SUMS_APART: none, sum_kernel does the rest; SUMS_ALONE: the head is one CTA, which needs
// neither fence nor counter.
enum { SUMS_LAST = 0, SUMS_APART = 1, SUMS_ALONE = 2 };
template <typename T, int D, int SUMS>
__global__ void __launch_bounds__(DecCfg<D>::THREADS, DecCfg<D>::PER_SM) step_kernel(const DecArgs a, const T* __restrict__ q,
                                                                  const T* __restrict__ k, const T* __restrict__ v,
                                                                  float* __restrict__ state, float* __restrict__ scratch,
                                                                  T* __restrict__ out) {
  typedef DecCfg<D> C;
  typedef RunCfg<D> R;
  // With d = 128 a CTA has one tile, which bulk copies bring and take back: 264 instead of 295 us for 128 heads, the sums apart.
  // (With d = 64 291 instead of 294, with d = 32 107 instead of 99.)
  constexpr bool BULK = SUMS == SUMS_APART && D == 128;
  extern __shared__ __align__(16) float tile[];    // BULK
  __shared__ __align__(8) uint64_t tile_here;
  __shared__ float ks[D], vs[D + 1];       // the token; (v, 1)
  __shared__ float qs[kQueries][D];
  __shared__ float red[kQueries][C::RPB][C::DV];
  __shared__ float s_q2[kQueries];
  __shared__ float s_kmax2;
  __shared__ int s_last;
  const int tid = threadIdx.x, r = tid / C::DV, c = tid - r * C::DV, lane = tid & 31;
  const int head = blockIdx.y;
  float* hs = state + head * a.head_floats;
  auto stage_queries = [&](long long qh, int ng) {
    for (int x = tid; x < ng * D; x += C::THREADS) qs[x / D][x % D] = ldf(q + qh * D + x);
  };
  auto norms = [&](int ng) {               // of the staged queries, one warp each
    if (tid < ng * 32) {
      const float n2 = warp_norm2<D>(qs[tid >> 5], lane);
      if (lane == 0) s_q2[tid >> 5] = n2;
    }
  };

  // BULK: lane l of the first warp copies run l of the tile.  x: floats from a 16-byte boundary to a run, the same for all of a
  // head, whose tiles start at multiples of four rows
  const int x = BULK ? (int)((uintptr_t)(hs + kHeader) >> 2 & 3) : 0;
  const bool copies = BULK && (int)blockIdx.x < C::NB2 / 2 && tid < kTile;
  float *own = nullptr, *image = nullptr;
  if constexpr (BULK) {
    static_assert(C::RPB == 2, "a tile, two halves, to a CTA");
    if (copies) {
      int ta, tb;
      upper_tile(blockIdx.x, C::NT, ta, tb);
      own = hs + kHeader + (long long)C::DV * ((ta * kTile + tid) * D + tb * kTile);
      image = ta == tb ? nullptr : hs + kHeader + (long long)C::DV * ((tb * kTile + tid) * D + ta * kTile);
      const uint32_t bytes = 4 * R::RUN + (x ? 16 : 0);
      if (tid == 0) {
        mbar_init(smem_u32(&tile_here), 1);
        mbar_fence_init();
        mbar_expect_tx(smem_u32(&tile_here), kTile * bytes);
      }
      __syncwarp((1u << kTile) - 1u);
      bulk_load(smem_u32(tile + tid * R::LD), own - x, bytes, smem_u32(&tile_here));
    }
  }

  // the token and the first queries travel with the block's rows (a step of one sequence is a chain of latencies)
  static_assert(C::THREADS >= 2 * D, "a thread an element of the token");
  const int ng0 = a.ratio < kQueries ? a.ratio : kQueries;
  const float tok = tid < D ? ldf(k + (long long)head * D + tid) : (tid < 2 * D ? ldf(v + (long long)head * D + tid - D) : 0.0f);
  constexpr int QPT = (kQueries * D + C::THREADS - 1) / C::THREADS;
  float q_first[QPT];
#pragma unroll
  for (int i = 0; i < QPT; ++i) {
    const int x = tid + i * C::THREADS;
    q_first[i] = x < ng0 * D ? ldf(q + (long long)head * a.ratio * D + x) : 0.0f;
  }
  const float kmax2 = hs[0];
  Block<D> blk;
  blk.place(blockIdx.x * C::RPB + r, a.p, hs + kHeader, c);
  const bool bulk = BULK && blk.kind == 2;
  if (!bulk) blk.load();
  if (tid < D) ks[tid] = tok;
  else if (tid < 2 * D) vs[tid - D] = tok;
  if (tid == 0) vs[D] = 1.0f;
#pragma unroll
  for (int i = 0; i < QPT; ++i) {
    const int x = tid + i * C::THREADS;
    if (x < ng0 * D) qs[x / D][x % D] = q_first[i];
  }
  __syncthreads();
  norms(ng0);
  constexpr int kLastWarp = C::THREADS / 32 - 1;         // a full warp; the queries have the first ones
  if ((tid >> 5) == kLastWarp) {
    const float n2 = warp_norm2<D>(ks, lane);
    if (lane == 0) s_kmax2 = fmaxf(kmax2, n2);
  }
  bool here = true;
  if (bulk) {
    here = mbar_wait(smem_u32(&tile_here), 0);
    if (!here) atomicCAS(&g_step_status, 0, 1);
    blk.load_staged(tile, r, x, c);
  }
  blk.add(ks, vs[c]);
  if (bulk) {
    blk.store_staged(tile, r, x, c);
    fence_proxy_async();
  }
  __syncthreads();
  if (copies && here) {
    const int skip = (4 - x) & 3;
    const uint32_t from = smem_u32(tile + tid * R::LD + x + skip), bytes = 4 * (R::RUN - (x ? 4 : 0));
    bulk_store(own + skip, from, bytes);
    if (image) bulk_store(image + skip, from + 4 * R::TILE, bytes);
  }
  auto scale = [&](int g) {
    return a.normalize ? (a.lim * rsqrtf(s_q2[g])) * (a.lim * rsqrtf(s_kmax2)) : 1.0f;
  };

  // this CTA's rows of the scratch, kQueries queries at a time
#pragma unroll 1
  for (int g0 = 0; g0 < a.ratio; g0 += kQueries) {
    const int ng = a.ratio - g0 < kQueries ? a.ratio - g0 : kQueries;
    const long long qh = (long long)head * a.ratio + g0;
    if (g0 > 0) {
      __syncthreads();
      stage_queries(qh, ng);
      __syncthreads();
      norms(ng);
      __syncthreads();
    }
#pragma unroll 1
    for (int g = 0; g < ng; ++g) red[g][r][c] = blk.read(a, qs[g], scale(g));
    __syncthreads();
    for (int x = tid; x < ng * C::DV; x += C::THREADS) {
      const int g = x / C::DV, cc = x - g * C::DV;
      float tot = 0.0f;
#pragma unroll
      for (int rr = 0; rr < C::RPB; ++rr) tot += red[g][rr][cc];
      __stcg(scratch + ((qh + g) * gridDim.x + blockIdx.x) * C::DV + cc, tot);
    }
  }
  if constexpr (SUMS == SUMS_APART) {
    if (!bulk) blk.store();
    else if (here) blk.store_edges(r, x, c);
    if (copies) tma_store_wait_read();     // the bulk copies have read this CTA's shared memory
    return;
  }
  if constexpr (SUMS == SUMS_LAST) {
    // One thread's fence, for all of the CTA: the others go on to their stores.  With few CTAs that leave several queries' shares
    // each, every thread fences its own ahead of the barrier.  us, every thread / the last one / the first one: 8 heads 7.47 / 7.55 /
    // 7.39, 9 heads 7.43 / 7.65 / 7.29, 20 heads 10.94 / 10.54 / 10.58, 64 heads of d = 32 7.73 / 7.47 / 7.21; 2 key/value heads of 4
    // queries 7.20 / 7.26 / 7.25, 16 of 4 11.73 / 10.99 / 11.00
    const bool each = a.ratio > 1 && gridDim.x * gridDim.y <= 100;
    if (each) __threadfence();
    __syncthreads();
    if (tid == 0) {
      if (!each) __threadfence();
      const int before = atomicAdd(reinterpret_cast<int*>(hs + 2), 1);
      s_last = before == (int)gridDim.x - 1;
    }
  }
  // The block is written only now: the fence above need not wait for it, and a CTA leaves with its stores in flight.
  blk.store();
  __syncthreads();
  if constexpr (SUMS == SUMS_LAST) {
    if (!s_last) return;
    __threadfence();
  }
  if (tid == 0) {
    hs[0] = s_kmax2;
    // the token count is an integer bit pattern in the float slot: exact past 2^24 tokens
    hs[1] = __int_as_float(__float_as_int(hs[1]) + 1);
    hs[2] = 0.0f;
  }
  for (int g0 = 0; g0 < a.ratio; g0 += kQueries) {
    const int ng = a.ratio - g0 < kQueries ? a.ratio - g0 : kQueries;
    const long long qh = (long long)head * a.ratio + g0;
    // all queries' rows at once: one wait for memory instead of one a query
    float tot[kQueries];
#pragma unroll
    for (int g = 0; g < kQueries; ++g) tot[g] = 0.0f;
    const float* src = scratch + qh * gridDim.x * C::DV + c;
    const long long per_query = (long long)gridDim.x * C::DV;
    if (ng == 1) {
#pragma unroll 8
      for (int b = r; b < (int)gridDim.x; b += C::RPB) tot[0] += __ldcg(src + (long long)b * C::DV);
    } else {
#pragma unroll 4
      for (int b = r; b < (int)gridDim.x; b += C::RPB) {
#pragma unroll
        for (int g = 0; g < kQueries; ++g)
          if (g < ng) tot[g] += __ldcg(src + g * per_query + (long long)b * C::DV);
      }
    }
#pragma unroll
    for (int g = 0; g < kQueries; ++g)
      if (g < ng) red[g][r][c] = tot[g];
    __syncthreads();
    for (int x = tid; x < ng * D; x += C::THREADS) {
      const int g = x / D, cc = x - g * D;
      float num = 0.0f, den = 0.0f;
#pragma unroll
      for (int rr = 0; rr < C::RPB; ++rr) { num += red[g][rr][cc]; den += red[g][rr][D]; }
      stf(out + qh * D + x, num / den);
    }
    __syncthreads();
  }
}

// The shares that step_kernel's CTAs left in the scratch, in their order: a CTA per query row, which it divides and writes; the
// first one of a key/value head also counts the token.
template <typename T, int D>
__global__ void __launch_bounds__(DecCfg<D>::THREADS) sum_kernel(const DecArgs a, int shares, const T* __restrict__ k,
                                                                 float* __restrict__ state, const float* __restrict__ scratch,
                                                                 T* __restrict__ out) {
  typedef DecCfg<D> C;
  __shared__ float red[C::RPB][C::DV];
  const int tid = threadIdx.x, r = tid / C::DV, c = tid - r * C::DV, lane = tid & 31;
  const int qh = blockIdx.x, head = qh / a.ratio;
  const float* src = scratch + (long long)qh * shares * C::DV + c;
  float tot = 0.0f;
#pragma unroll 10
  for (int b = r; b < shares; b += C::RPB) tot += __ldcg(src + (long long)b * C::DV);
  if (qh % a.ratio == 0 && tid < 32) {
    float n2 = 0.0f;
#pragma unroll
    for (int e = lane; e < D; e += 32) {
      const float x = ldf(k + (long long)head * D + e);
      n2 = fmaf(x, x, n2);
    }
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, m);
    if (lane == 0) {
      float* hs = state + head * a.head_floats;
      hs[0] = fmaxf(hs[0], n2);
      // the token count is an integer bit pattern in the float slot: exact past 2^24 tokens
      hs[1] = __int_as_float(__float_as_int(hs[1]) + 1);
    }
  }
  red[r][c] = tot;
  __syncthreads();
  if (tid < D) {
    float num = 0.0f, den = 0.0f;
#pragma unroll
    for (int rr = 0; rr < C::RPB; ++rr) { num += red[rr][tid]; den += red[rr][D]; }
    stf(out + (long long)qh * D + tid, num / den);
  }
}

// A few tokens of a prompt: one group of blocks per CTA, the tokens one after another.
template <typename T, int D>
__global__ void __launch_bounds__(DecCfg<D>::THREADS, DecCfg<D>::PER_SM) few_kernel(const DecArgs a, const T* __restrict__ k,
                                                                                    const T* __restrict__ v,
                                                                                    float* __restrict__ state) {
  typedef DecCfg<D> C;
  __shared__ __align__(16) float ks[kTokBatch][D];
  __shared__ float vs[kTokBatch][D + 1];   // (v, 1)
  __shared__ int s_kmax2_bits;   // max |k|^2 as its bit pattern: non-negative floats order like integers
  const int tid = threadIdx.x, r = tid / C::DV, c = tid - r * C::DV, lane = tid & 31;
  const int head = blockIdx.y;
  float* hs = state + head * a.head_floats;
  Block<D> blk;
  blk.place(blockIdx.x * C::RPB + r, a.p, hs + kHeader, c);
  blk.load();
  if (tid == 0) s_kmax2_bits = __float_as_int(hs[0]);
  __syncthreads();

  const T* kh = k + (long long)head * a.n_new * D;
  const T* vh = v + (long long)head * a.n_new * D;
  for (long long t0 = 0; t0 < a.n_new; t0 += kTokBatch) {
    const int nt = (int)((a.n_new - t0 < kTokBatch) ? a.n_new - t0 : kTokBatch);
    // stage the batch: 16-byte loads of k and v, converted to fp32
    constexpr int EPV = 16 / (int)sizeof(T), VPT = D / EPV;   // elements per load, loads per token
    for (int e = tid; e < nt * VPT; e += C::THREADS) {
      const int tok = e / VPT, x = (e - tok * VPT) * EPV;
      load16_to_f32(kh + (t0 + tok) * D + x, &ks[tok][x]);
      load16_to_f32(vh + (t0 + tok) * D + x, &vs[tok][x]);
      if (x == 0) vs[tok][D] = 1.0f;
    }
    __syncthreads();
    if (blockIdx.x == 0) {   // running maximum of |k|^2, the tokens spread over the CTA's full warps
      constexpr int kFullWarps = C::THREADS / 32;
      const int warp = tid >> 5;
      if (warp < kFullWarps) {
        float m = 0.0f;
        for (int tok = warp; tok < nt; tok += kFullWarps) m = fmaxf(m, warp_norm2<D>(ks[tok], lane));
        if (lane == 0) atomicMax(&s_kmax2_bits, __float_as_int(m));
      }
    }
    for (int tok = 0; tok < nt; ++tok) blk.add(ks[tok], vs[tok][c]);
    __syncthreads();
  }
  blk.store();
  if (blockIdx.x == 0 && tid == 0) {
    hs[0] = __int_as_float(s_kmax2_bits);
    hs[1] = __int_as_float(__float_as_int(hs[1]) + (int)a.n_new);
  }
}

// Prompt processing: S += sum over tokens of kx[a] kx[b] (v, 1)[c], kx = (k, 1, 0, 0, 0).
// A thread owns 4 x 4 pairs (a, b) of the upper triangle (of kx, so the first-order rows and the constant row
// are its last column of tiles) times 8 value columns, as 64 packed accumulators, and a share of the tile's
// normaliser column.  Per token it reads 4 + 4 + 8 floats of shared memory for 128 multiply-adds; with fewer
// pairs or columns per thread the loads would take the time (an LDS.128 moves 512 bytes per warp, four cycles
// of the SM's 128-byte port, against 32 for the multiply-adds).  The next batch's tokens are fetched into
// registers while the current one is processed.  64 heads x 4000 tokens, d = 64, bf16: 2.22 ms = 16 TFMA/s (5.59 ms
// when all ordered pairs were summed, 64 multiply-adds for 5 loads); the grid's last wave is nearly empty there.
template <int D> struct AppCfg {
  static constexpr int NT = D / 4 + 1;                       // tile rows of kx
  static constexpr int CG = D / 8;                           // column groups
  static constexpr int PE = 16 / CG;                         // pairs per thread of the normaliser column
  static constexpr int BPC = 128 / CG;                       // tiles per CTA
  static constexpr int THREADS = BPC * CG;
  __host__ __device__ static constexpr int tiles(int p) { return p == 2 ? NT * (NT + 1) / 2 : NT; }
  __host__ __device__ static constexpr int ctas(int p) { return (tiles(p) + BPC - 1) / BPC; }
};

template <typename T, int D>
__global__ void __launch_bounds__(AppCfg<D>::THREADS, 2) append_kernel(const DecArgs a, const T* __restrict__ k,
                                                                       const T* __restrict__ v,
                                                                       float* __restrict__ state) {
  typedef AppCfg<D> C;
  constexpr int DV = D + 1, KS = D + 4;
  constexpr int TB = 64 / (int)sizeof(T) * (D >= 128 ? 1 : 2) / 2;      // tokens per batch: bf16 32, float32 16 (D = 128: 8)
  constexpr int EPV = 16 / (int)sizeof(T), VPT = D / EPV;
  constexpr int NLD = (TB * VPT + C::THREADS - 1) / C::THREADS;         // 16-byte loads per thread, k and v each
  __shared__ __align__(16) float ks[TB][KS];
  __shared__ __align__(16) float vs[TB][D];
  __shared__ int s_kmax2_bits;
  const int tid = threadIdx.x, cg = tid % C::CG, head = blockIdx.y, lane = tid & 31;
  const int tile = blockIdx.x * C::BPC + tid / C::CG;
  const bool on = tile < C::tiles(a.p);
  int ta = 0, tb = C::NT - 1;
  if (a.p == 2) upper_tile(on ? tile : 0, C::NT, ta, tb);
  else ta = on ? tile : 0;
  const int a0 = ta * 4, b0 = tb * 4, c0 = cg * 8;
  const int ea = a0 + cg * C::PE / 4, eb = b0 + cg * C::PE % 4;         // this thread's first normaliser pair
  float* hs = state + head * a.head_floats;
  if (tid == 0) s_kmax2_bits = __float_as_int(hs[0]);

  uint64_t acc[4][2][8];            // [a][b pair][column]
  float acce[C::PE];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int c = 0; c < 8; ++c) acc[u][i][c] = 0ull;
#pragma unroll
  for (int e = 0; e < C::PE; ++e) acce[e] = 0.f;
  for (int e = tid; e < TB * 4; e += C::THREADS) ks[e >> 2][D + (e & 3)] = (e & 3) == 0 ? 1.0f : 0.0f;

  const T* kh = k + (long long)head * a.n_new * D;
  const T* vh = v + (long long)head * a.n_new * D;
  uint4 kr[NLD], vr[NLD];
  auto fetch = [&](long long t0) {   // tokens past the end read as zero: they add nothing
#pragma unroll
    for (int i = 0; i < NLD; ++i) {
      const int e = tid + i * C::THREADS;
      const bool ok = e < TB * VPT && t0 + e / VPT < a.n_new;
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
      kr[i] = ok ? __ldg(reinterpret_cast<const uint4*>(kh + t0 * D) + e) : zero;
      vr[i] = ok ? __ldg(reinterpret_cast<const uint4*>(vh + t0 * D) + e) : zero;
    }
  };
  fetch(0);
  for (long long t0 = 0; t0 < a.n_new; t0 += TB) {
    const int nt = (int)((a.n_new - t0 < TB) ? a.n_new - t0 : TB);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NLD; ++i) {
      const int e = tid + i * C::THREADS;
      if (e < TB * VPT) {
        store16_as_f32<T>(kr[i], &ks[e / VPT][(e % VPT) * EPV]);
        store16_as_f32<T>(vr[i], &vs[e / VPT][(e % VPT) * EPV]);
      }
    }
    __syncthreads();
    if (t0 + TB < a.n_new) fetch(t0 + TB);
    if (blockIdx.x == 0) {
      const int warp = tid >> 5;
      if (warp < C::THREADS / 32) {
        float m = 0.0f;
        for (int tok = warp; tok < nt; tok += C::THREADS / 32) m = fmaxf(m, warp_norm2<D>(ks[tok], lane));
        if (lane == 0) atomicMax(&s_kmax2_bits, __float_as_int(m));
      }
    }
    if (!on) continue;
#pragma unroll 2
    for (int tok = 0; tok < nt; ++tok) {
      const float4 ka = *reinterpret_cast<const float4*>(&ks[tok][a0]);
      const ulonglong2 kb = *reinterpret_cast<const ulonglong2*>(&ks[tok][b0]);
      const float4 v0 = *reinterpret_cast<const float4*>(&vs[tok][c0]), v1 = *reinterpret_cast<const float4*>(&vs[tok][c0 + 4]);
      const float kau[4] = {ka.x, ka.y, ka.z, ka.w}, vc[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
      uint64_t vv[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) vv[c] = pack2(vc[c], vc[c]);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint64_t kk = pack2(kau[u], kau[u]);
        const uint64_t t0p = mul2(kk, kb.x), t1p = mul2(kk, kb.y);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          acc[u][0][c] = fma2(t0p, vv[c], acc[u][0][c]);
          acc[u][1][c] = fma2(t1p, vv[c], acc[u][1][c]);
        }
      }
      const float ke = ks[tok][ea];
#pragma unroll
      for (int e = 0; e < C::PE; ++e) acce[e] = fmaf(ke, ks[tok][eb + e], acce[e]);
    }
  }
  __syncthreads();
  if (blockIdx.x == 0 && tid == 0) {
    hs[0] = __int_as_float(s_kmax2_bits);
    hs[1] = __int_as_float(__float_as_int(hs[1]) + (int)a.n_new);
  }
  if (!on) return;
  const int n2rows = (a.p == 2) ? D * D : 0;
  float* st = hs + kHeader;
  // the row of pair (a, b) and, off the diagonal of tiles, its mirror image; -1: a padding row of kx
  auto row_of = [&](int x, int y) -> int {
    if (y < D) return x * D + y;
    return (y == D && x <= D) ? n2rows + x : -1;
  };
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int x = a0 + u, y = b0 + i, row = row_of(x, y);
      if (row < 0 || (x == D && y < D)) continue;
      float f[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float lo, hi;
        unpack2(acc[u][i >> 1][c], lo, hi);
        f[c] = (i & 1) ? hi : lo;
      }
      float* r1 = st + (long long)row * DV + c0;
#pragma unroll
      for (int c = 0; c < 8; ++c) { f[c] += r1[c]; r1[c] = f[c]; }
      if (y < D && ta != tb) {
        float* r2 = st + (long long)(y * D + x) * DV + c0;
#pragma unroll
        for (int c = 0; c < 8; ++c) r2[c] = f[c];
      }
    }
#pragma unroll
  for (int e = 0; e < C::PE; ++e) {
    const int x = ea, y = eb + e, row = row_of(x, y);
    if (row < 0 || (x == D && y < D)) continue;
    const float f = acce[e] + st[(long long)row * DV + D];
    st[(long long)row * DV + D] = f;
    if (y < D && ta != tb) st[(long long)(y * D + x) * DV + D] = f;
  }
}

int rows_of(const fastmax_problem& p) { return 1 + p.d + (p.p == 2 ? p.d * p.d : 0); }

int check_decode(const fastmax_problem* prob) {
  int rc = check_problem(prob);
  if (rc) return rc;
  if (prob->d != 32 && prob->d != 64 && prob->d != 128)
    return fail(FASTMAX_E_ARG, "the decode state supports head dimensions 32, 64 and 128, got %d", prob->d);
  return FASTMAX_OK;
}

// CTAs per head of step_kernel: each leaves one partial row per query head in the scratch.
int step_ctas(const fastmax_problem& p) {
  if (p.d == 32) return DecCfg<32>::ctas(p.p);
  if (p.d == 64) return DecCfg<64>::ctas(p.p);
  return DecCfg<128>::ctas(p.p);
}

// From how many tokens on a prompt's kernels beat few_kernel, which reads and writes whole rows but walks the tokens
// one by one.  Measured, us, few_kernel / prompt kernel (p = 1 stays below its line on tensor cores, whose sums truncate: error
// 1.1 to 1.4 times few_kernel's at 14 to 23 tokens, for 12.4 / 10.5 at 16):
//   CUDA cores (float32, d = 32), 64 heads: d = 64, p = 2: 69 / 70 at 44 tokens; p = 1: 15.0 / 10.4 at 33, 10.4 / 10.4 at 20;
//                                 d = 128, p = 2: 462 / 391 at 44
//   fm_decode_tc.cu   d = 64, p = 2: 8 heads 12.7 / 14.7 at 16, 16.7 / 14.7 at 24; 64: 43.5 / 43.3 at 24, 49.5 / 43.3 at 28;
//                                    512: 277 / 324 at 24, 346 / 324 at 32
//                     d = 128, p = 2: 8 heads 37 / 43 at 16, 47 / 44 at 24; 64: 277 / 319 at 24, 336 / 320 at 32
long long append_min(const fastmax_problem& p) {
  const bool tc = p.dtype == FASTMAX_BF16 && p.d >= 64;
  return p.p == 1 ? 24 : (tc ? 28 : 40);
}

// From how many CTAs on a step leaves the heads' sums to sum_kernel: a CTA then ends without a fence and an atomic's way to
// memory and back, but the sums cost a kernel that starts when everything has been written, 9 to 13 us.  Measured, us a step, one
// kernel / two: d = 64 88.1 / 88.3 at 6400 CTAs (256 heads), 330 / 312 at 25600; d = 128, whose two kernels use bulk copies, 49.9
// / 48.9 (with the state out of L2 55.2 / 56.3) at 2224 (16 heads), 69.9 / 64.4 at 3336, 165.6 / 144 at 8896, 321 / 271 at
// 17792, 4 query heads each 102 / 86.7 at 4448; d = 32 17.5 / 16.7 (24.8 / 25.6) at 1024, 24.3 / 22.3 at 1600, 117 / 101 at 8192.
template <int D> constexpr long long kSharesFrom = D == 32 ? 1600 : D == 64 ? 8192 : 3072;

template <typename T, int D, bool READ>
int launch_decode(const fastmax_problem& p, const void* q, const void* k, const void* v, long long n_new,
                  float* state, float* scratch, void* out, cudaStream_t st) {
  DecArgs a{p.bh, p.bhkv, p.bhkv ? p.bh / p.bhkv : 1, p.p, p.normalize, p.a0, p.a1, p.a2, p.lim, n_new,
            kHeader + (long long)rows_of(p) * (D + 1)};
  if (p.bhkv == 0) return FASTMAX_OK;
  if (!READ && n_new >= append_min(p)) {
    if constexpr (sizeof(T) == 2 && D >= 64) {
      return decode_append_tc(p, k, v, n_new, state, st);
    } else {
      dim3 grid(AppCfg<D>::ctas(p.p), p.bhkv);
      FM_LAUNCH("fm_decode_append", st,
                (append_kernel<T, D><<<grid, AppCfg<D>::THREADS, 0, st>>>(a, (const T*)k, (const T*)v, state)));
    }
  } else {
    const dim3 grid(DecCfg<D>::ctas(p.p), p.bhkv);
    if constexpr (READ) {
      if (p.p == 2 && grid.x * (long long)p.bhkv >= kSharesFrom<D>) {
        const int smem = D == 128 ? RunCfg<D>::SMEM : 0;
        FM_CUDA_TRY(cudaFuncSetAttribute(step_kernel<T, D, SUMS_APART>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        FM_LAUNCH("fm_decode_step", st,
                  (step_kernel<T, D, SUMS_APART><<<grid, DecCfg<D>::THREADS, smem, st>>>(a, (const T*)q, (const T*)k, (const T*)v,
                                                                                   state, scratch, (T*)out)));
        FM_CUDA_TRY(cudaGetLastError());
        FM_LAUNCH("fm_decode_sum", st,
                  (sum_kernel<T, D><<<p.bh, DecCfg<D>::THREADS, 0, st>>>(a, (int)grid.x, (const T*)k, state, scratch, (T*)out)));
      } else if (grid.x == 1) {
        FM_LAUNCH("fm_decode_step", st,
                  (step_kernel<T, D, SUMS_ALONE><<<grid, DecCfg<D>::THREADS, 0, st>>>(a, (const T*)q, (const T*)k, (const T*)v, state,
                                                                                     scratch, (T*)out)));
      } else {
        FM_LAUNCH("fm_decode_step", st,
                  (step_kernel<T, D, SUMS_LAST><<<grid, DecCfg<D>::THREADS, 0, st>>>(a, (const T*)q, (const T*)k, (const T*)v, state,
                                                                                    scratch, (T*)out)));
      }
    } else
      FM_LAUNCH("fm_decode_append", st,
                (few_kernel<T, D><<<grid, DecCfg<D>::THREADS, 0, st>>>(a, (const T*)k, (const T*)v, state)));
  }
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

template <bool READ>
int dispatch_decode(const fastmax_problem& p, const void* q, const void* k, const void* v, long long n_new,
                    float* state, float* scratch, void* out, cudaStream_t st) {
#define FM_DEC(TT, DD) return launch_decode<TT, DD, READ>(p, q, k, v, n_new, state, scratch, out, st)
  if (p.dtype == FASTMAX_F32) {
    if (p.d == 32) FM_DEC(float, 32);
    if (p.d == 64) FM_DEC(float, 64);
    FM_DEC(float, 128);
  }
  if (p.d == 32) FM_DEC(__nv_bfloat16, 32);
  if (p.d == 64) FM_DEC(__nv_bfloat16, 64);
  FM_DEC(__nv_bfloat16, 128);
#undef FM_DEC
}

}  // namespace
}  // namespace fm

using namespace fm;

size_t fastmax_b200_decode_state_bytes(const fastmax_problem* prob) {
  if (!prob || prob->bhkv < 0 || prob->d <= 0) return 0;
  return sizeof(float) * (size_t)prob->bhkv * (kHeader + (size_t)rows_of(*prob) * (prob->d + 1));
}

size_t fastmax_b200_decode_scratch_bytes(const fastmax_problem* prob) {
  if (!prob || prob->bh < 0 || prob->d <= 0) return 0;
  return sizeof(float) * (size_t)prob->bh * step_ctas(*prob) * (prob->d + 1);
}

int fastmax_b200_decode_append(const fastmax_problem* prob, const void* k, const void* v, long long n_new,
                               void* state, void* stream) {
  int rc = check_decode(prob);
  if (rc) return rc;
  if (n_new < 0) return fail(FASTMAX_E_ARG, "negative token count");
  if (n_new == 0 || prob->bhkv == 0) return FASTMAX_OK;
  if (!k || !v || !state) return fail(FASTMAX_E_ARG, "NULL array");
  if (((uintptr_t)k | (uintptr_t)v) & 15) return fail(FASTMAX_E_ARG, "k and v must be 16-byte aligned");
  return dispatch_decode<false>(*prob, nullptr, k, v, n_new, (float*)state, nullptr, nullptr, (cudaStream_t)stream);
}

int fastmax_b200_decode_step(const fastmax_problem* prob, const void* q, const void* k, const void* v, void* state,
                             void* scratch, void* out, void* stream) {
  int rc = check_decode(prob);
  if (rc) return rc;
  if (prob->bh == 0) return FASTMAX_OK;
  if (!q || !k || !v || !state || !scratch || !out) return fail(FASTMAX_E_ARG, "NULL array");
  if (((uintptr_t)k | (uintptr_t)v) & 15) return fail(FASTMAX_E_ARG, "k and v must be 16-byte aligned");
  return dispatch_decode<true>(*prob, q, k, v, 1, (float*)state, (float*)scratch, out, (cudaStream_t)stream);
}

namespace fm {
int decode_step_status(int* out, cudaStream_t stream) {
  FM_CUDA_TRY(cudaMemcpyFromSymbolAsync(out, g_step_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
int decode_step_status_reset(cudaStream_t stream) {
  const int zero = 0;
  FM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_step_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
}  // namespace fm
