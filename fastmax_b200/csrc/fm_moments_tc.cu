// Chunk states of the moment-state form, second-order rows, on the tcgen05 tensor cores (bf16 operands, fp32
// accumulation), head dimension 64 (the read-out is fm_readout.cu):
//   T2[(a,b)][c] = sum_j y_j[a] y_j[b] z_j[c] over the tokens of a chunk: the features y_a y_b (each unordered pair
//   once) are formed on the CUDA cores and written to tensor memory as the A operand, the value tile is the MN-major
//   B operand delivered by TMA, and the accumulators stay in tensor memory for the whole chunk.
// The normaliser column is a second, small tensor-core kernel here; the first-order and constant rows of the state stay
// on the kernels of fm_first_tc.cu and fm_moments_ffma.cu.
#include <cstdlib>

#include "fm_common.cuh"
#include "fm_sm100.cuh"

namespace fm {

__device__ int g_mtc_status = 0;  // first protocol error seen by a kernel of this file

namespace {
using namespace sm100;

constexpr int D = 64;

__device__ __forceinline__ void report(int code) { atomicCAS(&g_mtc_status, 0, code); }
// 16 bytes from / 4 bytes to shared memory by shared-window address (keeps the access off the generic path)
__device__ __forceinline__ uint4 lds128(uint32_t saddr) {
  uint4 r;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(saddr));
  return r;
}
__device__ __forceinline__ void sts32(uint32_t saddr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(saddr), "r"(v) : "memory");
}

// =====================================================================================
// state build: T2[(a,b)][c] = sum_j y_j[a] y_j[b] z_j[c],  c < 64
// T2 is symmetric in (a, b), so each of the 2080 unordered pairs is formed once and its row is
// written to both of its places: 17 tiles of 128 pairs instead of 32 tiles of ordered ones.
// Five CTAs share one chunk of one head; four own four accumulator tiles of 128 pairs by 64
// columns (TMEM columns 0..255), the fifth one tile (see the pair table in the kernel), and each
// walks the chunk in blocks of 128 tokens.  The feature tiles are the A operand and live in
// tensor memory, never in shared memory: a TMEM lane of tile m holds its pair's product
// y[b] y[other] for the block's 128 tokens as 64 packed bf16 pairs (columns 256 + 64 m ..),
// written by the threads that own the lane, and the value tile that TMA delivered is the
// MN-major B operand of eight K=16 products per tile.
//   The sixteen generator warps form two independent halves, one per 64 tokens of the block
// (warps 0-7 and 8-15), each with its own named barrier, feature-buffer columns, mbarriers
// and MMA issuer warp, so that the latency chain of one half (transpose, barrier, row reads,
// TMEM stores, hand-off) overlaps that of the other.  A half first transposes its y rows
// into shared memory (yT[feature][token]), so that a thread reads its own row b once, as
// 16-byte vectors, and the tile's other row per tile (one row for the whole warp where the pair
// is feature x fixed feature, the warp's 32 rows rotated where it is a distance around the
// ring); warp w covers the TMEM lane quarter w % 4 and 32 tokens.  Shared-memory traffic per
// block is the transposition, the row reads and the tensor core's reads of the value tile, a
// fraction of what feature tiles staged in shared memory cost.  The y tile comes by TMA beside
// the value tile and is transposed one block ahead, between the stores of a pair of tiles and their hand-over.
//   What bounds it: the chain of a block (row reads, products, TMEM stores, hand-over) and the load/store unit, 1 500
// cycles a block for rotated rows.  Measured, 1024 heads x 8192 tokens of chunks with a state, a launch: 3.7 ms; 4.7 ms
// with the rows read from global memory by the threads that transpose them (32 lines a request kept the load/store unit
// 75-80 % busy); 3.85 ms with the transposition at the head of its own block, 4.5 ms with the second pair handed over at
// the start of the next block.
// =====================================================================================
struct StArgs {
  float* state;      // (heads, nchunk, F, DVP) fp32; rows a*64+b and b*64+a of each pair, columns 0..64 and padding
  int n, chunk, nchunk, dvp;
  size_t per_state;
  int skip_chunk;    // this chunk's state is not wanted (-1: none)
  int lower;         // only rows (b, a) with a / 16 <= b / 16 are wanted: all that the read-out's copies are made from
};

constexpr int ST_GEN_WARPS = 16;
constexpr int ST_THREADS = (ST_GEN_WARPS + 3) * 32;   // warps 0-15: generators; 16: TMA; 17, 18: MMA issuers
constexpr int ST_TILES = 4;           // accumulator tiles (and feature buffers) per CTA
constexpr int ST_SPLIT = 5;            // CTAs per (head, chunk): four of four tiles and one of one tile
constexpr int ST_NZ = 3;              // ring of value and feature tiles
constexpr int ST_ZTILE = 128 * 128;
constexpr int ST_STAGE = 2 * ST_ZTILE;  // z tile, y tile
constexpr int ST_YT_LD = 272;         // bytes per yT row: 128 tokens + 16 (conflict-free 16-byte reads down a column)
constexpr int ST_YT = 64 * ST_YT_LD;
constexpr int ST_OFF_Z = 0;
constexpr int ST_OFF_YT = ST_NZ * ST_STAGE;          // two transposed blocks
constexpr int ST_OFF_BAR = ST_OFF_YT + 2 * ST_YT;
constexpr int ST_NBAR = 5 * ST_TILES + 2 * ST_NZ + 1;
constexpr int ST_OFF_TMEM = ST_OFF_BAR + ST_NBAR * 8;
constexpr int ST_SMEM = ST_OFF_TMEM + 16 + 1024;
constexpr int ST_TM_A = 64 * ST_TILES;               // first TMEM column of the feature buffers
static_assert(ST_TILES == 4 && ST_GEN_WARPS == 16, "the epilogue gives one tile to each group of four warps");

__global__ void __launch_bounds__(ST_THREADS, 1)
state_tc_kernel(const __grid_constant__ CUtensorMap tmZ, const __grid_constant__ CUtensorMap tmY, const StArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + ST_OFF_BAR;
  // barriers: a_full[tile][half] | a_empty[tile][half] | z_full[NZ] | z_empty[NZ] | done
  auto BAR_AFULL = [&](int m, int h) { return bar0 + 8u * (2 * m + h); };
  auto BAR_AEMPTY = [&](int m, int h) { return bar0 + 8u * (2 * ST_TILES + 2 * m + h); };
  auto BAR_ZFULL = [&](int s) { return bar0 + 8u * (4 * ST_TILES + s); };
  auto BAR_ZEMPTY = [&](int s) { return bar0 + 8u * (4 * ST_TILES + ST_NZ + s); };
  auto BAR_DONE = [&]() { return bar0 + 8u * (4 * ST_TILES + 2 * ST_NZ); };
  // completes once, when half 0's first product of tile m is done (a_empty[m][0] completes every block, and a
  // late waiter on one parity of it could see two completions as none)
  auto BAR_START = [&](int m) { return bar0 + 8u * (4 * ST_TILES + 2 * ST_NZ + 1 + m); };
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + ST_OFF_TMEM);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int part = blockIdx.x % ST_SPLIT;
  const int hc = blockIdx.x / ST_SPLIT;           // head * nchunk + chunk
  const int head = hc / a.nchunk, chunk = hc % a.nchunk;
  if (chunk == a.skip_chunk) return;
  const int t_begin = chunk * a.chunk, t_end = min(a.n, t_begin + a.chunk);
  const int nblk = (t_end - t_begin + 127) / 128;
  const int ntile = part == 4 ? 1 : ST_TILES;

  if (tid == 0) {
    for (int m = 0; m < ST_TILES; ++m)
      for (int h = 0; h < 2; ++h) { mbar_init(BAR_AFULL(m, h), ST_GEN_WARPS / 2); mbar_init(BAR_AEMPTY(m, h), 1); }
    for (int m = 0; m < ST_TILES; ++m) mbar_init(BAR_START(m), 1);
    for (int s = 0; s < ST_NZ; ++s) { mbar_init(BAR_ZFULL(s), 1); mbar_init(BAR_ZEMPTY(s), 2 + ST_GEN_WARPS); }
    mbar_init(BAR_DONE(), 2);
    mbar_fence_init();
  }
  if (warp == ST_GEN_WARPS + 1) tmem_alloc(smem_u32((const void*)tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == ST_GEN_WARPS) {
    // ---- producer: value and feature tiles by TMA ----
    if (lane == 0) { tma_prefetch_desc(&tmZ); tma_prefetch_desc(&tmY); }
    for (int k = 0; k < nblk; ++k) {
      const int s = k % ST_NZ;
      if (!mbar_wait(BAR_ZEMPTY(s), (((k / ST_NZ) & 1) ^ 1))) { report(31); break; }
      if (lane == 0) {
        mbar_expect_tx(BAR_ZFULL(s), ST_STAGE);
        // rows past the end of the sequence are zero-filled; chunks are whole multiples of 128 tokens
        tma_load_3d(sbase + ST_OFF_Z + s * ST_STAGE, &tmZ, BAR_ZFULL(s), 0, t_begin + k * 128, head);
        tma_load_3d(sbase + ST_OFF_Z + s * ST_STAGE + ST_ZTILE, &tmY, BAR_ZFULL(s), 0, t_begin + k * 128, head);
      }
    }
  } else if (warp > ST_GEN_WARPS) {
    // Issuer warp w serves token half w of every block: the whole warp runs the loop, one elected
    // lane issues four K=16 products per tile.  Both halves add into the same accumulators; in the
    // first block half 1 lets half 0's product of a tile complete first, because that one starts
    // the accumulator.
    const int w = warp - ST_GEN_WARPS - 1;
    constexpr uint32_t idesc = idesc_bf16(128, 64, 0, 1);
    bool ok = true;
    for (int k = 0; ok && k < nblk; ++k) {
      const int s = k % ST_NZ;
      if (!mbar_wait_warp(BAR_ZFULL(s), (uint32_t)((k / ST_NZ) & 1))) { report(32); ok = false; break; }
      const uint32_t z_lo = desc_lo(sbase + ST_OFF_Z + s * ST_STAGE, ST_ZTILE) + (uint32_t)w * (4 * 128);
      if (ntile == 1) {
        // one tile: its four feature buffers are a ring over blocks, so that the threads that form the
        // features run ahead of the products instead of waiting for each one
        const int fb = k & 3;
        if (!mbar_wait_warp(BAR_AFULL(fb, w), (uint32_t)((k >> 2) & 1))) { report(33); ok = false; break; }
        if (k == 0 && w == 1 && !mbar_wait_warp(BAR_START(0), 0)) { report(36); ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          umma_ts_steps<4>(tmem, tmem + ST_TM_A + fb * 64 + w * 32, z_lo, idesc, (k > 0 || w == 1) ? 1u : 0u);
          umma_commit(BAR_AEMPTY(fb, w));
          if (k == 0 && w == 0) umma_commit(BAR_START(0));
        }
        __syncwarp();
      } else
      for (int m = 0; m < ntile; ++m) {
        if (!mbar_wait_warp(BAR_AFULL(m, w), (uint32_t)(k & 1))) { report(33); ok = false; break; }
        if (k == 0 && w == 1 && !mbar_wait_warp(BAR_START(m), 0)) { report(36); ok = false; break; }
        tc_fence_after();
        if (elect_one()) {
          umma_ts_steps<4>(tmem + m * 64, tmem + ST_TM_A + m * 64 + w * 32, z_lo, idesc, (k > 0 || w == 1) ? 1u : 0u);
          umma_commit(BAR_AEMPTY(m, w));
          if (k == 0 && w == 0) umma_commit(BAR_START(m));
        }
        __syncwarp();
      }
      if (ok && elect_one()) umma_commit(BAR_ZEMPTY(s));
      __syncwarp();
    }
    if (ok && elect_one()) umma_commit(BAR_DONE());
    __syncwarp();
  } else {
    const int h = warp >> 3, tq = (warp >> 2) & 1, qd = warp & 3;   // token half, 32-token quarter in it, TMEM lane quarter
    // This thread's lane of tile m holds the unordered pair {b, other(m)}: b is the thread's own feature
    // (the same in every tile, so its row is read once per block), other(m) the tile's.
    //   part 0: b = lane,      other = (lane + s) % 32,      s = 4 m + quarter = 0..15   (pairs inside features 0..31)
    //   part 1: b = 32 + lane, other = 4 m + quarter                                     (features 32..63 x 0..15)
    //   part 2: b = 32 + lane, other = 16 + 4 m + quarter                                (features 32..63 x 16..31)
    //   part 3: b = 32 + lane, other = 32 + (lane + s) % 32                              (pairs inside 32..63)
    //   part 4: one tile; quarter 0: b = lane, quarter 1: b = 32 + lane, other = b's partner at distance 16, of
    //           which lanes 0..15 are new pairs; quarters 2 and 3 repeat them and are not stored.
    // Distances 0..15 around the ring of 32 give every pair inside a group of 32 once, distance 16 gives the
    // remaining sixteen; 2080 pairs in 17 tiles of 128 lanes instead of 4096 ordered ones in 32.
    const int grp = part == 0 ? 0 : (part < 4 ? 1 : (qd & 1));
    const int b = grp * 32 + lane;
    const int o_off = (part == 3 || part == 4) ? grp * 32 : 0;
    const int o_sum = ((part == 1 || part == 2) ? 0 : lane) + (part == 4 ? 16 : (part == 2 ? 16 + qd : qd));
    auto other = [&](int m) { return o_off + ((o_sum + 4 * m) & 31); };
    const int tok_off = h * 64 + tq * 32;           // first of this warp's 32 tokens in the block
    // transposition duty inside the half: token pair jp (of 32) and 8 features from fg * 8
    const int jp = tid & 31, fg = (tid >> 5) & 7;
    // Its two rows of block k, 16 bytes each, from the y tile.  The lanes of every other group of four read the odd row
    // first: eight neighbouring lanes then meet eight different rows modulo 8, so eight different 16-byte banks.
    const uint32_t swap = (uint32_t)(jp >> 2) & 1;
    bool ok = true;
    uint4 rows[2];
    auto load_rows = [&](int k) {
      if (k >= nblk || !ok) return;
      const int s = k % ST_NZ;
      if (!mbar_wait(BAR_ZFULL(s), (uint32_t)((k / ST_NZ) & 1))) { report(37); ok = false; return; }
      const uint32_t r0 = h * 64 + 2 * jp + swap, r1 = r0 ^ 1;
      const uint32_t tile = sbase + ST_OFF_Z + s * ST_STAGE + ST_ZTILE;
      rows[0] = lds128(tile + r0 * 128 + ((fg ^ (r0 & 7)) << 4));
      rows[1] = lds128(tile + r1 * 128 + ((fg ^ (r1 & 7)) << 4));
    };
    // ... and into yT: word (feature f, token pair) = two consecutive tokens of feature f
    auto transpose = [&](int k) {
      if (k >= nblk) return;
      const uint4 even = swap ? rows[1] : rows[0], odd = swap ? rows[0] : rows[1];
      const uint32_t t0[4] = {even.x, even.y, even.z, even.w};
      const uint32_t t1[4] = {odd.x, odd.y, odd.z, odd.w};
      const uint32_t col = sbase + ST_OFF_YT + (k & 1) * ST_YT + (fg * 8) * ST_YT_LD + (h * 32 + jp) * 4;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        sts32(col + (2 * e) * ST_YT_LD, __byte_perm(t0[e], t1[e], 0x5410));
        sts32(col + (2 * e + 1) * ST_YT_LD, __byte_perm(t0[e], t1[e], 0x7632));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_ZEMPTY(k % ST_NZ));   // the y tile has been read
    };
    // the warp's stores to feature buffers m0 and m1 are complete: hand them over
    auto hand_over = [&](int m0, int m1) {
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(BAR_AFULL(m0, h));
        if (m1 >= 0) mbar_arrive(BAR_AFULL(m1, h));
      }
    };
    load_rows(0);
    transpose(0);
    const uint32_t ta = tmem + ST_TM_A + h * 32 + tq * 16 + ((uint32_t)(qd * 32) << 16);   // this warp's part of feature buffer 0
    for (int k = 0; k < nblk; ++k) {   // every generator thread takes part in every block's barrier
      const uint32_t yt = sbase + ST_OFF_YT + (k & 1) * ST_YT;
      if (h == 0) asm volatile("bar.sync 1, 256;" ::: "memory");
      else asm volatile("bar.sync 2, 256;" ::: "memory");
      // Block k is transposed, and every thread of the half is done with its reads of block k - 1: its buffer takes block
      // k + 1 below, while the products of block k are formed (a half reads only the token columns it wrote).
      load_rows(k + 1);
      if (!ok) continue;
      uint32_t yb[16];
      {
        const uint32_t rb = yt + b * ST_YT_LD + tok_off * 2;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const uint4 w4 = lds128(rb + v * 16);
          yb[4 * v] = w4.x; yb[4 * v + 1] = w4.y; yb[4 * v + 2] = w4.z; yb[4 * v + 3] = w4.w;
        }
      }
      // products of one tile: row a of the tile (a broadcast read) times this thread's row b
      auto products = [&](int m, uint32_t (&pr)[16]) {
        const uint32_t ra = yt + other(m) * ST_YT_LD + tok_off * 2;
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const uint4 w4 = lds128(ra + v * 16);
          const uint32_t ya[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const __nv_bfloat162 pv = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&yb[4 * v + e]),
                                              *reinterpret_cast<const __nv_bfloat162*>(&ya[e]));
            pr[4 * v + e] = *reinterpret_cast<const uint32_t*>(&pv);
          }
        }
      };
      // Tiles go two at a time, and the stores of one pair complete while the products of the next
      // are formed.  A feature buffer is free once the product that read it one block ago is done;
      // products complete in order, so the later tile's barrier covers the earlier one's too.
      uint32_t p0[16], p1[16], p2[16], p3[16];
      products(0, p0);
      if (ntile == 1) {
        const int fb = k & 3;                       // feature buffer of this block (a ring over blocks)
        if (!mbar_wait(BAR_AEMPTY(fb, h), (uint32_t)(((k >> 2) & 1) ^ 1))) { report(34); ok = false; continue; }
        tc_fence_after();
        tmem_st16(ta + 64 * fb, p0);
        transpose(k + 1);
        hand_over(fb, -1);
        continue;
      }
      products(1, p1);
      if (!mbar_wait(BAR_AEMPTY(1, h), (uint32_t)((k & 1) ^ 1))) { report(34); ok = false; continue; }
      tc_fence_after();
      tmem_st16(ta, p0);
      tmem_st16(ta + 64, p1);
      transpose(k + 1);
      products(2, p2);
      products(3, p3);
      hand_over(0, 1);
      if (!mbar_wait(BAR_AEMPTY(3, h), (uint32_t)((k & 1) ^ 1))) { report(34); ok = false; continue; }
      tc_fence_after();
      tmem_st16(ta + 128, p2);
      tmem_st16(ta + 192, p3);
      hand_over(2, 3);
    }
    // ---- epilogue: accumulator rows -> fp32 state (columns 0..63), the normaliser column from the
    // block state_ecol_tc_kernel left in the first-order rows, zero padding ----
    float* st = a.state + (size_t)hc * a.per_state;
    const int m = warp >> 2;                       // one tile per group of four warps
    const int o = other(m);
    const bool warp_mine = m < ntile && (part < 4 || qd < 2);   // the TMEM read is a whole-warp instruction
    const bool mine = warp_mine && (part < 4 || lane < 16);
    // column 64 of the pair's two rows (65..67 are padding, dvp == 68), asked for before the wait for the products
    uint32_t ecols[2] = {0u, 0u};
    if (ok && mine) {
      ecols[0] = __float_as_uint(st[(size_t)4096 * a.dvp + b * 64 + o]);
      ecols[1] = __float_as_uint(st[(size_t)4096 * a.dvp + o * 64 + b]);
    }
    if (ok && !mbar_wait(BAR_DONE(), 0)) { report(35); ok = false; }
    tc_fence_after();
    if (ok) {
      uint32_t tv[64];
      if (warp_mine) {
        tmem_ld64(tmem + m * 64 + ((uint32_t)(qd * 32) << 16), tv);
        tmem_wait_ld(tv);
      }
      // the pair's row goes to both of its places in the state, (b, other) and (other, b), or to those that are read
      for (int side = 0; mine && side < (o == b ? 1 : 2); ++side) {
      if (a.lower && (side == 0 ? (o >> 4) > (b >> 4) : (b >> 4) > (o >> 4))) continue;
      const int f = side == 0 ? b * 64 + o : o * 64 + b;
      float* dst = st + (size_t)f * a.dvp;
      const uint32_t ecol = ecols[side];
      // A thread owns its 272-byte row, so its stores share no sector with its neighbours': 32-byte stores
      // (whole sectors) wherever the row allows.  A row that starts on a 32-byte boundary is 8 x 32 + 16
      // bytes, one that starts 16 bytes past a boundary is 16 + 8 x 32 (rows and matrices are 16-byte multiples).
      if (((uintptr_t)dst & 16) != 0) {
        *(float4*)dst = make_float4(__uint_as_float(tv[0]), __uint_as_float(tv[1]), __uint_as_float(tv[2]),
                                    __uint_as_float(tv[3]));
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          uint32_t w[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            const int col = 4 + 8 * e + q;
            w[q] = col < 64 ? tv[col < 64 ? col : 0] : (col == 64 ? ecol : 0u);
          }
          stg32(dst + 4 + 8 * e, w, true);
        }
      } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          uint32_t w[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) w[q] = tv[8 * e + q];
          stg32(dst + 8 * e, w, true);
        }
        *(float4*)(dst + 64) = make_float4(__uint_as_float(ecol), 0.f, 0.f, 0.f);
      }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == ST_GEN_WARPS + 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Normaliser column of the second-order rows on the tensor cores:
//   state[(a,b)][64] = E[a][b] = sum_j e_j y_j[a] y_j[b] = (Y^T (e o Y))[a][b]   (e = 1, or -dvec)
// One CTA per (head, chunk).  A 128-token tile of y, as TMA delivers it, is at once the MN-major A
// operand (features along M) and -- when e = 1 -- the MN-major B operand; with e = -dvec four warps
// write the scaled rows e_j y_j (rounded to bf16 once, from the fp32 product) into a second tile
// with the same swizzled offsets.  An M = 128 operand has two 64-wide blocks; the second one is
// simply the 16 KB that follow the tile in shared memory (the next ring stage, or the first scaled
// tile after the last stage), so TMEM lanes 64..127 receive products of whatever lies there and are
// never read; lane a < 64, column b of the accumulator is E[a][b].  The result is left as a dense
// 64 x 64 block in the state matrix's own first-order rows (4096.. of 4161, 17.7 KB), which nothing has
// written yet: state_tc_kernel, next on the stream, copies E[a][b] into column 64 of the row (a, b) it
// writes anyway (4-byte stores scattered over 4096 rows cost more than the whole product), and the
// first-order state kernels then overwrite the block with the real rows.
constexpr int EC_THREADS = 192;       // warps 0-3: scaled copy and epilogue; 4: TMA; 5: MMA issuer
constexpr int EC_NS = 4;              // y-tile ring
constexpr int EC_STAGE = ST_ZTILE;
constexpr int EC_OFF_B = EC_NS * EC_STAGE;           // two scaled tiles
constexpr int EC_OFF_BAR = EC_OFF_B + 2 * ST_ZTILE;
constexpr int EC_NBAR = 2 * EC_NS + 4 + 1;
constexpr int EC_OFF_TMEM = EC_OFF_BAR + EC_NBAR * 8;
constexpr int EC_SMEM = EC_OFF_TMEM + 16 + 1024;

__global__ void __launch_bounds__(EC_THREADS, 2)
state_ecol_tc_kernel(const __grid_constant__ CUtensorMap tmY, const float* __restrict__ dvec,
                     float* __restrict__ state, int n, int chunk, int nchunk, int dvp, size_t per_state,
                     int skip_chunk) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + EC_OFF_BAR;
  // barriers: y_full[NS] | y_empty[NS] | b_full[2] | b_empty[2] | done
  auto BAR_YFULL = [&](int s) { return bar0 + 8u * s; };
  auto BAR_YEMPTY = [&](int s) { return bar0 + 8u * (EC_NS + s); };
  auto BAR_BFULL = [&](int b) { return bar0 + 8u * (2 * EC_NS + b); };
  auto BAR_BEMPTY = [&](int b) { return bar0 + 8u * (2 * EC_NS + 2 + b); };
  const uint32_t BAR_DONE = bar0 + 8u * (2 * EC_NS + 4);
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + EC_OFF_TMEM);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hc = blockIdx.x, head = hc / nchunk, ck = hc % nchunk;
  if (ck == skip_chunk) return;
  const int t_begin = ck * chunk, t_end = min(n, t_begin + chunk);
  const int nblk = (t_end - t_begin + 127) / 128;
  const bool scaled = dvec != nullptr;

  if (tid == 0) {
    for (int s = 0; s < EC_NS; ++s) { mbar_init(BAR_YFULL(s), 1); mbar_init(BAR_YEMPTY(s), 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(BAR_BFULL(b), 4); mbar_init(BAR_BEMPTY(b), 1); }
    mbar_init(BAR_DONE, 1);
    mbar_fence_init();
  }
  if (warp == 5) tmem_alloc(smem_u32((const void*)tmem_slot), 64);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 4) {
    if (lane == 0) tma_prefetch_desc(&tmY);
    for (int k = 0; k < nblk; ++k) {
      const int s = k % EC_NS;
      if (!mbar_wait(BAR_YEMPTY(s), (((k / EC_NS) & 1) ^ 1))) { report(41); break; }
      if (lane == 0) {
        mbar_expect_tx(BAR_YFULL(s), EC_STAGE);
        // rows past the end of the sequence are zero-filled; chunks are whole multiples of 128 tokens
        tma_load_3d(sbase + s * EC_STAGE, &tmY, BAR_YFULL(s), 0, t_begin + k * 128, head);
      }
    }
  } else if (warp == 5) {
    constexpr uint32_t idesc = idesc_bf16(128, 64, 1, 1);
    bool ok = true;
    for (int k = 0; ok && k < nblk; ++k) {
      const int s = k % EC_NS, bb = k & 1;
      if (!mbar_wait_warp(BAR_YFULL(s), (uint32_t)((k / EC_NS) & 1))) { report(42); ok = false; break; }
      if (scaled && !mbar_wait_warp(BAR_BFULL(bb), (uint32_t)((k >> 1) & 1))) { report(43); ok = false; break; }
      tc_fence_after();
      if (elect_one()) {
        const uint32_t a_lo = desc_lo(sbase + s * EC_STAGE, ST_ZTILE);
        const uint32_t b_lo = scaled ? desc_lo(sbase + EC_OFF_B + bb * ST_ZTILE, ST_ZTILE) : a_lo;
        umma_ss_mn_steps<8>(tmem, a_lo, b_lo, idesc, k > 0 ? 1u : 0u);
        umma_commit(BAR_YEMPTY(s));
        if (scaled) umma_commit(BAR_BEMPTY(bb));
      }
      __syncwarp();
    }
    if (ok && elect_one()) umma_commit(BAR_DONE);
    __syncwarp();
  } else {
    bool ok = true;
    if (scaled) {
      // thread j owns token row j of the block: the eight 16-byte pieces of the row keep their
      // (swizzled) offsets, so the copy never has to know which piece is which.  Rows are 128 bytes apart, so neighbouring
      // lanes begin at different pieces (32 heads of 32768: 101 us when all began at the first, on the same banks, 50 now).
      for (int k = 0; ok && k < nblk; ++k) {
        const int s = k % EC_NS, bb = k & 1;
        const int tok = t_begin + k * 128 + tid;
        const float e = (tok < t_end) ? -__ldg(dvec + (size_t)head * n + tok) : 0.f;
        if (!mbar_wait(BAR_YFULL(s), (uint32_t)((k / EC_NS) & 1))) { report(44); ok = false; break; }
        if (!mbar_wait(BAR_BEMPTY(bb), (uint32_t)(((k >> 1) & 1) ^ 1))) { report(45); ok = false; break; }
        const uint32_t src = sbase + s * EC_STAGE + tid * 128, dst = sbase + EC_OFF_B + bb * ST_ZTILE + tid * 128;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t piece = ((c + lane) & 7) * 16;
          const uint4 w = lds128(src + piece);
          const uint32_t in[4] = {w.x, w.y, w.z, w.w};
          uint32_t o[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            o[q] = pack_bf16(e * __uint_as_float(in[q] << 16), e * __uint_as_float(in[q] & 0xFFFF0000u));
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + piece), "r"(o[0]), "r"(o[1]), "r"(o[2]),
                       "r"(o[3]) : "memory");
        }
        fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR_BFULL(bb));
      }
    }
    if (ok && !mbar_wait(BAR_DONE, 0)) { report(46); ok = false; }
    tc_fence_after();
    if (ok && warp < 2) {
      uint32_t tv[64];
      tmem_ld64(tmem + ((uint32_t)(warp * 32) << 16), tv);
      tmem_wait_ld(tv);
      // E[a][0..63] as one contiguous row of the scratch block (see the header comment)
      float4* row = (float4*)(state + (size_t)hc * per_state + (size_t)4096 * dvp + (size_t)(warp * 32 + lane) * 64);
#pragma unroll
      for (int e = 0; e < 16; ++e)
        row[e] = make_float4(__uint_as_float(tv[4 * e]), __uint_as_float(tv[4 * e + 1]),
                             __uint_as_float(tv[4 * e + 2]), __uint_as_float(tv[4 * e + 3]));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem, 64);
  }
}

typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                             const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                             CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                             CUtensorMapFloatOOBfill);
EncodeFn encode_fn() {
  static EncodeFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return (EncodeFn)p;
  }();
  return fn;
}
// (mats, rows, 64) bf16 as a rank-3 map with boxes of 128 x 64, 128-byte swizzle
int make_map(CUtensorMap* m, const void* base, size_t mats, size_t rows) {
  EncodeFn enc = encode_fn();
  if (!enc) return fail(FASTMAX_E_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t gdim[3] = {64, (cuuint64_t)rows, (cuuint64_t)mats};
  cuuint64_t gstr[2] = {128, (cuuint64_t)rows * 128};
  cuuint32_t box[3] = {64, 128, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), gdim, gstr, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(FASTMAX_E_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
  return FASTMAX_OK;
}

}  // namespace

int moments_tc_status(int* out, cudaStream_t stream) {
  FM_CUDA_TRY(cudaMemcpyFromSymbolAsync(out, g_mtc_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
int moments_tc_status_reset(cudaStream_t stream) {
  const int zero = 0;
  FM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_mtc_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}

// impl == FASTMAX_IMPL_MOMENTS_FFMA, or FASTMAX_B200_NO_TC_MOMENTS=1 in the environment, keeps the
// moment family on the CUDA-core kernels (used by the tests to compare the two implementations of
// the same stages).
bool moments_tc_supports(const fastmax_problem& p) {
  static const bool off = [] {
    const char* e = getenv("FASTMAX_B200_NO_TC_MOMENTS");
    return e && e[0] == '1';
  }();
  return !off && p.impl != FASTMAX_IMPL_MOMENTS_FFMA && p.dtype == FASTMAX_BF16 && p.d == 64 && p.p == 2 && p.bh == p.bhkv;
}

// Second-order rows of the chunk states of (y, z | e) on the tensor cores: columns 0..63 by
// state_tc_kernel, the e column (e = 1 when dvec is null, else -dvec) by state_ecol_tc_kernel.
// The first-order and constant rows are NOT valid afterwards (they held the e column's scratch
// block): the caller builds them next, with first_tc_chunk_state or moments_chunk_state's p = 1
// row range, both of which write every element of those rows.
int moments_tc_chunk_state(const Ctx& c, int heads, int n, int chunk, const void* y, const void* z,
                           const float* dvec, float* state) {
  if (heads == 0 || n == 0) return FASTMAX_OK;
  const MomentDims m = moment_dims(64);
  const int nchunk = (n + chunk - 1) / chunk;
  CUtensorMap tz;
  int rc;
  if ((rc = make_map(&tz, z, heads, n))) return rc;
  StArgs a;
  a.state = state; a.n = n; a.chunk = chunk; a.nchunk = nchunk; a.dvp = m.dvp;
  a.per_state = (size_t)m.f * m.dvp;
  a.skip_chunk = c.skip_chunk;
  a.lower = c.lower_rows ? 1 : 0;
  // the normaliser column first: the state kernel picks it up in its epilogue
  CUtensorMap ty;
  if ((rc = make_map(&ty, y, heads, n))) return rc;
  FM_CUDA_TRY(cudaFuncSetAttribute(state_ecol_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, EC_SMEM));
  FM_LAUNCH("fm_moments_state_ecol", c.stream,
            (state_ecol_tc_kernel<<<(unsigned)((size_t)heads * nchunk), EC_THREADS, EC_SMEM, c.stream>>>(
                ty, dvec, state, n, chunk, nchunk, m.dvp, a.per_state, a.skip_chunk)));
  FM_CUDA_TRY(cudaGetLastError());
  FM_CUDA_TRY(cudaFuncSetAttribute(state_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_SMEM));
  FM_LAUNCH("fm_moments_tc_state", c.stream,
            (state_tc_kernel<<<(unsigned)((size_t)heads * nchunk * ST_SPLIT), ST_THREADS, ST_SMEM, c.stream>>>(tz, ty, a)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

}  // namespace fm
