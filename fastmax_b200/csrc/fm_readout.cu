// Read-out of second-order prefix states on the tcgen05 tensor cores (bf16 operands, fp32 accumulation), head
// dimension 64, and the bf16 operand copies of the states it multiplies.
//
// For a token x and the prefix state S2[a][b][c] (symmetric in a, b; c = 0..63 value columns, c = 64 the normaliser
// column E), with S1 and S0 the first-order and constant rows:
//   type A:  r[c] = a2 sum_ab x_a x_b S2[a][b][c] + a1 sum_a x_a S1[a][c] + a0 S0[c]      (numerator | denominator, grad_v)
//   type B:  r[a] = 2 a2 sum_b x_b sum_c ut_c S2[a][b][c] + a1 sum_c ut_c S1[a][c]         (grad_q, grad_k)
// with ut = [u | e].  Both contract one index on the tensor cores and the other on the CUDA cores in fp32, straight from
// tensor memory.  Both use the symmetry, each in the way its order of contraction allows:
//   type A contracts a first, T[(b, c)] = sum_a x_a S'[a][b][c], where S' keeps the blocks of 16 features a with
//     block(a) <= block(b), doubled above the diagonal: 10 of 16 K steps (16, 32, 48 or 64 deep by the block of b);
//   type B contracts c first, M[(a, b)] = sum_c u_c S2[a][b][c], for the unordered pairs only: 36 blocks of 8 x 8
//     features instead of 64, and each M enters both r_a and r_b.
// Both are persistent: one CTA per SM walks groups of 256 tokens, and the barriers and rings run on from one group to the
// next.  What bounds them: type A needs 84 K steps of 128 x 128 x 16 per 128 tokens (5 400 cycles) and 2 080 packed FMAs
// per thread, whose three 64-bit operands cost the register file 2.7 cycles and more instead of 2 (5 700 of its
// scheduler's cycles); type B 76 steps (4 900) and 2 080 FMAs.  Measured for 1024 heads x 7 952 tokens read out: type A
// 3.9 ms, type B 3.2 ms a launch (17 000 and 14 000 cycles per 128 tokens), 14.0 ms for the four of a training step, where a
// kernel with all ordered pairs, a CTA per group and no walk took 20.9 ms for its three (A, B and both on shared T).  Without its FMAs type A takes 0.82 of
// that, without its products 0.78, without either 0.56: the hand-offs of the two T buffers.  Tried and slower: T read
// 64 columns at a time one read ahead (type A 4.3 ms), an issuer warp per buffer (4.6 and 4.5), polling instead of
// suspended waits (no change).
// (Replaces the d*d-wide feature contraction of the reference, `old stuff/fastmax_cuda_forward_quad.cu`:111-135, 240-268
// and the matching backward loops.)
#include "fm_readout.cuh"

namespace fm {

__device__ int g_readout_status = 0;  // first protocol error seen by a kernel of this file

namespace {
using namespace rdo;

__device__ __forceinline__ void report(int code) { atomicCAS(&g_readout_status, 0, code); }

// ---- operand copies of one state ---------------------------------------------------------------------------
// Type B: 19 slices of 128 rows with c along K (128-byte swizzle).  Slices 0..17 hold two 8 x 8 blocks (alpha <= beta)
// of pairs each, block beta (beta + 1) / 2 + alpha; slice 18 has S1 (row a, c along K) and E (row a, b along K).
// Rows of a block are ordered for packed arithmetic: two neighbouring columns of M are the pairs (2i, 2k), (2i+1, 2k+1)
// or (2i+1, 2k), (2i, 2k+1), so that a packed FMA meets two neighbouring features of a and two of b.
constexpr int B_SLICES = 19;
constexpr int B_BYTES = B_SLICES * TILE;
__host__ __device__ constexpr int b_col(int a8, int b8) {
  return (((a8 >> 1) * 4 + (b8 >> 1)) * 2 + ((a8 ^ b8) & 1)) * 2 + (b8 & 1);
}
// The 64 x 65 block S2[a][b][:] of feature b (rows a < 16 (b / 16 + 1) are enough) -> its places in the copies, 16 bytes
// a thread: a warp writes 128-byte runs in both layouts.
__device__ __forceinline__ void write_feature(const float (*blk)[BLK_LD], int b, char* ca, char* cb, int t) {
  const int bb = b >> 4, warp = t >> 5, lane = t & 31;
  if (ca)
    for (int i = warp; i < 4 * (bb + 1); i += 8) {      // eight features a, one half of the value columns
      const int oct = i >> 1, c = (i & 1) * 32 + lane;
      const float f = (oct >> 1) < bb ? 2.f : 1.f;
      float v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = f * blk[oct * 8 + e][c];
      *(uint4*)(ca + a_slice(c >> 4, b >> 3) + (oct >> 1) * 4096 + (oct & 1) * 2048 + ((c >> 3) & 1) * 1024 + (b & 7) * 128 +
                (c & 7) * 16) =
          make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
    }
  if (cb) {
    const int beta = b >> 3;
    for (int a = t >> 3; a < 8 * (beta + 1); a += 32) { // a row of 64 value columns by eight threads
      const int w = t & 7;
      const int kb = beta * (beta + 1) / 2 + (a >> 3), row = (kb & 1) * 64 + b_col(a & 7, b & 7);
      const float4 v0 = *(const float4*)&blk[a][8 * w], v1 = *(const float4*)&blk[a][8 * w + 4];
      *(uint4*)(cb + (kb >> 1) * TILE + swz(row, w * 16)) =
          make_uint4(pack_bf16(v0.x, v0.y), pack_bf16(v0.z, v0.w), pack_bf16(v1.x, v1.y), pack_bf16(v1.z, v1.w));
    }
  }
  if (t < 16 * (bb + 1)) {
    // the normaliser column: its mirror image stands in for the rows that are not read
    const __nv_bfloat16 e = __float2bfloat16_rn(blk[t][64]);
    char* const dst[2] = {ca, cb ? cb + 18 * TILE : nullptr};
#pragma unroll
    for (int k = 0; k < 2; ++k)
      if (dst[k]) {
        *(__nv_bfloat16*)(dst[k] + swz(64 + b, t * 2)) = e;
        if ((t >> 4) < bb) *(__nv_bfloat16*)(dst[k] + swz(64 + t, b * 2)) = e;
      }
  }
}
// first-order rows (already summed) of one fp32 state
__device__ __forceinline__ void write_first(const float* __restrict__ st, float (*blk)[BLK_LD], int dvp, char* ca, char* cb,
                                            int t) {
  const float* src = st + (size_t)64 * 64 * dvp;
  for (int i = t; i < 64 * dvp; i += 256) (&blk[0][0])[i] = src[i];      // dvp == BLK_LD
  __syncthreads();
  for (int i = t; i < 64 * 32; i += 256) {
    const int r = i >> 5, w = i & 31;
    if (ca) *(uint32_t*)(ca + swz(r, w * 4)) = pack_bf16(blk[2 * w][r], blk[2 * w + 1][r]);
    if (cb) *(uint32_t*)(cb + 18 * TILE + swz(r, w * 4)) = pack_bf16(blk[r][2 * w], blk[r][2 * w + 1]);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(256) copies_kernel(const float* __restrict__ state, char* __restrict__ ca,
                                                     char* __restrict__ cb, int dvp, size_t per_state) {
  __shared__ __align__(16) float blk[64][BLK_LD];
  const int m = blockIdx.y, b = blockIdx.x, t = threadIdx.x;
  const float* st = state + (size_t)m * per_state;
  char* da = ca ? ca + (size_t)m * A_BYTES : nullptr;
  char* db = cb ? cb + (size_t)m * B_BYTES : nullptr;
  if (b == 64) { write_first(st, blk, dvp, da, db, t); return; }
  const float* src = st + (size_t)b * 64 * dvp;      // rows (b, a)
  const int na = 16 * ((b >> 4) + 1);
  for (int i = t; i < na * dvp; i += 256) (&blk[0][0])[i] = src[i];        // dvp == BLK_LD
  __syncthreads();
  write_feature(blk, b, da, db, t);
}

// Running sum over the chunks of a head and the copies in one pass, second-order rows only: the copies of chunk m get
// base + the sum of the raw states of the chunks before m (after m when reverse).  One CTA per (head, b) keeps its block
// of the running sum in registers, in fp32, and reads rows (b, a) with block(a) <= block(b) of every raw chunk state
// once, two chunks ahead by bulk copies; the fp32 states are left as they are.  The first chunk in scan order has nothing
// before it: without a base no read-out asks for its copies and they are not written (skip_first).  The CTA with b == 64
// copies the first-order rows (already summed in place).
// Bound by HBM: 0.71 MB read and up to 0.66 MB written per chunk state; 0.98 ms a launch for 1024 heads of five chunks
// (6.1 TB/s; 1.30 with one chunk ahead in registers and three CTAs an SM), 131 us for 32 heads of sixteen (156).
constexpr int PC_NS = 2, PC_BLK = 64 * BLK_LD * 4;      // chunk states in flight; bytes of a block
__global__ void __launch_bounds__(256, 4) prefix_copies_kernel(const float* __restrict__ state,
                                                            const float* __restrict__ base, char* __restrict__ ca,
                                                            char* __restrict__ cb, int nchunk, int dvp,
                                                            size_t per_state, int reverse, int skip_first) {
  extern __shared__ __align__(128) uint8_t blocks[];
  __shared__ __align__(8) uint64_t bars[PC_NS];
  float(*blk)[BLK_LD] = (float(*)[BLK_LD])(blocks + PC_NS * PC_BLK);
  const int head = blockIdx.y, b = 64 - (int)blockIdx.x, t = threadIdx.x;     // the longest first
  auto at_a = [&](int c) { return ca ? ca + (size_t)(head * nchunk + c) * A_BYTES : nullptr; };
  auto at_b = [&](int c) { return cb ? cb + (size_t)(head * nchunk + c) * B_BYTES : nullptr; };
  if (b == 64) {
    for (int i = skip_first; i < nchunk; ++i) {
      const int c = reverse ? nchunk - 1 - i : i;
      write_first(state + (size_t)(head * nchunk + c) * per_state, blk, dvp, at_a(c), at_b(c), t);
    }
    return;
  }
  const int NV = 16 * ((b >> 4) + 1) * 68 / 4;       // float4 pieces of the rows (b, a) that are read (dvp == 68)
  const size_t blk_off = (size_t)b * 64 * dvp;       // rows (b, a = 0..63) are contiguous
  const uint32_t bar = smem_u32(bars);
  // the last chunk in scan order is never added to anything that is written (and may not have been built)
  auto load = [&](int i) {
    if (i + 1 >= nchunk) return;
    const int c = reverse ? nchunk - 1 - i : i, s = i % PC_NS;
    mbar_expect_tx(bar + 8 * s, NV * 16);
    bulk_load(smem_u32(blocks) + s * PC_BLK, state + (size_t)(head * nchunk + c) * per_state + blk_off, NV * 16, bar + 8 * s);
  };
  if (t == 0) {
    for (int s = 0; s < PC_NS; ++s) mbar_init(bar + 8 * s, 1);
    mbar_fence_init();
    for (int i = 0; i < PC_NS; ++i) load(i);
  }
  float4 run[5];
#pragma unroll
  for (int u = 0; u < 5; ++u) {
    const int v = t + u * 256;
    run[u] = (base && v < NV) ? *(const float4*)(base + (size_t)head * per_state + blk_off + 4 * v)
                              : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  bool ok = true;
  for (int i = 0; i < nchunk; ++i) {
    const int c = reverse ? nchunk - 1 - i : i, s = i % PC_NS;
    const bool wanted = i >= skip_first;
    // the exclusive running sum of this chunk, transposed through shared memory
    if (ok && i + 1 < nchunk && !mbar_wait(bar + 8 * s, (uint32_t)((i / PC_NS) & 1))) { report(91); ok = false; }
#pragma unroll
    for (int u = 0; u < 5; ++u) {
      const int v = t + u * 256;
      if (v < NV) {
        *(float4*)(&blk[0][0] + 4 * v) = run[u];
        if (i + 1 < nchunk) {
          const float4 x = *(const float4*)(blocks + s * PC_BLK + 16 * v);
          run[u].x += x.x; run[u].y += x.y; run[u].z += x.z; run[u].w += x.w;
        }
      }
    }
    __syncthreads();
    if (t == 0 && ok) load(i + PC_NS);
    if (wanted) write_feature(blk, b, at_a(c), at_b(c), t);
    __syncthreads();
  }
}

// zero rows of the groups with an empty state, by `threads` threads of this CTA
__device__ __forceinline__ void write_zeros(const RdArgs& a, int t, int threads) {
  for (int w = blockIdx.x; w < a.heads * a.zero_groups; w += gridDim.x) {
    const int head = w / a.zero_groups, tok0 = (a.zero_first + w % a.zero_groups) * 256;
    const int rows = min(256, a.n - tok0);
    float4* dst = (float4*)(a.out + ((size_t)head * a.n + tok0) * D);
    for (int i = t; i < rows * (D / 4); i += threads) dst[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a.den)
      for (int i = t; i < rows; i += threads) a.den[(size_t)head * a.n + tok0 + i] = 0.f;
  }
}
// ---- type A ---------------------------------------------------------------------------------------------------
// Two token tiles of 128 rows with two 128-column T buffers each.  Eight warps and one issuer warp per tile: the two sets
// of four warps take one half of the columns of every slice, that is eight of its sixteen value columns.  A thread
// loads its 64 columns, hands the buffer back at once and then works from registers: a buffer is away for some 500
// cycles (release -> issue -> product -> commit -> wait), which is what two buffers of a tile have to cover.
constexpr int RA_NS = 4;                                  // ring stages
constexpr int RA_THREADS = 5 * 128;                       // four warpgroups (tile, set), one of producer and issuers
constexpr int RA_UT_LD = 36;                              // floats per staged row
constexpr int RA_OFF_X = 0;                               // [2 items][2 tiles]
constexpr int RA_OFF_ST = 4 * TILE;
constexpr int RA_OFF_UT = RA_OFF_ST + RA_NS * A_STAGE;    // [tile][set][128][36] first-order + constant part
constexpr int RA_OFF_VEC = RA_OFF_UT + 4 * 128 * RA_UT_LD * 4;   // [warpgroup][2 items]
constexpr int RA_VEC = 132;
constexpr int RA_OFF_BAR = RA_OFF_VEC + 8 * RA_VEC * 4;
constexpr int RA_NBAR = 4 + 2 * RA_NS + 8;
constexpr int RA_OFF_TMEM = RA_OFF_BAR + RA_NBAR * 8;
constexpr int RA_SMEM = RA_OFF_TMEM + 16 + 1024;
static_assert(RA_SMEM <= 227 * 1024, "shared memory");
// registers a thread after the split; its sum must not pass that of the launch (or the block never starts)
constexpr int RA_REGS = 104, RA_REGS_REST = 64, RB_REGS = 232, RB_REGS_REST = 40;
static_assert(4 * RA_REGS + RA_REGS_REST <= 5 * 96 && 2 * RB_REGS + RB_REGS_REST <= 3 * 168, "register split");

__global__ void __launch_bounds__(RA_THREADS, 1)
readout_a_kernel(const __grid_constant__ CUtensorMap tmX, const RdArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + RA_OFF_BAR;
  // barriers: x_full[2] | x_empty[2] | st_full[NS] | st_empty[NS] | t_full[tile][buf] | t_free[tile][buf]
  auto BAR_XFULL = [&](int i) { return bar0 + 8u * i; };
  auto BAR_XEMPTY = [&](int i) { return bar0 + 8u * (2 + i); };
  auto BAR_FULL = [&](int s) { return bar0 + 8u * (4 + s); };
  auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (4 + RA_NS + s); };
  auto BAR_TFULL = [&](int t, int b) { return bar0 + 8u * (4 + 2 * RA_NS + 2 * t + b); };
  auto BAR_TFREE = [&](int t, int b) { return bar0 + 8u * (8 + 2 * RA_NS + 2 * t + b); };
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + RA_OFF_TMEM);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(BAR_XFULL(i), 1); mbar_init(BAR_XEMPTY(i), 16 + 2); }
    for (int s = 0; s < RA_NS; ++s) { mbar_init(BAR_FULL(s), 1); mbar_init(BAR_EMPTY(s), 2); }
    for (int t = 0; t < 2; ++t)
      for (int b = 0; b < 2; ++b) { mbar_init(BAR_TFULL(t, b), 1); mbar_init(BAR_TFREE(t, b), 8); }
    mbar_fence_init();
  }
  if (warp == 0) tmem_alloc(smem_u32((const void*)tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp >= 16) {
    regs_down<RA_REGS_REST>();
    if (warp == 16) {
      // ---------------- producer ----------------
      if (lane == 0) {
        tma_prefetch_desc(&tmX);
        bool ok = true;
        int st = 0, k = 0;            // running number of the ring step and of the item
        for (Walk w(a); ok && w.more(); w.next(a), ++k) {
          const int tok0 = w.tok0(a);
          const int xb = k & 1;
          if (!mbar_wait(BAR_XEMPTY(xb), (((k >> 1) & 1) ^ 1))) { report(20); break; }
          mbar_expect_tx(BAR_XFULL(xb), 2 * TILE);
          for (int t = 0; t < 2; ++t)     // rows past the end of the sequence read as zero
            tma_load_3d(sbase + RA_OFF_X + (2 * xb + t) * TILE, &tmX, BAR_XFULL(xb), 0, tok0 + t * 128, w.head);
          const char* src = a.copies + (size_t)w.state(a) * A_BYTES;
          for (int n = 0; n < A_STEPS; ++n, ++st) {
            const int s = st % RA_NS;
            if (!mbar_wait(BAR_EMPTY(s), (((st / RA_NS) & 1) ^ 1))) { report(21); ok = false; break; }
            const uint32_t bytes = n == 0 ? TILE : A_STAGE;
            mbar_expect_tx(BAR_FULL(s), bytes);
            bulk_load(sbase + RA_OFF_ST + s * A_STAGE, src, bytes, BAR_FULL(s));
            src += bytes;
          }
        }
      }
      __syncwarp();
    } else if (warp < 19) {
      // ---------------- MMA issuers: one per tile ----------------
      const int t = warp - 17;
      constexpr uint32_t idesc = idesc_bf16(128, 128, 0, 0), idesc64 = idesc_bf16(128, 64, 0, 0);
      const uint32_t st0 = ((sbase + RA_OFF_ST) & 0x3FFFFu) >> 4;
      bool ok = true;
      int st = 0, k = 0;
      for (int left = Walk(a).left; ok && left > 0; --left, ++k) {
        const int xb = k & 1;
        if (!mbar_wait_warp(BAR_XFULL(xb), (uint32_t)((k >> 1) & 1))) { report(22); break; }
        const uint32_t x_lo = desc_lo(sbase + RA_OFF_X + (2 * xb + t) * TILE, 16);
        for (int n = 0; ok && n < A_STEPS; ++n, ++st) {
          const int s = st % RA_NS, deep = (((n - 1) & 3) >> 1) + 1;    // K steps of the step's first slice
          if (!mbar_wait_warp(BAR_FULL(s), (uint32_t)((st / RA_NS) & 1))) { report(23); ok = false; break; }
          const uint32_t b0 = st0 + (uint32_t)s * (A_STAGE >> 4);
          for (int buf = 0; buf < 2; ++buf) {
            if (!mbar_wait_warp(BAR_TFREE(t, buf), (uint32_t)((st & 1) ^ 1))) { report(24); ok = false; break; } 
            tc_fence_after();
            const uint32_t d = tmem + t * 256 + buf * 128;
            if (elect_one()) {
              if (n == 0) {
                // buffer 0: x . S1, buffer 1: x . E
                umma_ss_k64(d, x_lo, (b0 + (buf ? 8192u >> 4 : 0u)) | (1u << 16), idesc64);
              } else {
                mma_steps(d, x_lo, (b0 + (buf ? (uint32_t)deep * (4096 >> 4) : 0u)) | ((2048u >> 4) << 16), idesc,
                          buf ? 5 - deep : deep);
              }
              umma_commit(BAR_TFULL(t, buf));
              if (buf) {
                umma_commit(BAR_EMPTY(s));
                if (n == A_STEPS - 1) umma_commit(BAR_XEMPTY(xb));
              }
            }
            __syncwarp();
          }
        }
      }
    }
  } else {
    // ---------------- contraction ----------------
    regs_up<RA_REGS>();
    const int wg = warp >> 2, t = wg >> 1, h = wg & 1, qd = warp & 3;
    const int row = qd * 32 + lane;                        // token row in the tile, TMEM lane
    const uint32_t tb = tmem + t * 256 + h * 64 + ((uint32_t)(qd * 32) << 16);
    float* vecs = (float*)(smem + RA_OFF_VEC) + wg * 2 * RA_VEC;
    float* ut = (float*)(smem + RA_OFF_UT) + (size_t)((t * 2 + h) * 128 + row) * RA_UT_LD;
    const uint32_t ut_s = smem_u32(ut);
    write_zeros(a, tid, 512);
    // What an item needs from global memory is asked for one item ahead.  vec: constant row [65], and for set 1
    // S1[:, 64] [64].
    auto first_rows = [&](const Walk& w) { return a.state + (size_t)w.state(a) * a.per_state + (size_t)(64 * 64) * a.dvp; };
    auto const_of = [&](const Walk& w) { return w.more() && row <= 64 ? __ldg(first_rows(w) + (size_t)64 * a.dvp + row) : 0.f; };
    auto norm_of = [&](const Walk& w) { return w.more() && h && row < 64 ? __ldg(first_rows(w) + (size_t)row * a.dvp + 64) : 0.f; };
    auto word_of = [&](const stat_t* st, const Walk& w) { return st && w.more() ? st[w.head] : (stat_t)0; };
    Walk w(a);
    float s0next = const_of(w), n1next = norm_of(w);
    stat_t qnext = word_of(a.stat_q, w), knext = word_of(a.stat_k, w);
    bool ok = true;
    int st = 0, k = 0;
    auto full = [&](int buf) {
      if (ok && !mbar_wait(BAR_TFULL(t, buf), (uint32_t)(st & 1))) { report(26); ok = false; }
      tc_fence_after();
    };
    auto release = [&](int buf) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_TFREE(t, buf));
    };
    for (; w.more(); ++k) {
      const int xb = k & 1;
      const float c = a.stat_q ? stat_scale(&qnext, 0, a.lim) * stat_scale(&knext, 0, a.lim) : 1.f;
      const float A1 = a.a1 * c, A2 = a.a2 * c * c;
      const int tok = w.tok0(a) + t * 128 + row;
      const bool tok_ok = tok < a.n;
      const size_t grow = (size_t)w.head * a.n + (tok_ok ? tok : 0);
      const uint32_t xrow = sbase + RA_OFF_X + (2 * xb + t) * TILE + row * 128, xs = (uint32_t)(row & 7) << 4;
      float* vec = vecs + xb * RA_VEC;    // the set's warps are done with the one of two items ago since the last barrier
      if (row <= 64) vec[row] = s0next;
      if (h && row < 64) vec[68 + row] = n1next;
      w.next(a);
      s0next = const_of(w);
      n1next = norm_of(w);
      qnext = word_of(a.stat_q, w);
      knext = word_of(a.stat_k, w);
      asm volatile("bar.sync %0, 128;" ::"r"(1 + wg) : "memory");
      if (ok && !mbar_wait(BAR_XFULL(xb), (uint32_t)((k >> 1) & 1))) { report(25); ok = false; }
      // ---- step 0, buffer 0: x . S1, of which this set stages the value columns it will write
      full(0);
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t tv[16];
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t (&t8)[8] = *(uint32_t(*)[8])(tv + 8 * g);
          tmem_ld8(tb - h * 64 + (2 * (2 * hf + g) + h) * 8, t8);
        }
        tmem_wait_ld(tv);
        if (hf == 1) release(0);
#pragma unroll
        for (int g = 0; g < 2; ++g)
#pragma unroll
          for (int e = 0; e < 8; e += 4) {
            const int cc = (2 * (2 * hf + g) + h) * 8 + e;
            float4 v;
            v.x = fmaf(A1, __uint_as_float(tv[8 * g + e]), a.a0 * vec[cc]);
            v.y = fmaf(A1, __uint_as_float(tv[8 * g + e + 1]), a.a0 * vec[cc + 1]);
            v.z = fmaf(A1, __uint_as_float(tv[8 * g + e + 2]), a.a0 * vec[cc + 2]);
            v.w = fmaf(A1, __uint_as_float(tv[8 * g + e + 3]), a.a0 * vec[cc + 3]);
            *(float4*)(ut + (2 * hf + g) * 8 + e) = v;
          }
      }
      // ---- buffer 1: x . E, the normaliser, by set 1
      full(1);
      if (h == 0) {
        release(1);
      } else {
        uint32_t tv[64];
        tmem_ld64(tb - h * 64 + 128, tv);
        tmem_wait_ld(tv);
        release(1);
        uint64_t s4[4] = {0ull, 0ull, 0ull, 0ull};
        float first = 0.f;
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          const uint4 xw = lds128(xrow + (((uint32_t)v << 4) ^ xs));
          const uint32_t ww[4] = {xw.x, xw.y, xw.z, xw.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int i = v * 8 + 2 * e;
            s4[e] = fma2(pack2(bf_lo(ww[e]), bf_hi(ww[e])), pack2u(tv[i], tv[i + 1]), s4[e]);
            first = fmaf(bf_lo(ww[e]), vec[68 + i], first);
            first = fmaf(bf_hi(ww[e]), vec[69 + i], first);
          }
        }
        if (ok && a.den && tok_ok) {
          float lo, hi;
          unpack2(add2(add2(s4[0], s4[1]), add2(s4[2], s4[3])), lo, hi);
          a.den[grow] = fmaf(A2, lo + hi, fmaf(A1, first, a.a0 * vec[64]));
        }
      }
      ++st;
      // ---- steps 1..16: eight value columns over the eight octets of features b
#pragma unroll 1
      for (int g = 0; g < 4; ++g) {
        uint64_t acc[8] = {0ull, 0ull, 0ull, 0ull, 0ull, 0ull, 0ull, 0ull};   // even and odd features apart
        auto slice = [&](int buf, int oct) {
          uint32_t tv[64];
          full(buf);
          tmem_ld64(tb + buf * 128, tv);
          const uint4 xw = lds128(xrow + (((uint32_t)oct << 4) ^ xs));
          const uint32_t ww[4] = {xw.x, xw.y, xw.z, xw.w};
          tmem_wait_ld(tv);
          release(buf);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint64_t x0 = pack2(bf_lo(ww[i]), bf_lo(ww[i])), x1 = pack2(bf_hi(ww[i]), bf_hi(ww[i]));
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[e] = fma2(x0, pack2u(tv[16 * i + 2 * e], tv[16 * i + 2 * e + 1]), acc[e]);
#pragma unroll
            for (int e = 0; e < 4; ++e)
              acc[4 + e] = fma2(x1, pack2u(tv[16 * i + 8 + 2 * e], tv[16 * i + 9 + 2 * e]), acc[4 + e]);
          }
        };
#pragma unroll 1
        for (int j = 0; j < 4; ++j, ++st) {
          slice(0, j);
          slice(1, 7 - j);
        }
        const int cg = 2 * g + h;
        const ulonglong2 b0 = lds_v2(ut_s + g * 32), b1 = lds_v2(ut_s + g * 32 + 16);
        const uint64_t bs[4] = {b0.x, b0.y, b1.x, b1.y}, k2 = pack2(A2, A2);
        uint32_t o[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float lo, hi;
          unpack2(fma2(k2, add2(acc[e], acc[4 + e]), bs[e]), lo, hi);
          o[2 * e] = __float_as_uint(lo);
          o[2 * e + 1] = __float_as_uint(hi);
        }
        if (ok && tok_ok) stg32(a.out + grow * D + cg * 8, o, a.wide_io != 0);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_XEMPTY(xb));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// ---- type B ---------------------------------------------------------------------------------------------------
// Four warps and one issuer warp per tile; a thread keeps the 64 running sums of its token as packed pairs, so the walk
// over the 36 blocks is unrolled.  A slice is loaded whole and its buffer handed back at once, as in type A; the
// registers for that come from the third warpgroup (producer and issuers).
constexpr int RB_NS = 5;
constexpr int RB_THREADS = 384;
constexpr int RB_OFF_X = 0;                               // [2 items][x0 x1 u0 u1]
constexpr int RB_OFF_ST = 8 * TILE;
constexpr int RB_OFF_VEC = RB_OFF_ST + RB_NS * TILE;
constexpr int RB_VEC = 196;                               // S1[:, 64] [64], e [128], scale
constexpr int RB_OFF_BAR = RB_OFF_VEC + 4 * RB_VEC * 4;   // [2 tiles][2 items]
constexpr int RB_NBAR = 4 + 2 * RB_NS + 8;
constexpr int RB_OFF_TMEM = RB_OFF_BAR + RB_NBAR * 8;
constexpr int RB_SMEM = RB_OFF_TMEM + 16 + 1024;
static_assert(RB_SMEM <= 227 * 1024, "shared memory");

__global__ void __launch_bounds__(RB_THREADS, 1)
readout_b_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmU, const RdArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + RB_OFF_BAR;
  // barriers: x_full[2] | x_empty[2] | st_full[NS] | st_empty[NS] | t_full[tile][buf] | t_free[tile][buf]
  auto BAR_XFULL = [&](int i) { return bar0 + 8u * i; };
  auto BAR_XEMPTY = [&](int i) { return bar0 + 8u * (2 + i); };
  auto BAR_FULL = [&](int s) { return bar0 + 8u * (4 + s); };
  auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (4 + RB_NS + s); };
  auto BAR_TFULL = [&](int t, int b) { return bar0 + 8u * (4 + 2 * RB_NS + 2 * t + b); };
  auto BAR_TFREE = [&](int t, int b) { return bar0 + 8u * (8 + 2 * RB_NS + 2 * t + b); };
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + RB_OFF_TMEM);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) { mbar_init(BAR_XFULL(i), 1); mbar_init(BAR_XEMPTY(i), 8 + 2); }
    for (int s = 0; s < RB_NS; ++s) { mbar_init(BAR_FULL(s), 1); mbar_init(BAR_EMPTY(s), 2); }
    for (int t = 0; t < 2; ++t)
      for (int b = 0; b < 2; ++b) { mbar_init(BAR_TFULL(t, b), 1); mbar_init(BAR_TFREE(t, b), 4); }
    mbar_fence_init();
  }
  if (warp == 0) tmem_alloc(smem_u32((const void*)tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp >= 8) {
  regs_down<RB_REGS_REST>();
  if (warp == 8) {
    // ---------------- producer ----------------
    if (lane == 0) {
      tma_prefetch_desc(&tmX);
      tma_prefetch_desc(&tmU);
      bool ok = true;
      int st = 0, k = 0;
      for (Walk w(a); ok && w.more(); w.next(a), ++k) {
        const int tok0 = w.tok0(a);
        const int xb = k & 1;
        if (!mbar_wait(BAR_XEMPTY(xb), (((k >> 1) & 1) ^ 1))) { report(30); break; }
        mbar_expect_tx(BAR_XFULL(xb), 4 * TILE);
        for (int t = 0; t < 2; ++t) {
          const uint32_t x = sbase + RB_OFF_X + (4 * xb + t) * TILE;
          tma_load_3d(x, &tmX, BAR_XFULL(xb), 0, tok0 + t * 128, w.head);
          tma_load_3d(x + 2 * TILE, &tmU, BAR_XFULL(xb), 0, tok0 + t * 128, w.head);
        }
        const char* src = a.copies + (size_t)w.state(a) * B_BYTES;
        for (int n = 0; n < B_SLICES; ++n, ++st) {
          const int s = st % RB_NS;
          if (!mbar_wait(BAR_EMPTY(s), (((st / RB_NS) & 1) ^ 1))) { report(31); ok = false; break; }
          mbar_expect_tx(BAR_FULL(s), TILE);
          bulk_load(sbase + RB_OFF_ST + s * TILE, src + (size_t)n * TILE, TILE, BAR_FULL(s));
        }
      }
    }
    __syncwarp();
  } else if (warp < 11) {
    // ---------------- MMA issuers: one per tile ----------------
    const int t = warp - 9;
    constexpr uint32_t idesc = idesc_bf16(128, 128, 0, 0), idesc64 = idesc_bf16(128, 64, 0, 0);
    const uint32_t st0 = desc_lo(sbase + RB_OFF_ST, 16);
    bool ok = true;
    int st = 0, k = 0;
    for (int left = Walk(a).left; ok && left > 0; --left, ++k) {
      const int xb = k & 1;
      if (!mbar_wait_warp(BAR_XFULL(xb), (uint32_t)((k >> 1) & 1))) { report(32); break; }
      const uint32_t x_lo = desc_lo(sbase + RB_OFF_X + (4 * xb + t) * TILE, 16);
      const uint32_t u_lo = desc_lo(sbase + RB_OFF_X + (4 * xb + 2 + t) * TILE, 16);
      for (int n = 0; n < B_SLICES; ++n, ++st) {
        const int s = st % RB_NS, buf = st & 1;
        if (!mbar_wait_warp(BAR_FULL(s), (uint32_t)((st / RB_NS) & 1))) { report(33); ok = false; break; }
        if (!mbar_wait_warp(BAR_TFREE(t, buf), (uint32_t)(((st >> 1) & 1) ^ 1))) { report(34); ok = false; break; } 
        tc_fence_after();
        const uint32_t d = tmem + t * 256 + buf * 128, b0 = st0 + (uint32_t)s * (TILE >> 4);
        if (elect_one()) {
          if (n < 18) {
            umma_ss_k64(d, u_lo, b0, idesc);
          } else {
            umma_ss_k64(d, u_lo, b0, idesc64);
            umma_ss_k64(d + 64, x_lo, b0 + (8192 >> 4), idesc64);
          }
          umma_commit(BAR_TFULL(t, buf));
          umma_commit(BAR_EMPTY(s));
          if (n == B_SLICES - 1) umma_commit(BAR_XEMPTY(xb));
        }
        __syncwarp();
      }
    }
  }
  } else {
    // ---------------- contraction: four warps per tile ----------------
    regs_up<RB_REGS>();
    const int t = warp >> 2, qd = warp & 3;
    const int row = qd * 32 + lane;
    const uint32_t tb = tmem + t * 256 + ((uint32_t)(qd * 32) << 16);
    float* vecs = (float*)(smem + RB_OFF_VEC) + 2 * t * RB_VEC;
    write_zeros(a, tid, 256);
    // what an item needs from global memory is asked for at the start of the item before and staged a few slices later
    auto vec_of = [&](const Walk& w) {
      if (!w.more() || row >= 64) return 0.f;
      return __ldg(a.state + (size_t)w.state(a) * a.per_state + (size_t)(64 * 64 + row) * a.dvp + 64);
    };
    auto word_of = [&](const stat_t* st, const Walk& w) { return st && w.more() ? st[w.head] : (stat_t)0; };
    auto e_of = [&](const Walk& w) {
      const int tok = w.tok0(a) + t * 128 + row;
      return !w.more() || tok >= a.n ? 0.f : (a.uvec ? -__ldg(a.uvec + (size_t)w.head * a.n + tok) : 1.f);
    };
    Walk w(a);
    auto stage = [&](float* vec, float v, stat_t wq, stat_t wk, float e) {
      if (row < 64) vec[row] = v;
      vec[64 + row] = e;
      if (row == 0) vec[192] = a.stat_q ? stat_scale(&wq, 0, a.lim) * stat_scale(&wk, 0, a.lim) : 1.f;
    };
    stage(vecs, vec_of(w), word_of(a.stat_q, w), word_of(a.stat_k, w), e_of(w));
    bool ok = true;
    int st = 0, k = 0;
    auto full = [&](int slice) {
      if (ok && !mbar_wait(BAR_TFULL(t, slice & 1), (uint32_t)((slice >> 1) & 1))) { report(36); ok = false; }
      tc_fence_after();
    };
    auto release = [&](int slice) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_TFREE(t, slice & 1));
    };
    for (; w.more(); ++k) {
      const int xb = k & 1;
      const int tok = w.tok0(a) + t * 128 + row;
      float* dst = a.out + ((size_t)w.head * a.n + tok) * D;
      const uint32_t xrow = sbase + RB_OFF_X + (4 * xb + t) * TILE + row * 128, xs = (uint32_t)(row & 7) << 4;
      const float* vec = vecs + xb * RB_VEC;
      w.next(a);
      const float vnext = vec_of(w), enext = e_of(w);
      const stat_t qnext = word_of(a.stat_q, w), knext = word_of(a.stat_k, w);
      // this item's values are staged, and nobody reads those of the item before any more
      asm volatile("bar.sync %0, 128;" ::"r"(1 + t) : "memory");
      if (ok && !mbar_wait(BAR_XFULL(xb), (uint32_t)((k >> 1) & 1))) { report(35); ok = false; }
      uint64_t r[32];
#pragma unroll
      for (int e = 0; e < 32; ++e) r[e] = 0ull;
      // block (alpha, beta) of M from tv[0] on; wa, wb: the words of the token's features of alpha and beta.
      // Neighbouring products share an operand (the register file delivers two packed operands a product at full rate).
      auto block = [&](const uint32_t* tv, const int alpha, const int beta, const uint4& xa, const uint4& xb4) {
        const uint32_t wa[4] = {xa.x, xa.y, xa.z, xa.w}, wb[4] = {xb4.x, xb4.y, xb4.z, xb4.w};
        uint64_t fb[4];
#pragma unroll
        for (int bp = 0; bp < 4; ++bp) fb[bp] = pack2(bf_lo(wb[bp]), bf_hi(wb[bp]));
        uint64_t* rb = r + 4 * beta;
#pragma unroll
        for (int ap = 0; ap < 4; ++ap) {
          const uint64_t fa = pack2(bf_lo(wa[ap]), bf_hi(wa[ap])), fs = pack2(bf_hi(wa[ap]), bf_lo(wa[ap]));
          uint64_t ra = r[4 * alpha + ap], rs = 0ull;
#pragma unroll
          for (int bp = 0; bp < 4; ++bp) {
            const uint64_t P = pack2u(tv[16 * ap + 4 * bp], tv[16 * ap + 4 * bp + 1]);
            rb[bp] = fma2(fa, P, rb[bp]);
            if (alpha != beta) ra = fma2(fb[bp], P, ra);
          }
#pragma unroll
          for (int bp = 0; bp < 4; ++bp) {
            const uint64_t Q = pack2u(tv[16 * ap + 4 * bp + 2], tv[16 * ap + 4 * bp + 3]);
            rb[bp] = fma2(fs, Q, rb[bp]);
            if (alpha != beta) rs = fma2(fb[bp], Q, rs);
          }
          if (alpha != beta) {
            float s0, s1;
            unpack2(rs, s0, s1);
            r[4 * alpha + ap] = add2(ra, pack2(s1, s0));
          }
        }
      };
      auto words = [&](int oct) { return lds128(xrow + (((uint32_t)oct << 4) ^ xs)); };
#pragma unroll
      for (int n = 0; n < 18; ++n, ++st) {
        int b0 = 0, b1 = 0;
#pragma unroll
        for (int i = 1; i < 8; ++i) {
          if (i * (i + 1) / 2 <= 2 * n) b0 = i;
          if (i * (i + 1) / 2 <= 2 * n + 1) b1 = i;
        }
        const int a0 = 2 * n - b0 * (b0 + 1) / 2, a1 = 2 * n + 1 - b1 * (b1 + 1) / 2;
        uint32_t tv[128];
        full(st);
        tmem_ld64(tb + (st & 1) * 128, tv);
        tmem_ld64(tb + (st & 1) * 128 + 64, tv + 64);
        const uint4 xa0 = words(a0), xb0 = words(b0);
        tmem_wait_ld(tv);
        release(st);
        if (n == 5) stage(vecs + (xb ^ 1) * RB_VEC, vnext, qnext, knext, enext);
        block(tv, a0, b0, xa0, xb0);
        block(tv + 64, a1, b1, words(a1), words(b1));
      }
      // ---- last slice: u . S1[a][0..63] and x . E; the running sums take their factor here
      {
        uint32_t tv[128];
        full(st);
        tmem_ld64(tb + (st & 1) * 128, tv);
        tmem_ld64(tb + (st & 1) * 128 + 64, tv + 64);
        tmem_wait_ld(tv);
        release(st);
        ++st;
        const float ue = vec[64 + row], c = vec[192], A1 = a.a1 * c, K2 = 2.f * a.a2 * c * c;
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          uint32_t o[8];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int f = v * 8 + 2 * e;
            float s0, s1;
            unpack2(r[f >> 1], s0, s1);
            s0 = fmaf(ue, __uint_as_float(tv[64 + f]), s0);
            s1 = fmaf(ue, __uint_as_float(tv[65 + f]), s1);
            o[2 * e] = __float_as_uint(fmaf(K2, s0, A1 * fmaf(ue, vec[f], __uint_as_float(tv[f]))));
            o[2 * e + 1] = __float_as_uint(fmaf(K2, s1, A1 * fmaf(ue, vec[f + 1], __uint_as_float(tv[f + 1]))));
          }
          if (ok && tok < a.n) stg32(dst + v * 8, o, a.wide_io != 0);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_XEMPTY(xb));
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace

int readout_status(int* out, cudaStream_t stream) {
  FM_CUDA_TRY(cudaMemcpyFromSymbolAsync(out, g_readout_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
int readout_status_reset(cudaStream_t stream) {
  const int zero = 0;
  FM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_readout_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}

size_t moments_tc_copy_a_bytes(int mats) { return (size_t)mats * A_BYTES; }
size_t moments_tc_copy_b_bytes(int mats) { return (size_t)mats * B_BYTES; }

int moments_tc_convert(const Ctx& c, int mats, const float* state, const StateCopies& to) {
  if (mats == 0) return FASTMAX_OK;
  const MomentDims m = moment_dims(64);
  if ((((uintptr_t)to.a | (uintptr_t)to.b) & 15) != 0)
    return fail(FASTMAX_E_ARG, "the copies of the moment states must be 16-byte aligned");
  dim3 grid(65, mats);
  FM_LAUNCH("fm_moments_state_bf16", c.stream,
            (copies_kernel<<<grid, 256, 0, c.stream>>>(state, (char*)to.a, (char*)to.b, m.dvp, (size_t)m.f * m.dvp)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

// Exclusive running sums over chunks (from `base`, per head, may be null) of the second-order rows, written as the
// copies that are asked for; the fp32 states stay raw.  The first-order rows are the caller's business (moments_prefix
// with a row range).
int moments_tc_prefix_convert(const Ctx& c, int heads, int nchunk, const float* state, const float* base, int reverse,
                              const StateCopies& to) {
  if (heads == 0 || nchunk == 0) return FASTMAX_OK;
  const MomentDims m = moment_dims(64);
  if ((((uintptr_t)state | (uintptr_t)base | (uintptr_t)to.a | (uintptr_t)to.b) & 15) != 0)
    return fail(FASTMAX_E_ARG, "moment states, totals and copies must be 16-byte aligned");
  dim3 grid(65, heads);
  FM_CUDA_TRY(cudaFuncSetAttribute(prefix_copies_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (PC_NS + 1) * PC_BLK));
  FM_LAUNCH("fm_moments_prefix_bf16", c.stream,
            (prefix_copies_kernel<<<grid, 256, (PC_NS + 1) * PC_BLK, c.stream>>>(state, base, (char*)to.a, (char*)to.b, nchunk, m.dvp,
                                                              (size_t)m.f * m.dvp, reverse, base ? 0 : 1)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

// Type A of the tokens x into (out, den), complete with the first-order and constant terms of the fp32 states, whose
// first-order rows are running sums; type B with (u, uvec) into out.  Results overwrite.
static int readout(const Ctx& c, bool type_b, int heads, int n, int chunk, int state_per_chunk, const void* x,
                   const void* u, const float* uvec, const void* copies, const stat_t* stats, const float* state,
                   float* out, float* den) {
  if (heads == 0 || n == 0) return FASTMAX_OK;
  const fastmax_problem& p = c.p;
  CUtensorMap tx, tu;
  int rc;
  if ((rc = tma_map_bf16(&tx, x, heads, n, D, 128))) return rc;
  if (type_b && (rc = tma_map_bf16(&tu, u, heads, n, D, 128))) return rc;
  const MomentDims md = moment_dims(64);
  RdArgs a;
  a.copies = (const char*)copies; a.state = state; a.uvec = uvec; a.out = out; a.den = den;
  a.stat_q = p.normalize ? stats : nullptr;
  a.stat_k = p.normalize ? stats + p.bh : nullptr;
  a.a0 = p.a0; a.a1 = p.a1; a.a2 = p.a2; a.lim = p.lim;
  a.per_state = (size_t)md.f * md.dvp; a.dvp = md.dvp; a.heads = heads; a.n = n;
  a.chunk = state_per_chunk ? chunk : 0;
  a.nchunk = (n + chunk - 1) / chunk;
  a.per_chunk = chunk / 256;
  a.first = 0;
  a.groups = (n + 255) / 256;
  a.zero_first = 0;
  a.zero_groups = 0;
  if (state_per_chunk && c.zero_chunk >= 0) {
    // chunks are multiples of 256 tokens; the empty one is the first or the last
    const int per = chunk / 256;
    a.zero_first = c.zero_chunk * per;
    a.zero_groups = min(per, a.groups - a.zero_first);
    if (c.zero_chunk == 0) a.first = a.zero_groups;
    a.groups -= a.zero_groups;
  }
  a.wide_io = ((uintptr_t)out & 31) == 0;
  const int work = heads * (a.groups > a.zero_groups ? a.groups : a.zero_groups);
  const unsigned grid = (unsigned)(work < 148 ? work : 148);
  a.items = heads * a.groups;
  if (type_b) {
    FM_CUDA_TRY(cudaFuncSetAttribute(readout_b_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RB_SMEM));
    FM_LAUNCH("fm_moments_tc_readout_b", c.stream, (readout_b_kernel<<<grid, RB_THREADS, RB_SMEM, c.stream>>>(tx, tu, a)));
  } else {
    FM_CUDA_TRY(cudaFuncSetAttribute(readout_a_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, RA_SMEM));
    FM_LAUNCH("fm_moments_tc_readout_a", c.stream, (readout_a_kernel<<<grid, RA_THREADS, RA_SMEM, c.stream>>>(tx, a)));
  }
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}
int moments_tc_readout_a(const Ctx& c, int heads, int n, int chunk, int state_per_chunk, const void* x,
                         const void* copies_a, const stat_t* stats, const float* state, float* out, float* den) {
  return readout(c, false, heads, n, chunk, state_per_chunk, x, nullptr, nullptr, copies_a, stats, state, out, den);
}
int moments_tc_readout_b(const Ctx& c, int heads, int n, int chunk, int state_per_chunk, const void* x, const void* u,
                         const float* uvec, const void* copies_b, const stat_t* stats, const float* state, float* out) {
  return readout(c, true, heads, n, chunk, state_per_chunk, x, u, uvec, copies_b, stats, state, out, nullptr);
}

}  // namespace fm
