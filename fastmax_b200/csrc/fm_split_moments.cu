// Unmasked second-order forward in float32 on the tensor cores, in moment form (d = 64): the sums over all keys
//   S2[(a, b)][c] = sum_j k_j[a] k_j[b] (v_j, 1)[c],  S1, S0
// once per key/value head, then for every query row r = a2 q (x) q . S2 + a1 q . S1 + a0 S0 and out = r[0..63] / r[64].
// The score form costs 4 n d operations a query (a multiply-add counts two); this 2 x 65 for each of 2 560 pairs of features (the
// blocks of 16 on and below the diagonal) and 65 lower terms, 5 300 d, whatever n is, and for the sums 2 x 65 x 2 145 = 4 400 d a
// key.  Every operand is the exact sum of three bf16
// parts (fm_dense_split.cu), every product sum six sums of bf16 products, the small ones first.
//   pair_sums_kernel   features are formed in fp32 (one rounding), split and put in tensor memory as the A operand, 128
//                      unordered pairs a tile; B are the value parts.  An accumulator holds 64 tokens and is added to
//                      fp32 registers (the tensor core truncates when it adds).  Bound by the generators' chain: 4 000 cycles
//                      a block of 64 tokens and two tiles, against 1 560 of products.
//   copies3_kernel     the type A operand copies (fm_readout.cuh) of the three parts of the sums.
//   readout3_kernel    the type A read-out with six products to a slice, and the division.  Bound by the products: 504 K
//                      steps of 128 x 128 x 16 per 128 rows, 32 600 cycles.
// 64 heads x 10 000: sums 1.32 ms, copies 0.03, read-out 0.90, operand parts 0.12, where the score form takes 7.1 ms.  2-norm
// error against float64 of N(0,1) inputs, normalised, 2.4e-7 (score form 2.6e-7); other inputs at split_moments_faster.  The transposed key block written one block ahead: no change.
#include "fm_readout.cuh"

namespace fm {

__device__ int g_smom_status = 0;

namespace {
using namespace rdo;

__device__ __forceinline__ void report(int code) { atomicCAS(&g_smom_status, 0, code); }

// ---- sums over the keys ---------------------------------------------------------------------------------------
// Rows as in fm_decode_tc.cu: lane L of tile t is the pair (b, b + s mod 64), b = L % 64, s = 2 t + L / 64, s = 0..32 (half
// of s = 32); row 64 of the transposed block is ones (the first-order rows and the constant row), row 65 zeros.
constexpr int TB = 64;                                  // tokens per block
constexpr int PS_GEN = 512, PS_THREADS = 19 * 32;       // 16 generator warps, producer, two issuers
constexpr int PS_NS = 3;
constexpr int PS_STAGE = 3 * TB * D * 2;                // value parts of a block
constexpr int PS_ROWS = D + 2, PS_LD = TB * 4 + 16, PS_YT = PS_ROWS * PS_LD;
constexpr int PS_TILES = 17;
constexpr int PS_OFF_Y = PS_NS * PS_STAGE;              // two transposed blocks, fp32
constexpr int PS_OFF_EP = PS_OFF_Y + 2 * PS_YT;         // float ep[2][128][65], then the second share of the last column
constexpr int PS_OFF_E = PS_OFF_EP + 2 * 128 * 65 * 4;
constexpr int PS_OFF_BAR = PS_OFF_E + 2 * 128 * 4;
constexpr int PS_NBAR = 2 * PS_NS + 4;
constexpr int PS_OFF_TMEM = PS_OFF_BAR + PS_NBAR * 8;
constexpr int PS_SMEM = PS_OFF_TMEM + 16 + 1024;
static_assert(PS_SMEM <= 227 * 1024, "shared memory");
constexpr int PS_TM = 256;                              // tensor memory columns of a tile: sums 64, two operands of 3 x 32
// byte offset of token chunk c (4 tokens) of row f inside a transposed block: 16 bytes between rows, so that any eight
// neighbouring rows (a lane's second one is its own plus the tile's distance) are read from different banks
// (64 heads of 10000 keys 1152 us; 1320 with the pieces of 256-byte rows permuted, which suits aligned eights only)
__device__ __forceinline__ uint32_t yt_off(int f, int c) { return (uint32_t)(f * PS_LD + c * 16); }

__global__ void __launch_bounds__(PS_THREADS, 1)
pair_sums_kernel(const __grid_constant__ CUtensorMap tmV, const float* __restrict__ k, const stat_t* __restrict__ stat_k, float lim,
                 float* __restrict__ state, int n, int dvp, size_t per_state) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + PS_OFF_BAR;
  auto BAR_VF = [&](int s) { return bar0 + 8u * s; };
  auto BAR_VE = [&](int s) { return bar0 + 8u * (PS_NS + s); };
  auto BAR_A = [&](int t) { return bar0 + 8u * (2 * PS_NS + t); };
  auto BAR_DONE = [&](int t) { return bar0 + 8u * (2 * PS_NS + 2 + t); };
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + PS_OFF_TMEM);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head = blockIdx.y, tile0 = blockIdx.x * 2, active = min(2, PS_TILES - tile0);
  const int nblk = (n + TB - 1) / TB;
  if (tid == 0) {
    for (int s = 0; s < PS_NS; ++s) { mbar_init(BAR_VF(s), 1); mbar_init(BAR_VE(s), active); }
    for (int t = 0; t < 2; ++t) { mbar_init(BAR_A(t), 8); mbar_init(BAR_DONE(t), 1); }
    mbar_fence_init();
  }
  if (warp == 17) tmem_alloc(smem_u32((const void*)tmem_slot), 512);
  for (int i = tid; i < 2 * TB; i += PS_THREADS) *(float*)(smem + PS_OFF_Y + (i / TB) * PS_YT + (D + 1) * PS_LD + (i % TB) * 4) = 0.f;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  bool ok = true;
  if (warp == 16) {
    if (lane == 0) tma_prefetch_desc(&tmV);
    for (int j = 0; j < nblk; ++j) {
      const int s = j % PS_NS;
      if (!mbar_wait(BAR_VE(s), (uint32_t)(((j / PS_NS) & 1) ^ 1))) { report(81); break; }
      if (lane == 0) {
        mbar_expect_tx(BAR_VF(s), PS_STAGE);
        for (int part = 0; part < 3; ++part)     // rows past the last key read as zero
          tma_load_3d(sbase + s * PS_STAGE + part * (TB * D * 2), &tmV, BAR_VF(s), part * D, j * TB, head);
      }
    }
  } else if (warp >= 17) {
    const int t = warp - 17;
    if (t < active) {
      constexpr uint32_t idesc = idesc_bf16(128, 64, 0, 1);
      const uint32_t acc = tmem + t * PS_TM;
      for (int j = 0; j < nblk; ++j) {
        const int s = j % PS_NS;
        if (!mbar_wait_warp(BAR_VF(s), (uint32_t)((j / PS_NS) & 1))) { report(82); break; }
        if (!mbar_wait_warp(BAR_A(t), (uint32_t)(j & 1))) { report(83); break; }
        tc_fence_after();
        const uint32_t v0 = desc_lo(sbase + s * PS_STAGE, 8192), step = 8192 >> 4, op = acc + 64 + (j & 1) * 96;
        if (elect_one()) {
          umma_ts_steps<TB / 16>(acc, op + 64, v0, idesc, 0u);                // l h
          umma_ts_steps<TB / 16>(acc, op, v0 + 2 * step, idesc, 1u);          // h l
          umma_ts_steps<TB / 16>(acc, op + 32, v0 + step, idesc, 1u);         // m m
          umma_ts_steps<TB / 16>(acc, op + 32, v0, idesc, 1u);                // m h
          umma_ts_steps<TB / 16>(acc, op, v0 + step, idesc, 1u);              // h m
          umma_ts_steps<TB / 16>(acc, op, v0, idesc, 1u);                     // h h
          umma_commit(BAR_DONE(t));
          umma_commit(BAR_VE(s));
        }
        __syncwarp();
      }
    }
    __syncwarp();
  } else {
    const int t = warp >> 3, qd = warp & 3, hf = (warp >> 2) & 1;    // tile, lane quarter, half of the block's tokens
    const int L = qd * 32 + lane, tile = tile0 + t;
    const bool on = t < active;
    int fx = D + 1, fy = D + 1;                                      // this lane's two feature rows
    if (on) {
      const int b = L & 63, s = 2 * tile + (L >> 6);
      if (s < D / 2) { fx = b; fy = (b + s) & (D - 1); }
      else if (s == D / 2) {
        if (b < D / 2) { fx = b; fy = b + D / 2; }
        else if (b == D / 2) { fx = D; fy = D; }
      } else { fx = b; fy = D; }
    }
    const uint32_t tl = tmem + t * PS_TM + ((uint32_t)(qd * 32) << 16);
    uint64_t run[16], e_run = 0ull;
#pragma unroll
    for (int i = 0; i < 16; ++i) run[i] = 0ull;
    auto promote = [&]() {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t v[16];
        tmem_ld16(tl + hf * 32 + h * 16, v);
        tmem_wait_ld(v);
#pragma unroll
        for (int i = 0; i < 8; ++i) run[8 * h + i] = add2(run[8 * h + i], pack2u(v[2 * i], v[2 * i + 1]));
      }
    };
    // four features of one token per thread and load, two loads a block; tokens past the end read as zero
    const float* kh = k + (size_t)head * n * D;
    const float ks = pow2_of(stat_scale(stat_k, head, lim));
    float4 kr[2];
    auto fetch = [&](int j) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int idx = tid + i * PS_GEN, tok = j * TB + idx / 16;
        kr[i] = (j < nblk && tok < n) ? __ldg((const float4*)(kh + (size_t)tok * D) + idx % 16) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    fetch(0);
    for (int j = 0; j < nblk; ++j) {
      uint8_t* yt = smem + PS_OFF_Y + (j & 1) * PS_YT;
      const uint32_t yt_s = sbase + PS_OFF_Y + (j & 1) * PS_YT;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int idx = tid + i * PS_GEN, tok = idx / 16, f0 = (idx % 16) * 4;
        // lane pairs begin at different features, or the sixteen of a token would meet two banks
        const float4 w = kr[i];
        const bool r1 = (idx >> 1) & 1, r2 = (idx >> 2) & 1;
        const float a0 = r1 ? w.y : w.x, a1 = r1 ? w.z : w.y, a2 = r1 ? w.w : w.z, a3 = r1 ? w.x : w.w;
        const float v[4] = {r2 ? a2 : a0, r2 ? a3 : a1, r2 ? a0 : a2, r2 ? a1 : a3};
#pragma unroll
        for (int e = 0; e < 4; ++e)
          *(float*)(yt + yt_off(f0 + ((e + (idx >> 1)) & 3), tok >> 2) + (tok & 3) * 4) = ks * v[e];
      }
      if (tid < TB) *(float*)(yt + yt_off(D, tid >> 2) + (tid & 3) * 4) = j * TB + tid < n ? 1.f : 0.f;
      asm volatile("bar.sync 1, 512;" ::: "memory");
      fetch(j + 1);
      if (!on) continue;
      uint64_t e2 = 0ull;
      // sixteen tokens at a time: their operand words and the running sums fit the registers
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t hi[8], mi[8], lo[8];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int chunk = hf * 8 + half * 4 + c;
          const ulonglong2 x = lds_v2(yt_s + yt_off(fx, chunk)), y = lds_v2(yt_s + yt_off(fy, chunk));
          const uint64_t p0 = mul2(x.x, y.x), p1 = mul2(x.y, y.y);
          e2 = add2(e2, add2(p0, p1));
          split3(p0, hi[2 * c], mi[2 * c], lo[2 * c]);
          split3(p1, hi[2 * c + 1], mi[2 * c + 1], lo[2 * c + 1]);
        }
        // (the products of the block before last, which read these columns, were done when the last one's sums were taken)
        const uint32_t op = tl + 64 + (j & 1) * 96 + hf * 16 + half * 8;
        tmem_st8(op, hi);
        tmem_st8(op + 32, mi);
        tmem_st8(op + 64, lo);
      }
      e_run = add2(e_run, e2);
      if (j > 0) {      // take the previous block's sums over
        if (ok && !mbar_wait(BAR_DONE(t), (uint32_t)((j - 1) & 1))) { report(84); ok = false; }
        tc_fence_after();
        promote();
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_A(t));
    }
    if (on) {
      if (ok && !mbar_wait(BAR_DONE(t), (uint32_t)((nblk - 1) & 1))) { report(85); ok = false; }
      tc_fence_after();
      promote();
      float* ep = (float*)(smem + PS_OFF_EP) + (t * 128 + L) * 65;
#pragma unroll
      for (int i = 0; i < 16; ++i) unpack2(run[i], ep[hf * 32 + 2 * i], ep[hf * 32 + 2 * i + 1]);
      float e0, e1;
      unpack2(e_run, e0, e1);
      if (hf == 0) ep[64] = e0 + e1;
      else ((float*)(smem + PS_OFF_E))[t * 128 + L] = e0 + e1;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 17) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  // whole rows of the sums, a pair's to both of its places
  float* st = state + (size_t)head * per_state;
  for (int rr = warp; rr < active * 128; rr += PS_THREADS / 32) {
    const int t = rr >> 7, L = rr & 127, b = L & 63, s = 2 * (tile0 + t) + (L >> 6);
    int row1, row2;
    if (s < D / 2 || (s == D / 2 && b < D / 2)) {
      const int o = (b + s) & (D - 1);
      row1 = b * D + o;
      row2 = o * D + b;
    } else if (s == D / 2) {
      if (b != D / 2) continue;
      row1 = row2 = D * D + D;
    } else {
      row1 = row2 = D * D + b;
    }
    const float* ep = (const float*)(smem + PS_OFF_EP) + rr * 65;
    for (int c = lane; c < 65; c += 32) {
      const float f = ep[c] + (c == 64 ? ((const float*)(smem + PS_OFF_E))[rr] : 0.f);
      st[(size_t)row1 * dvp + c] = f;
      if (row2 != row1) st[(size_t)row2 * dvp + c] = f;
    }
  }
}

// ---- operand copies: per step of the type A copies the three parts one after another ------------------------------
constexpr int C3_BYTES = 3 * A_BYTES;
__device__ __forceinline__ int a3_slice(int g, int oct, int part) {
  const int j = oct < 4 ? oct : 7 - oct;
  return 3 * TILE + ((g * 4 + j) * 3 + part) * A_STAGE + (oct < 4 ? 0 : ((j >> 1) + 1) * 4096);
}
__device__ __forceinline__ __nv_bfloat16 next_part(float& x) {       // the leading part of x, which keeps the rest
  const __nv_bfloat16 h = __float2bfloat16_rn(x);
  x -= __bfloat162float(h);
  return h;
}
__global__ void __launch_bounds__(256) copies3_kernel(const float* __restrict__ state, char* __restrict__ copies, int dvp,
                                                      size_t per_state) {
  __shared__ __align__(16) float blk[64][BLK_LD];
  const int m = blockIdx.y, b = blockIdx.x, t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const float* src = state + (size_t)m * per_state + (size_t)b * 64 * dvp;     // rows (b, a); b == 64: first-order rows
  char* dst = copies + (size_t)m * C3_BYTES;
  const int bb = b >> 4, na = b == 64 ? 64 : 16 * (bb + 1);
  for (int i = t; i < na * dvp; i += 256) (&blk[0][0])[i] = i % dvp < 65 ? src[i] : 0.f;        // dvp == BLK_LD
  __syncthreads();
  if (b == 64) {
    for (int i = t; i < 64 * 32; i += 256) {
      const int r = i >> 5, w = i & 31;
      uint32_t p[3];
      split3(pack2(blk[2 * w][r], blk[2 * w + 1][r]), p[0], p[1], p[2]);
#pragma unroll
      for (int part = 0; part < 3; ++part) *(uint32_t*)(dst + part * TILE + swz(r, w * 4)) = p[part];
    }
    return;
  }
  for (int i = warp; i < 4 * (bb + 1); i += 8) {      // eight features a, one half of the value columns
    const int oct = i >> 1, c = (i & 1) * 32 + lane;
    const float f = (oct >> 1) < bb ? 2.f : 1.f;
    uint32_t p[3][4];
#pragma unroll
    for (int e = 0; e < 4; ++e)
      split3(pack2(f * blk[oct * 8 + 2 * e][c], f * blk[oct * 8 + 2 * e + 1][c]), p[0][e], p[1][e], p[2][e]);
#pragma unroll
    for (int part = 0; part < 3; ++part)
      *(uint4*)(dst + a3_slice(c >> 4, b >> 3, part) + (oct >> 1) * 4096 + (oct & 1) * 2048 + ((c >> 3) & 1) * 1024 +
                (b & 7) * 128 + (c & 7) * 16) = make_uint4(p[part][0], p[part][1], p[part][2], p[part][3]);
  }
  if (t < na) {
    float x = blk[t][64];
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      const __nv_bfloat16 e = next_part(x);
      *(__nv_bfloat16*)(dst + part * TILE + swz(64 + b, t * 2)) = e;
      if ((t >> 4) < bb) *(__nv_bfloat16*)(dst + part * TILE + swz(64 + t, b * 2)) = e;
    }
  }
}

// ---- read-out -------------------------------------------------------------------------------------------------------
// The arrangement of the bf16 type A read-out: two token tiles with two T buffers each, two sets of four warps to a tile.
// Differences: three parts of everything (one x buffer, a ring of two stages of 60 KB), six products to a slice, the
// first-order and constant part waits in the output rows instead of shared memory, and the result is divided.
constexpr int R3_NS = 2, R3_STAGE = 3 * A_STAGE;
constexpr int R3_THREADS = 5 * 128, R3_REGS = 104, R3_REGS_REST = 64;
static_assert(4 * R3_REGS + R3_REGS_REST <= 5 * 96, "a register split above the launch's never starts");
constexpr int R3_OFF_X = 0;                               // [2 tiles][3 parts]
constexpr int R3_OFF_ST = 6 * TILE;
constexpr int R3_OFF_VEC = R3_OFF_ST + R3_NS * R3_STAGE;  // [warpgroup][2 items]: constant row [65], S1[:, 64] [64]
constexpr int R3_VEC = 132;
constexpr int R3_OFF_DEN = R3_OFF_VEC + 8 * R3_VEC * 4;   // [2 tiles][128]
constexpr int R3_OFF_BAR = R3_OFF_DEN + 2 * 128 * 4;
constexpr int R3_NBAR = 2 + 2 * R3_NS + 8;
constexpr int R3_OFF_TMEM = R3_OFF_BAR + R3_NBAR * 8;
constexpr int R3_SMEM = R3_OFF_TMEM + 16 + 1024;
static_assert(R3_SMEM <= 227 * 1024, "shared memory");

__global__ void __launch_bounds__(R3_THREADS, 1)
readout3_kernel(const __grid_constant__ CUtensorMap tmX, const RdArgs a, const int ratio) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + R3_OFF_BAR;
  // barriers: x_full | x_empty | st_full[NS] | st_empty[NS] | t_full[tile][buf] | t_free[tile][buf]
  const uint32_t BAR_XFULL = bar0, BAR_XEMPTY = bar0 + 8u;
  auto BAR_FULL = [&](int s) { return bar0 + 8u * (2 + s); };
  auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (2 + R3_NS + s); };
  auto BAR_TFULL = [&](int t, int b) { return bar0 + 8u * (2 + 2 * R3_NS + 2 * t + b); };
  auto BAR_TFREE = [&](int t, int b) { return bar0 + 8u * (6 + 2 * R3_NS + 2 * t + b); };
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + R3_OFF_TMEM);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    mbar_init(BAR_XFULL, 1);
    mbar_init(BAR_XEMPTY, 16 + 2);
    for (int s = 0; s < R3_NS; ++s) { mbar_init(BAR_FULL(s), 1); mbar_init(BAR_EMPTY(s), 2); }
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
    regs_down<R3_REGS_REST>();
    if (warp == 16) {
      // ---------------- producer ----------------
      if (lane == 0) {
        tma_prefetch_desc(&tmX);
        bool ok = true;
        int st = 0, k = 0;            // running number of the ring step and of the item
        for (Walk w(a); ok && w.more(); w.next(a), ++k) {
          const int tok0 = w.tok0(a);
          if (!mbar_wait(BAR_XEMPTY, (uint32_t)((k & 1) ^ 1))) { report(90); break; }
          mbar_expect_tx(BAR_XFULL, 6 * TILE);
          for (int t = 0; t < 2; ++t)     // rows past the last query read as zero
            for (int part = 0; part < 3; ++part)
              tma_load_3d(sbase + R3_OFF_X + (3 * t + part) * TILE, &tmX, BAR_XFULL, part * D, tok0 + t * 128, w.head);
          const char* src = a.copies + (size_t)(w.head / ratio) * C3_BYTES;
          for (int n = 0; n < A_STEPS; ++n, ++st) {
            const int s = st % R3_NS;
            if (!mbar_wait(BAR_EMPTY(s), (((st / R3_NS) & 1) ^ 1))) { report(91); ok = false; break; }
            const uint32_t bytes = n == 0 ? 3 * TILE : R3_STAGE;
            mbar_expect_tx(BAR_FULL(s), bytes);
            bulk_load(sbase + R3_OFF_ST + s * R3_STAGE, src, bytes, BAR_FULL(s));
            src += bytes;
          }
        }
      }
      __syncwarp();
    } else if (warp < 19) {
      // ---------------- MMA issuers: one per tile ----------------
      const int t = warp - 17;
      constexpr uint32_t idesc = idesc_bf16(128, 128, 0, 0), idesc64 = idesc_bf16(128, 64, 0, 0);
      const uint32_t st0 = ((sbase + R3_OFF_ST) & 0x3FFFFu) >> 4;
      const uint32_t x_lo = desc_lo(sbase + R3_OFF_X + 3 * t * TILE, 16);
      bool ok = true;
      int st = 0, k = 0;
      for (int left = Walk(a).left; ok && left > 0; --left, ++k) {
        if (!mbar_wait_warp(BAR_XFULL, (uint32_t)(k & 1))) { report(92); break; }
        for (int n = 0; ok && n < A_STEPS; ++n, ++st) {
          const int s = st % R3_NS, deep = (((n - 1) & 3) >> 1) + 1;    // K steps of the step's first slice
          if (!mbar_wait_warp(BAR_FULL(s), (uint32_t)((st / R3_NS) & 1))) { report(93); ok = false; break; }
          const uint32_t b0 = st0 + (uint32_t)s * (R3_STAGE >> 4);
          for (int buf = 0; buf < 2; ++buf) {
            if (!mbar_wait_warp(BAR_TFREE(t, buf), (uint32_t)((st & 1) ^ 1))) { report(94); ok = false; break; }
            tc_fence_after();
            const uint32_t d = tmem + t * 256 + buf * 128;
            const int steps = buf ? 5 - deep : deep;
            if (elect_one()) {
#pragma unroll
              for (int i = 0; i < 6; ++i) {
                constexpr int kX[6] = {2, 0, 1, 1, 0, 0}, kS[6] = {0, 2, 1, 0, 1, 0};     // small products first
                const uint32_t x = x_lo + kX[i] * (TILE >> 4);
                if (n == 0)          // buffer 0: x . S1, buffer 1: x . E
                  umma_ss_k64(d, x, (b0 + kS[i] * (TILE >> 4) + (buf ? 8192u >> 4 : 0u)) | (1u << 16), idesc64, i > 0);
                else
                  mma_steps(d, x, (b0 + kS[i] * (A_STAGE >> 4) + (buf ? (uint32_t)deep * (4096 >> 4) : 0u)) | ((2048u >> 4) << 16),
                            idesc, steps, i > 0);
              }
              umma_commit(BAR_TFULL(t, buf));
              if (buf) {
                umma_commit(BAR_EMPTY(s));
                if (n == A_STEPS - 1) umma_commit(BAR_XEMPTY);
              }
            }
            __syncwarp();
          }
        }
      }
    }
  } else {
    // ---------------- contraction ----------------
    regs_up<R3_REGS>();
    const int wg = warp >> 2, t = wg >> 1, h = wg & 1, qd = warp & 3;
    const int row = qd * 32 + lane;                        // token row in the tile, TMEM lane
    const uint32_t tb = tmem + t * 256 + ((uint32_t)(qd * 32) << 16);
    float* vecs = (float*)(smem + R3_OFF_VEC) + wg * 2 * R3_VEC;
    float* dens = (float*)(smem + R3_OFF_DEN) + t * 128;
    const uint32_t xrow = sbase + R3_OFF_X + 3 * t * TILE + row * 128, xs = (uint32_t)(row & 7) << 4;
    // features 8 oct .. 8 oct + 7 of the token, the sums of their parts
    auto features = [&](int oct, float (&x)[8]) {
#pragma unroll
      for (int part = 0; part < 3; ++part) {
        const uint4 w = lds128(xrow + part * TILE + (((uint32_t)oct << 4) ^ xs));
        const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          x[2 * e] = part == 0 ? bf_lo(ww[e]) : x[2 * e] + bf_lo(ww[e]);
          x[2 * e + 1] = part == 0 ? bf_hi(ww[e]) : x[2 * e + 1] + bf_hi(ww[e]);
        }
      }
    };
    // what an item needs from global memory is asked for one item ahead
    auto first_rows = [&](const Walk& w) { return a.state + (size_t)(w.head / ratio) * a.per_state + (size_t)(64 * 64) * a.dvp; };
    auto const_of = [&](const Walk& w) { return w.more() && row <= 64 ? __ldg(first_rows(w) + (size_t)64 * a.dvp + row) : 0.f; };
    auto norm_of = [&](const Walk& w) { return w.more() && h && row < 64 ? __ldg(first_rows(w) + (size_t)row * a.dvp + 64) : 0.f; };
    // (past the end the last head's words again: without a branch the loop keeps 16 bytes in local memory instead of 132, 1.5 %)
    auto q_of = [&](const Walk& w) { return a.stat_q[min(w.head, a.heads - 1)]; };
    auto k_of = [&](const Walk& w) { return a.stat_k[min(w.head, a.heads - 1) / ratio]; };
    Walk w(a);
    float s0next = const_of(w), n1next = norm_of(w);
    stat_t qnext = q_of(w), knext = k_of(w);
    bool ok = true;
    int st = 0, k = 0;
    auto full = [&](int buf) {
      if (ok && !mbar_wait(BAR_TFULL(t, buf), (uint32_t)(st & 1))) { report(96); ok = false; }
      tc_fence_after();
    };
    auto release = [&](int buf) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_TFREE(t, buf));
    };
    for (; w.more(); ++k) {
      // what pow2_of has left of the scales of the queries and of the keys
      const float c = beyond_pow2(stat_scale(&qnext, 0, a.lim)) * beyond_pow2(stat_scale(&knext, 0, a.lim));
      const float A1 = a.a1 * c, A2 = a.a2 * c * c;
      const int tok = w.tok0(a) + t * 128 + row;
      const bool tok_ok = tok < a.n;
      const size_t grow = (size_t)w.head * a.n + (tok_ok ? tok : 0);
      float* out = a.out + grow * D;
      float* vec = vecs + (k & 1) * R3_VEC;  // the set's warps are done with the one of two items ago since the last barrier
      if (row <= 64) vec[row] = s0next;
      if (h && row < 64) vec[68 + row] = n1next;
      w.next(a);
      s0next = const_of(w);
      n1next = norm_of(w);
      qnext = q_of(w);
      knext = k_of(w);
      asm volatile("bar.sync %0, 128;" ::"r"(1 + wg) : "memory");
      if (ok && !mbar_wait(BAR_XFULL, (uint32_t)(k & 1))) { report(95); ok = false; }
      // ---- step 0, buffer 0: x . S1; this set puts the value columns it will write into the output rows
      full(0);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int cc = (2 * i + h) * 8;
        uint32_t t8[8];
        tmem_ld8(tb + cc, t8);
        tmem_wait_ld(t8);
        if (i == 3) release(0);
#pragma unroll
        for (int e = 0; e < 8; ++e) t8[e] = __float_as_uint(fmaf(A1, __uint_as_float(t8[e]), a.a0 * vec[cc + e]));
        if (ok && tok_ok) stg32(out + cc, t8, a.wide_io != 0);
      }
      // ---- buffer 1: x . E, the normaliser, by set 1
      full(1);
      if (h == 0) {
        release(1);
      } else {
        uint32_t tv[64];
        tmem_ld64(tb + 128, tv);
        tmem_wait_ld(tv);
        release(1);
        float second[4] = {0.f, 0.f, 0.f, 0.f}, first[2] = {0.f, 0.f};
#pragma unroll
        for (int v = 0; v < 8; ++v) {
          float x[8];
          features(v, x);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            second[e & 3] = fmaf(x[e], __uint_as_float(tv[v * 8 + e]), second[e & 3]);
            first[e & 1] = fmaf(x[e], vec[68 + v * 8 + e], first[e & 1]);
          }
        }
        const float den = fmaf(A2, (second[0] + second[1]) + (second[2] + second[3]), fmaf(A1, first[0] + first[1], a.a0 * vec[64]));
        dens[row] = den;
        if (ok && a.den && tok_ok) a.den[grow] = den;
      }
      ++st;
      // (the next item's denominators are written after this set has taken part in all steps between)
      asm volatile("bar.sync %0, 256;" ::"r"(5 + t) : "memory");
      const float den = dens[row];
      // ---- steps 1..16: eight value columns over the eight octets of features b
#pragma unroll 1
      for (int g = 0; g < 4; ++g) {
        uint64_t acc[8] = {0ull, 0ull, 0ull, 0ull, 0ull, 0ull, 0ull, 0ull};   // even and odd features apart
        auto slice = [&](int buf, int oct) {
          uint32_t tv[64];
          full(buf);
          tmem_ld64(tb + h * 64 + buf * 128, tv);
          float x[8];
          features(oct, x);
          tmem_wait_ld(tv);
          release(buf);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint64_t x0 = pack2(x[2 * i], x[2 * i]), x1 = pack2(x[2 * i + 1], x[2 * i + 1]);
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
        if (ok && tok_ok) {
          const int cc = (2 * g + h) * 8;
          uint32_t o[8];
          ldg32(out + cc, o, a.wide_io != 0);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float lo, hi;
            unpack2(add2(acc[e], acc[4 + e]), lo, hi);
            o[2 * e] = __float_as_uint(fmaf(A2, lo, __uint_as_float(o[2 * e])) / den);
            o[2 * e + 1] = __float_as_uint(fmaf(A2, hi, __uint_as_float(o[2 * e + 1])) / den);
          }
          stg32(out + cc, o, a.wide_io != 0);
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_XEMPTY);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

size_t up256(size_t x) { return (x + 255) / 256 * 256; }
struct Layout { size_t q3, v3, state, copies, bytes; };
Layout layout(const fastmax_problem& p) {
  const MomentDims m = moment_dims(64);
  Layout l;
  l.q3 = 0;
  l.v3 = up256((size_t)p.bh * p.nq * 64 * 6);
  l.state = l.v3 + up256((size_t)p.bhkv * p.nk * 64 * 6);
  l.copies = l.state + up256((size_t)p.bhkv * m.f * m.dvp * 4);
  l.bytes = l.copies + (size_t)p.bhkv * C3_BYTES;
  return l;
}

}  // namespace

int split_moments_status(int* out, cudaStream_t stream) {
  FM_CUDA_TRY(cudaMemcpyFromSymbolAsync(out, g_smom_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
int split_moments_status_reset(cudaStream_t stream) {
  const int zero = 0;
  FM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_smom_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}

// The score form costs 1.05 ps a pair.  The moment form: 1.45 ns a query row, 2.1 us per block of 64 keys and wave of CTAs
// (nine a key head), and its launches.  Measured, all kernels of a forward, us, score / moment:
//   64 heads: 6267 / 2471 at 10 000, 1357 / 1106 at 4200, 1090 / 968 at 3600; 16: 556 / 393 at 5000; 8: 875 / 541 at 10 000,
//   569 / 411 at 7500, 323 / 354 at 6000; 2: 1101 / 791 at 20 000; 1: 1065 / 1144 at 30 000
//   32 on 8 key heads: 585 / 400 at 4000, 397 / 315 at 3000; 8 on 2, 40 000 queries: 790 / 609 for 2000 keys
//
// And only where the terms of f(s) = a0 + a1 s + a2 s^2 cannot cancel to less than a fifth of their sizes.  The sums over
// feature pairs are rounded relative to a2 |q|^2 |k|^2, whatever the score is; the score form's are relative to f.  With
// normalised rows |s| <= |q| |k| <= lim^2, which bounds the loss; without nothing does.  2-norm errors against float64, 64 heads
// x 4097, score / moment: keys that share a direction of norm 80 which the queries do not see, not normalised, 4.4e-7 / 1.6e-5,
// of norm 800 3.9e-6 / 1.6e-3; normalised, the usual coefficients (1, 1, 0.5), N(0,1) 1.8e-7 / 1.7e-7, q and k along one direction
// 1.9e-7 / 1.2e-7, along opposite ones (where f is a fifth) 1.9e-7 / 3.8e-7; (1, 0, -1), a tenth, 2.0e-7 / 3.1e-7; (1, -1.5, 0.5),
// no bound, 7.0e-7 / 4.8e-6; (1, 1, 0.5) and lim 4, a hundredth and less, 1.9e-7 / 4.0e-7.
static bool terms_hardly_cancel(const fastmax_problem& p) {
  if (!p.normalize) return false;
  const double a0 = p.a0, a1 = p.a1, a2 = p.a2, most = (double)p.lim * p.lim;
  auto f = [&](double s) { return a0 + s * (a1 + s * a2); };
  double least = f(-most) < f(most) ? f(-most) : f(most);
  if (a2 > 0 && fabs(a1) < 2 * a2 * most && f(-a1 / (2 * a2)) < least) least = f(-a1 / (2 * a2));
  return fabs(a0) + most * (fabs(a1) + most * fabs(a2)) <= 5 * least;
}
bool split_moments_faster(const fastmax_problem& p) {
  if (!dense_split_supports(p) || p.mask || p.p != 2 || p.d != 64 || p.bh % p.bhkv || p.bhkv > 65535) return false;
  if (!terms_hardly_cancel(p)) return false;
  const double us_pairs = 1.05e-6 * p.bh * p.nq * p.nk;
  const double us_moment = 60 + 1.45e-3 * p.bh * p.nq + ((9 * p.bhkv + 147) / 148) * (p.nk / 64.0) * 2.1;
  return us_moment < us_pairs;
}
size_t split_moments_bytes(const fastmax_problem& p) { return layout(p).bytes; }

int split_moments_forward(const Ctx& c, const void* q, const void* k, const void* v, const stat_t* stats, const FwdOut& o,
                          void* workspace) {
  const fastmax_problem& p = c.p;
  if (p.bh == 0 || p.nq == 0) return FASTMAX_OK;
  const Layout l = layout(p);
  const MomentDims m = moment_dims(64);
  char* ws = (char*)workspace;
  float* state = (float*)(ws + l.state);
  int rc;
  if ((rc = split3_scaled_q(c, q, ws + l.q3, v, ws + l.v3, stats))) return rc;
  CUtensorMap tv, tx;
  if ((rc = tma_map_bf16(&tv, ws + l.v3, p.bhkv, p.nk, 3 * 64, TB))) return rc;
  if ((rc = tma_map_bf16(&tx, ws + l.q3, p.bh, p.nq, 3 * 64, 128))) return rc;
  FM_CUDA_TRY(cudaFuncSetAttribute(pair_sums_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PS_SMEM));
  const dim3 sums((PS_TILES + 1) / 2, p.bhkv);
  FM_LAUNCH("fm_split_pair_sums", c.stream, (pair_sums_kernel<<<sums, PS_THREADS, PS_SMEM, c.stream>>>(
                                                tv, (const float*)k, stats + p.bh, p.lim, state, p.nk, m.dvp, (size_t)m.f * m.dvp)));
  FM_CUDA_TRY(cudaGetLastError());
  const dim3 grid(65, p.bhkv);
  FM_LAUNCH("fm_split_state_copies", c.stream,
            (copies3_kernel<<<grid, 256, 0, c.stream>>>(state, ws + l.copies, m.dvp, (size_t)m.f * m.dvp)));
  FM_CUDA_TRY(cudaGetLastError());
  RdArgs a = {};
  a.copies = ws + l.copies;
  a.state = state;
  a.out = (float*)o.out;
  a.den = o.den;
  a.stat_q = stats;
  a.stat_k = stats + p.bh;
  a.a0 = p.a0; a.a1 = p.a1; a.a2 = p.a2; a.lim = p.lim;
  a.per_state = (size_t)m.f * m.dvp;
  a.dvp = m.dvp;
  a.heads = p.bh;
  a.n = p.nq;
  a.groups = (p.nq + 255) / 256;
  a.items = p.bh * a.groups;
  a.wide_io = ((uintptr_t)o.out & 31) == 0;
  FM_CUDA_TRY(cudaFuncSetAttribute(readout3_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, R3_SMEM));
  const unsigned ctas = (unsigned)(a.items < 148 ? a.items : 148);
  FM_LAUNCH("fm_split_readout", c.stream, (readout3_kernel<<<ctas, R3_THREADS, R3_SMEM, c.stream>>>(tx, a, p.bh / p.bhkv)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

}  // namespace fm
