// First-order part of the moment-state form on the tcgen05 tensor cores (bf16 operands,
// fp32 accumulation), head dimension 64 or 128.  This is the whole computation when p = 1
// -- the case the reference's current CUDA kernels implement (fastmax_cuda_forward.cu:
// 25-197, fastmax_cuda_backward.cu:26-871: moments Sum v, Sum k, Sum k (x) v and their
// gradient counterparts) -- and the first-order rows of the state when p = 2.
//
//   state    S1[a][c] = sum_j y_j[a] z_j[c]          one MMA per 128-token tile: both operands
//                                                     are the raw token tiles TMA delivered
//                                                     (A = Y^T and B = Z, both MN-major)
//            S1[a][D] = sum_j y_j[a] e_j,  S0[c] = sum_j z_j[c],  S0[D] = sum_j e_j
//                                                     small vector sums on the CUDA cores
//   readout A  r_i[c] = A1 sum_a x_i[a] S1[a][c] + A0 S0[c]           (c <= D; c = D: normaliser)
//   readout B  r_i[a] = A1 (sum_c u_i[c] S1[a][c] + e_i S1[a][D])
//                                                     one GEMM of the raw token tile against a
//                                                     bf16 copy of S1 (MN-major B for type A,
//                                                     the same bytes K-major for type B)
// All of it is bound by HBM traffic: every token row is read once per stage.
#include <cstdlib>

#include "fm_common.cuh"
#include "fm_sm100.cuh"

namespace fm {

__device__ int g_ftc_status = 0;  // first protocol error seen by a kernel of this file

namespace {
using namespace sm100;

__device__ __forceinline__ void report(int code) { atomicCAS(&g_ftc_status, 0, code); }

// 16 bytes from shared memory by shared-window address (keeps the epilogue's vector reads off the generic path)
__device__ __forceinline__ uint4 lds128u(uint32_t saddr) {
  uint4 r;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(saddr));
  return r;
}
__device__ __forceinline__ float4 lds128f(uint32_t saddr) {
  float4 r;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "r"(saddr));
  return r;
}

constexpr int F1_THREADS = 192;  // warp 0: TMA producer, warp 1: MMA issuer, warps 2-5: vector sums, epilogue

// =====================================================================================
// state build
// =====================================================================================
struct F1StateArgs {
  const void* y;       // (heads, n, D) bf16 feature source (k, or q)
  const void* z;       // (heads, n, D) bf16 values (v, or grad_out/den)
  const float* dvec;   // e_j = -dvec[j] when not null, else 1
  float* state;        // (heads, nchunk, rows, DVP) fp32; rows f_lin .. f_lin + D are written
  int n, chunk, nchunk, dvp, rows, f_lin;   // f_lin: stored index of the first first-order row
  int skip_chunk;      // this chunk's state is not wanted (-1: none)
};

template <int DD>
struct F1S {
  static constexpr int NSUB = DD / 64;
  // Tokens per tile and ring depth are chosen so that a CTA needs 96 KB of shared memory: two CTAs per SM,
  // each with two of its three 32 KB stages in flight while the third is consumed, keep enough bytes on the
  // way from HBM (one CTA with two 64 KB stages reached 58 % of the copy bandwidth).
  static constexpr int TOK = (DD == 128) ? 64 : 128;
  static constexpr int NS = 3;
  static constexpr int SUBTILE = TOK * 128;       // TOK tokens x 64 bf16
  static constexpr int TILE = NSUB * SUBTILE;     // one operand tile: TOK tokens x DD bf16
  static constexpr int STAGE = 2 * TILE;          // Y then Z
  static constexpr int VROW = 2 * DD + 4;         // a warp's sums: z [DD], y e [DD], e
  static constexpr int OFF_VEC = NS * STAGE;
  static constexpr int OFF_BAR = OFF_VEC + 4 * VROW * 4;
  static constexpr int NBAR = 2 * NS + 1;
  static constexpr int OFF_TMEM = OFF_BAR + NBAR * 8;
  static constexpr int SMEM = OFF_TMEM + 16 + 1024;
};

template <int DD>
__global__ void __launch_bounds__(F1_THREADS, 2)
first_state_kernel(const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmZ,
                   const F1StateArgs a) {
  using C = F1S<DD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + C::OFF_BAR;
  auto BAR_FULL = [&](int s) { return bar0 + 8u * s; };
  auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (C::NS + s); };
  auto BAR_DONE = [&]() { return bar0 + 8u * (2 * C::NS); };
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + C::OFF_TMEM);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hc = blockIdx.x, head = hc / a.nchunk, chunk = hc % a.nchunk;
  if (chunk == a.skip_chunk) return;
  const int t_begin = chunk * a.chunk, t_end = min(a.n, t_begin + a.chunk);
  constexpr int TOK = C::TOK;
  const int nblk = (t_end - t_begin + TOK - 1) / TOK;

  if (tid == 0) {
    // a stage is free when the MMAs that read it are done and the vector sums have read it
    for (int s = 0; s < C::NS; ++s) { mbar_init(BAR_FULL(s), 1); mbar_init(BAR_EMPTY(s), 1 + 4); }
    mbar_init(BAR_DONE(), 1);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(smem_u32((const void*)tmem_slot), 128);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) { tma_prefetch_desc(&tmY); tma_prefetch_desc(&tmZ); }
    for (int k = 0; k < nblk; ++k) {
      const int s = k % C::NS;
      if (!mbar_wait(BAR_EMPTY(s), (((k / C::NS) & 1) ^ 1))) { report(41); break; }
      if (lane == 0) {
        mbar_expect_tx(BAR_FULL(s), C::STAGE);
        const uint32_t dst = sbase + s * C::STAGE;
        for (int sub = 0; sub < C::NSUB; ++sub) {
          tma_load_3d(dst + sub * C::SUBTILE, &tmY, BAR_FULL(s), sub * 64, t_begin + k * TOK, head);
          tma_load_3d(dst + C::TILE + sub * C::SUBTILE, &tmZ, BAR_FULL(s), sub * 64, t_begin + k * TOK, head);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // M = 128 rows of the accumulator; with DD = 64 the second 64-row block of A is the Z
      // tile that follows Y in the stage (valid memory), and those rows are never read back
      constexpr uint32_t idesc = idesc_bf16(128, DD, 1, 1);
      bool ok = true;
      for (int k = 0; ok && k < nblk; ++k) {
        const int s = k % C::NS;
        if (!mbar_wait(BAR_FULL(s), (uint32_t)((k / C::NS) & 1))) { report(42); ok = false; break; }
        tc_fence_after();
        const uint32_t y_lo = desc_lo(sbase + s * C::STAGE, C::SUBTILE);
        const uint32_t z_lo = desc_lo(sbase + s * C::STAGE + C::TILE, C::SUBTILE);
        umma_ss_mn_steps<TOK / 16>(tmem, y_lo, z_lo, idesc, k > 0 ? 1u : 0u);
        umma_commit(BAR_EMPTY(s));
      }
      if (ok) umma_commit(BAR_DONE());
    }
    __syncwarp();
  } else {
    // ---- vector sums over the chunk's tokens, read from the tiles TMA delivered ----
    // 16 bytes a thread, a row's pieces side by side: element (row r, column c) of a 64-column sub-tile sits at
    // r*128 + (((c>>3) ^ (r&7))<<4) + (c&7)*2.  (A pair of columns a thread through the generic path, the sums of threads
    // added by atomics, bound the kernel: 404 us for 256 heads x 16384 x 128 and 76 for 256 x 4096 x 64; 356 and 63 now.)
    const int t = tid - 64;                       // 0..127
    constexpr int LPR = DD / 8, RPS = 128 / LPR, STEPS = TOK / RPS;
    static_assert(RPS % 8 == 0, "a thread's rows have one swizzle");
    const int sub_r = t / LPR, piece = t % LPR;
    const uint32_t at0 = sbase + (uint32_t)((piece >> 3) * C::SUBTILE + sub_r * 128 + (((piece & 7) ^ (sub_r & 7)) << 4));
    const float* dv = a.dvec ? a.dvec + (size_t)head * a.n : nullptr;
    uint64_t sz[4] = {0, 0, 0, 0}, sye[4] = {0, 0, 0, 0};
    float se = 0.f, ev[STEPS];
    auto fetch = [&](int k) {                     // e of this thread's rows of tile k, asked for a tile ahead
#pragma unroll
      for (int st = 0; st < STEPS; ++st) {
        const int tok = t_begin + k * TOK + st * RPS + sub_r;
        ev[st] = tok < t_end ? (dv ? -__ldg(dv + tok) : 1.f) : 0.f;
      }
    };
    fetch(0);
    bool ok = true;
    for (int k = 0; k < nblk; ++k) {
      const int s = k % C::NS;
      float e[STEPS];
#pragma unroll
      for (int st = 0; st < STEPS; ++st) e[st] = ev[st];
      fetch(k + 1);
      if (!mbar_wait(BAR_FULL(s), (uint32_t)((k / C::NS) & 1))) { report(46); ok = false; break; }
      const uint32_t yt = at0 + s * C::STAGE, zt = yt + C::TILE;
#pragma unroll
      for (int st = 0; st < STEPS; ++st) {        // (rows past the end of the sequence hold zeros)
        const uint4 yv = lds128u(yt + st * (RPS * 128)), zv = lds128u(zt + st * (RPS * 128));
        const uint32_t yw[4] = {yv.x, yv.y, yv.z, yv.w}, zw[4] = {zv.x, zv.y, zv.z, zv.w};
        const uint64_t e2 = pack2(e[st], e[st]);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          sz[x] = add2(sz[x], pack2u(zw[x] << 16, zw[x] & 0xFFFF0000u));
          sye[x] = fma2(pack2u(yw[x] << 16, yw[x] & 0xFFFF0000u), e2, sye[x]);
        }
        se += e[st];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_EMPTY(s));
    }
    // the rows of a warp, then (in the epilogue) the warps, in a fixed order
    float* const sums = (float*)(smem + C::OFF_VEC);
    float* const mine = sums + (warp - 2) * C::VROW;
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      float f[4];
      unpack2(sz[x], f[0], f[1]);
      unpack2(sye[x], f[2], f[3]);
#pragma unroll
      for (int k = LPR; k < 32; k <<= 1)
#pragma unroll
        for (int y = 0; y < 4; ++y) f[y] += __shfl_xor_sync(0xffffffffu, f[y], k);
      if (lane < LPR) {
        *(float2*)(mine + piece * 8 + 2 * x) = make_float2(f[0], f[1]);
        *(float2*)(mine + DD + piece * 8 + 2 * x) = make_float2(f[2], f[3]);
      }
    }
#pragma unroll
    for (int k = LPR; k < 32; k <<= 1) se += __shfl_xor_sync(0xffffffffu, se, k);
    if (lane == 0) mine[2 * DD] = se;
    // named barrier among the four epilogue warps only
    asm volatile("bar.sync 1, 128;" ::: "memory");
    auto vsum = [&](int i) { return (sums[i] + sums[C::VROW + i]) + (sums[2 * C::VROW + i] + sums[3 * C::VROW + i]); };
    // ---- epilogue ----
    if (ok && !mbar_wait(BAR_DONE(), 0)) { report(43); ok = false; }
    tc_fence_after();
    float* st = a.state + (size_t)hc * a.rows * a.dvp;
    const int qd = warp & 3;                      // TMEM lane quarter this warp may read
    if (ok && qd * 32 < DD) {
      const int arow = qd * 32 + lane;            // accumulator row = feature index a
      float* dst = st + (size_t)(a.f_lin + arow) * a.dvp;
#pragma unroll 1
      for (int hcol = 0; hcol < DD / 64; ++hcol) {
        uint32_t tv[64];
        tmem_ld64(tmem + ((uint32_t)(qd * 32) << 16) + hcol * 64, tv);
        tmem_wait_ld(tv);
#pragma unroll
        for (int e4 = 0; e4 < 16; ++e4)
          ((float4*)(dst + hcol * 64))[e4] = make_float4(__uint_as_float(tv[4 * e4]), __uint_as_float(tv[4 * e4 + 1]),
                                                         __uint_as_float(tv[4 * e4 + 2]), __uint_as_float(tv[4 * e4 + 3]));
      }
      dst[DD] = vsum(DD + arow);
      for (int cc = DD + 1; cc < a.dvp; ++cc) dst[cc] = 0.f;
    }
    // constant row: [sum z | sum e | 0]
    float* crow = st + (size_t)(a.f_lin + DD) * a.dvp;
    for (int cc = t; cc < a.dvp; cc += 128) crow[cc] = (cc < DD) ? vsum(cc) : (cc == DD ? vsum(2 * DD) : 0.f);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 128);
  }
}


// =====================================================================================
// read-out
// =====================================================================================
struct F1ReadArgs {
  const void* x;        // (heads, n, D) bf16 tokens (type A: the MMA operand; both: normaliser dot)
  const float* uvec;    // type B: e_i = -uvec[i] when not null, else 1
  const float* state;   // fp32 states (first-order rows are read for the vector terms)
  float* o_add;         // (heads, n, D) fp32 result
  float* den_add;       // type A: (heads, n) normaliser part, may be null
  const stat_t* stat_q;
  const stat_t* stat_k;
  float a0, a1, lim;
  int n, chunk, nchunk, per_chunk, dvp, rows, f_lin, type_b, accumulate;
  int run;              // tiles per CTA (all of one state)
  // final != 0: the read-out is the whole result (p = 1, unmasked): write bf16 rows to out_final
  // instead of fp32 to o_add.  1: type A divided by its normaliser (which goes to den_final);
  // 2: plain rounding; the per-head dot with x is added to *dots when dots is not null.
  int final;
  void* out_final;
  float* den_final;
  float* dots;
  int wide_io;          // out_final / o_add / x are 32-byte aligned: 32-byte accesses in the epilogue
  int zero_chunk;       // per-chunk mode: the tokens of this chunk read an empty state (-1: none)
};

template <int DD>
struct F1R {
  static constexpr int NSUB = DD / 64;
  static constexpr int TILE = NSUB * 16384;        // 128 tokens x DD bf16
  static constexpr int SMAT = DD * DD * 2;         // bf16 copy of S1, NSUB sub-tiles of DD rows x 64
  static constexpr int OFF_S = 2 * TILE;           // two token-tile stages first
  static constexpr int OFF_VEC = OFF_S + SMAT;     // normaliser column [DD] | constant row [DD + 1]
  static constexpr int OFF_BAR = OFF_VEC + (2 * DD + 8) * 4;
  static constexpr int NBAR = 9;                   // s_full | t_full[2] | t_empty[2] | a_full[2] | a_free[2]
  static constexpr int OFF_TMEM = OFF_BAR + NBAR * 8;
  static constexpr int SMEM = OFF_TMEM + 16 + 1024;
  static constexpr int TCOLS = 2 * DD;             // two accumulators
};

// One CTA reads out a run of consecutive 128-token tiles that share one state: the bf16 state
// copy is loaded once, token tiles stream through two stages, and two TMEM accumulators let the
// epilogue of a tile overlap the load and the product of the next one.
template <int DD>
__global__ void __launch_bounds__(F1_THREADS, 2)
first_readout_kernel(const __grid_constant__ CUtensorMap tmT, const __grid_constant__ CUtensorMap tmS,
                     const F1ReadArgs a) {
  using C = F1R<DD>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + C::OFF_BAR;
  const uint32_t BAR_SF = bar0;
  auto BAR_TF = [&](int b) { return bar0 + 8u * (1 + b); };
  auto BAR_TE = [&](int b) { return bar0 + 8u * (3 + b); };
  auto BAR_AF = [&](int b) { return bar0 + 8u * (5 + b); };
  auto BAR_AE = [&](int b) { return bar0 + 8u * (7 + b); };
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + C::OFF_TMEM);
  float* ncol = (float*)(smem + C::OFF_VEC);       // S1[a][DD], a < DD
  float* crow = ncol + DD;                         // constant row, DD + 1 values
  const uint32_t ncol_s = sbase + C::OFF_VEC;      // the same vectors by shared-window address
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles = (a.n + 127) / 128;
  const int runs = (tiles + a.run - 1) / a.run;
  const int head = blockIdx.x / runs;
  const int tile0 = (blockIdx.x % runs) * a.run;
  const int nt = min(a.run, tiles - tile0);        // tiles of this run
  const int mat = head * (a.per_chunk ? a.nchunk : 1) + (a.per_chunk ? (tile0 * 128) / a.chunk : 0);
  if (a.per_chunk && (tile0 * 128) / a.chunk == a.zero_chunk) {
    // the run lies in one chunk, whose state is empty: the result is zero -- nothing to add, or zeros to write
    if (!a.accumulate) {
      const int row0 = tile0 * 128, rows = min(nt * 128, a.n - row0);
      for (int i = tid; i < rows * (DD / 4); i += F1_THREADS)
        *(float4*)(a.o_add + ((size_t)head * a.n + row0) * DD + (size_t)i * 4) = make_float4(0.f, 0.f, 0.f, 0.f);
      if (!a.type_b && a.den_add)
        for (int i = tid; i < rows; i += F1_THREADS) a.den_add[(size_t)head * a.n + row0 + i] = 0.f;
    }
    return;
  }

  if (tid == 0) {
    mbar_init(BAR_SF, 1);
    for (int b = 0; b < 2; ++b) {
      mbar_init(BAR_TF(b), 1);
      // a stage is free once the product that read it is done and, where the epilogue reads x from it for
      // the normaliser dot (type A), once its four warps have done so
      mbar_init(BAR_TE(b), (!a.type_b && (a.den_add || a.final == 1)) ? 5 : 1);
      mbar_init(BAR_AF(b), 1);
      mbar_init(BAR_AE(b), 4);
    }
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(smem_u32((const void*)tmem_slot), C::TCOLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ================= TMA producer =================
    if (lane == 0) {
      mbar_expect_tx(BAR_SF, C::SMAT);
      for (int sub = 0; sub < C::NSUB; ++sub)
        tma_load_3d(sbase + C::OFF_S + sub * (DD * 128), &tmS, BAR_SF, sub * 64, 0, mat);
    }
    for (int i = 0; i < nt; ++i) {
      const int b = i & 1;
      if (!mbar_wait(BAR_TE(b), (uint32_t)(((i >> 1) & 1) ^ 1))) { report(47); break; }
      if (lane == 0) {
        mbar_expect_tx(BAR_TF(b), C::TILE);
        for (int sub = 0; sub < C::NSUB; ++sub)
          tma_load_3d(sbase + b * C::TILE + sub * 16384, &tmT, BAR_TF(b), sub * 64, (tile0 + i) * 128, head);
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer (whole warp, one elected lane issues) =================
    bool ok = mbar_wait_warp(BAR_SF, 0);
    if (!ok) report(44);
    for (int i = 0; ok && i < nt; ++i) {
      const int b = i & 1;
      if (!mbar_wait_warp(BAR_TF(b), (uint32_t)((i >> 1) & 1))) { report(44); break; }
      if (!mbar_wait_warp(BAR_AE(b), (uint32_t)(((i >> 1) & 1) ^ 1))) { report(48); break; }
      tc_fence_after();
      const uint32_t t_lo = desc_lo(sbase + b * C::TILE, 16);
      const uint32_t acc = tmem + b * DD;
      if (elect_one()) {
        if (a.type_b) {
          // acc[i][a'] = sum_c u_i[c] S1[a'][c]: B = S1 rows a' with c contiguous (K-major)
          constexpr uint32_t idesc = idesc_bf16(128, DD, 0, 0);
          const uint32_t s_lo = desc_lo(sbase + C::OFF_S, 16);
#pragma unroll
          for (int sub = 0; sub < C::NSUB; ++sub)
            umma_ss_k64(acc, t_lo + sub * (16384 >> 4), s_lo + sub * ((DD * 128) >> 4), idesc, sub > 0);
        } else {
          // acc[i][c] = sum_a x_i[a] S1[a][c]: B = the same bytes, K = rows a, N = c contiguous (MN-major)
          constexpr uint32_t idesc = idesc_bf16(128, DD, 0, 1);
          const uint32_t s_lo = desc_lo(sbase + C::OFF_S, DD * 128);
#pragma unroll
          for (int sub = 0; sub < C::NSUB; ++sub)
            umma_ss_kmn_steps<4>(acc, t_lo + sub * (16384 >> 4), s_lo + sub * 4 * 128, idesc, sub > 0);
        }
        umma_commit(BAR_AF(b));
        umma_commit(BAR_TE(b));
      }
      __syncwarp();
    }
    __syncwarp();
  } else {
    // ================= epilogue warps =================
    const int qd = warp & 3, t = tid - 64;
    const float c = stat_scale(a.stat_q, head, a.lim) * stat_scale(a.stat_k, head, a.lim);
    const float A1 = a.a1 * c;
    const float* st = a.state + (size_t)mat * a.rows * a.dvp + (size_t)a.f_lin * a.dvp;   // first-order rows
    for (int i = t; i < 2 * DD + 1; i += 128)
      ncol[i] = (i < DD) ? __ldg(st + (size_t)i * a.dvp + DD) : __ldg(st + (size_t)DD * a.dvp + (i - DD));
    asm volatile("bar.sync 1, 128;" ::: "memory");
    // type A adds a0 * (constant row) to every element: scaled once here (the value column DD stays raw);
    // the loops below read these vectors four values per shared-memory access
    if (!a.type_b)
      for (int i = t; i < DD; i += 128) crow[i] *= a.a0;
    asm volatile("bar.sync 1, 128;" ::: "memory");
    float part = 0.f;
    bool ok = true;
    for (int i = 0; i < nt; ++i) {
      const int b = i & 1;
      const int tok = (tile0 + i) * 128 + qd * 32 + lane;
      const bool tok_ok = tok < a.n;
      const size_t grow = (size_t)head * a.n + (tok_ok ? tok : 0);
      float extra = 0.f;   // type A: normaliser part; type B: e_i
      if (a.type_b) {
        extra = tok_ok ? (a.uvec ? -a.uvec[grow] : 1.f) : 0.f;
      } else if (a.den_add || a.final == 1) {
        // x_i . (normaliser column): the row is read from the token tile TMA delivered (128-byte rows of a
        // 64-column sub-tile, 16-byte pieces XOR-swizzled by the row), not from global memory again
        if (!mbar_wait(BAR_TF(b), (uint32_t)((i >> 1) & 1))) { report(49); ok = false; break; }
        const int r = qd * 32 + lane;
        const uint32_t trow = sbase + b * C::TILE + r * 128;
        float dot = 0.f;
#pragma unroll
        for (int sb = 0; sb < C::NSUB; ++sb)
#pragma unroll
          for (int pc = 0; pc < 8; ++pc) {
            const uint4 xv = lds128u(trow + sb * 16384 + ((pc ^ (r & 7)) << 4));
            const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
            const float4 n0 = lds128f(ncol_s + (sb * 64 + 8 * pc) * 4), n1 = lds128f(ncol_s + (sb * 64 + 8 * pc + 4) * 4);
            const float nc[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              dot = fmaf(__uint_as_float(xw[e] << 16), nc[2 * e], dot);
              dot = fmaf(__uint_as_float(xw[e] & 0xFFFF0000u), nc[2 * e + 1], dot);
            }
          }
        extra = A1 * dot + a.a0 * crow[DD];
        // this warp is done with the stage
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR_TE(b));
      }
      if (!mbar_wait(BAR_AF(b), (uint32_t)((i >> 1) & 1))) { report(45); ok = false; break; }
      tc_fence_after();
      const float scale = (a.final == 1) ? 1.0f / extra : 1.0f;
#pragma unroll 1
      for (int hcol = 0; hcol < DD / 64; ++hcol) {
        uint32_t tv[64];
        tmem_ld64(tmem + b * DD + ((uint32_t)(qd * 32) << 16) + hcol * 64, tv);
        tmem_wait_ld(tv);
        if (hcol + 1 == DD / 64) {   // the accumulator is in registers: the next product may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(BAR_AE(b));
        }
        if (tok_ok) {
          const bool wide = a.wide_io != 0;
#pragma unroll
          for (int v16 = 0; v16 < 4; ++v16) {
            float r[16];
            const uint32_t vecp = (a.type_b ? ncol_s : ncol_s + DD * 4) + (hcol * 64 + 16 * v16) * 4;
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
              const float4 c4 = lds128f(vecp + 16 * q4);
              const float cv[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const float acc = __uint_as_float(tv[16 * v16 + 4 * q4 + e]);
                r[4 * q4 + e] = a.type_b ? A1 * fmaf(extra, cv[e], acc) : fmaf(A1, acc, cv[e]);
              }
            }
            if (a.final) {
              uint32_t w[8];
#pragma unroll
              for (int e = 0; e < 8; ++e) w[e] = pack_bf16(r[2 * e] * scale, r[2 * e + 1] * scale);
              stg32((__nv_bfloat16*)a.out_final + grow * DD + hcol * 64 + 16 * v16, w, wide);
              if (a.dots) {
                uint32_t xw[8];
                ldg32((const __nv_bfloat16*)a.x + grow * DD + hcol * 64 + 16 * v16, xw, wide);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                  part = fmaf(r[2 * e], __uint_as_float(xw[e] << 16), part);
                  part = fmaf(r[2 * e + 1], __uint_as_float(xw[e] & 0xFFFF0000u), part);
                }
              }
            } else {
#pragma unroll
              for (int h8 = 0; h8 < 2; ++h8) {
                float* dst = a.o_add + grow * DD + hcol * 64 + 16 * v16 + 8 * h8;
                uint32_t w[8];
                if (a.accumulate) {
                  ldg32(dst, w, wide);
#pragma unroll
                  for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(r[8 * h8 + e] + __uint_as_float(w[e]));
                } else {
#pragma unroll
                  for (int e = 0; e < 8; ++e) w[e] = __float_as_uint(r[8 * h8 + e]);
                }
                stg32(dst, w, wide);
              }
            }
          }
        }
      }
      if (a.final) {
        if (a.final == 1 && tok_ok) a.den_final[grow] = extra;
      } else if (!a.type_b && a.den_add && tok_ok) {
        a.den_add[grow] = extra + (a.accumulate ? a.den_add[grow] : 0.f);
      }
    }
    if (ok && a.final && a.dots) {
#pragma unroll
      for (int m = 16; m >= 1; m >>= 1) part += __shfl_xor_sync(0xffffffffu, part, m);
      if (lane == 0) atomicAdd(a.dots + head, part);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, C::TCOLS);
  }
}

// bf16 copy of the first-order block: out[m][a][c] = state[m][f_lin + a][c], a, c < D; with nchunk > 0 times the
// first-order coefficient of the matrix's head
__global__ void __launch_bounds__(256) s1_to_bf16_kernel(const float* __restrict__ state,
                                                         __nv_bfloat16* __restrict__ out, int d, int dvp,
                                                         int rows, int f_lin, int nchunk, const stat_t* stat_q,
                                                         const stat_t* stat_k, float a1, float lim) {
  const int head = nchunk > 0 ? blockIdx.x / nchunk : 0;
  const float scale = nchunk > 0 ? a1 * (stat_scale(stat_q, head, lim) * stat_scale(stat_k, head, lim)) : 1.f;
  const float* src = state + (size_t)blockIdx.x * rows * dvp + (size_t)f_lin * dvp;
  __nv_bfloat16* dst = out + (size_t)blockIdx.x * d * d;
  for (int i = threadIdx.x; i < d * d; i += 256) dst[i] = __float2bfloat16_rn(scale * src[(size_t)(i / d) * dvp + i % d]);
}

// =====================================================================================
// unmasked backward of p = 1: grad_q and the states of (q, gs | e) from one read of the query side
// =====================================================================================
// What the three passes before it did -- gs = grad_out / den and dvec (fm_gprep), grad_q (read-out type B) and the
// states (first_state_kernel) -- moved q, grad_out and out once each, gs three times and grad_q once: seven tensors.
// Here a tile of gs exists in shared memory only, four tensors move.
//
//   per 128-token tile   gs = grad_out / den, rounded to bf16, written over the tile TMA delivered; dvec = gs . out
//                        T = gs S1^T                 grad_q_i[a] = A1 (T_i[a] - dvec_i S1[a][D])
//                        Q1 += q^T gs                the state's first-order rows; its vectors on the CUDA cores
//                        grad_q takes the place of gs and leaves by TMA
//
// Bound by HBM.  Persistent CTAs, one per SM, walk runs of tiles (one state each), so the loads of the next run's tiles
// are under way while a run's state is written: warp 0 TMA loads, warp 1 MMA issuer, warp 2 TMA stores, warps 4-19
// everything else (eight of them spent 7 300 cycles on a tile of d = 128, which HBM delivers in 5 600: 1 026 us for 256 heads
// x 16384, 780 with sixteen -- 5.5 TB/s; the three passes before took 1 341).  Rows are walked
// 16 bytes a thread, a row's pieces side by side, so that reads of out coalesce and a thread keeps the sums over its eight
// features in registers.  TMEM: two accumulators for T, two for Q1.
struct F1GradArgs {
  const __nv_bfloat16* out;   // (heads, n, D)
  const float* den;           // (heads, n)
  const float* total;         // (heads, rows, dvp): key/value totals
  float* states;              // (heads, runs, rows, dvp): states of the runs of (q, gs | -dvec)
  float* dots;                // per head: sum of grad_q . q is added, or null
  const stat_t* stat_q;
  const stat_t* stat_k;
  float a1, lim;
  int heads, n, dvp, rows, f_lin;
  int run, runs;              // tiles per run, runs per head
};

constexpr int FG_THREADS = 640, FG_FIRST = 4, FG_WARPS = 16;   // the first warp of those and their number

template <int DD>
struct F1G {
  static constexpr int NSUB = DD / 64;
  static constexpr int TILE = NSUB * 16384;        // 128 tokens x DD bf16
  static constexpr int STAGE = 2 * TILE;           // q, then grad_out / gs / grad_q
  static constexpr int NS = DD == 128 ? 2 : 4;     // 128 KB of tiles
  static constexpr bool AHEAD = NS > 2;            // gs of the next tile before grad_q of this one
  static constexpr int SMAT = DD * DD * 2;
  static constexpr int OFF_S = NS * STAGE;         // bf16 copies of S1 of this run's head and the next one's
  static constexpr int OFF_NCOL = OFF_S + 2 * SMAT;         // float S1[a][D] of the same
  static constexpr int OFF_E = OFF_NCOL + 2 * DD * 4;       // float e[NS][128]
  static constexpr int VROW = 2 * DD + 4;          // a warp's sums: q e [DD], gs [DD], e
  static constexpr int OFF_VEC = OFF_E + NS * 512;
  static constexpr int OFF_BAR = OFF_VEC + FG_WARPS * VROW * 4;
  static constexpr int NBAR = 4 * NS + 9;          // full, gs, grad_q, empty per stage; T, state, S full, S empty twice; meet
  static constexpr int OFF_TMEM = OFF_BAR + NBAR * 8;
  static constexpr int SMEM = OFF_TMEM + 16 + 1024;
};

// The tiles a CTA walks: runs blockIdx.x, blockIdx.x + gridDim.x, ... of all heads, tile by tile.
struct F1Walk {
  int g = 0, m = 0;          // tiles and runs before this one
  int item, head, first, t, nt;
  const F1GradArgs& a;
  __device__ __forceinline__ F1Walk(const F1GradArgs& args) : item((int)blockIdx.x), a(args) { open(); }
  __device__ __forceinline__ void open() {
    t = 0;
    head = item / a.runs;
    first = (item % a.runs) * a.run;
    nt = min(a.run, (a.n + 127) / 128 - first);
  }
  __device__ __forceinline__ bool live() const { return item < a.heads * a.runs; }
  __device__ __forceinline__ bool last() const { return t + 1 == nt; }
  __device__ __forceinline__ int token() const { return (first + t) * 128; }
  __device__ __forceinline__ void next() {
    ++g;
    if (++t == nt) {
      ++m;
      item += (int)gridDim.x;
      open();
    }
  }
};

template <int DD>
__global__ void __launch_bounds__(FG_THREADS, 1)
first_grad_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmG,
                  const __grid_constant__ CUtensorMap tmS, const __grid_constant__ CUtensorMap tmO, const F1GradArgs a) {
  using C = F1G<DD>;
  constexpr int NS = C::NS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + C::OFF_BAR;
  auto BAR_FULL = [&](int s) { return bar0 + 8u * s; };
  auto BAR_GS = [&](int s) { return bar0 + 8u * (NS + s); };
  auto BAR_DQ = [&](int s) { return bar0 + 8u * (2 * NS + s); };
  auto BAR_EMPTY = [&](int s) { return bar0 + 8u * (3 * NS + s); };
  auto BAR_T = [&](int b) { return bar0 + 8u * (4 * NS + b); };
  auto BAR_STATE = [&](int b) { return bar0 + 8u * (4 * NS + 2 + b); };
  auto BAR_SF = [&](int b) { return bar0 + 8u * (4 * NS + 4 + b); };
  auto BAR_SE = [&](int b) { return bar0 + 8u * (4 * NS + 6 + b); };
  const uint32_t BAR_MEET = bar0 + 8u * (4 * NS + 8);
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + C::OFF_TMEM);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) {
      mbar_init(BAR_FULL(s), 1);
      mbar_init(BAR_GS(s), FG_WARPS);
      mbar_init(BAR_DQ(s), FG_WARPS);
      mbar_init(BAR_EMPTY(s), 1);                  // grad_q has left it
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(BAR_T(b), 1);
      mbar_init(BAR_STATE(b), 1);
      mbar_init(BAR_SF(b), 1);
      mbar_init(BAR_SE(b), 1);
    }
    mbar_init(BAR_MEET, FG_WARPS);
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(smem_u32((const void*)tmem_slot), 4 * DD);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  F1Walk w(a);
  if (warp == 0) {
    // ================= TMA producer =================
    for (; w.live(); w.next()) {
      const int s = w.g % NS;
      if (w.t == 0) {
        if (!mbar_wait(BAR_SE(w.m & 1), (uint32_t)(((w.m >> 1) & 1) ^ 1))) { report(50); break; }
        if (lane == 0) {
          mbar_expect_tx(BAR_SF(w.m & 1), C::SMAT);
          for (int sub = 0; sub < C::NSUB; ++sub)
            tma_load_3d(sbase + C::OFF_S + (w.m & 1) * C::SMAT + sub * (DD * 128), &tmS, BAR_SF(w.m & 1), sub * 64, 0, w.head);
        }
      }
      if (!mbar_wait(BAR_EMPTY(s), (uint32_t)(((w.g / NS) & 1) ^ 1))) { report(51); break; }
      if (lane == 0) {
        mbar_expect_tx(BAR_FULL(s), C::STAGE);
        const uint32_t dst = sbase + s * C::STAGE;
        for (int sub = 0; sub < C::NSUB; ++sub) {
          tma_load_3d(dst + C::TILE + sub * 16384, &tmG, BAR_FULL(s), sub * 64, w.token(), w.head);
          tma_load_3d(dst + sub * 16384, &tmQ, BAR_FULL(s), sub * 64, w.token(), w.head);
        }
      }
    }
  } else if (warp == 1) {
    // ================= MMA issuer (whole warp, one elected lane issues) =================
    for (; w.live(); w.next()) {
      const int s = w.g % NS, mb = w.m & 1;
      const uint32_t ph = (uint32_t)((w.g / NS) & 1);
      if (w.t == 0 && !mbar_wait_warp(BAR_SF(mb), (uint32_t)((w.m >> 1) & 1))) { report(52); break; }
      // whoever forms gs has waited for the tile, and has read the accumulators that are overwritten here: T of two tiles
      // ago before this gs, the state of two runs ago before the run's first gs
      if (!mbar_wait_warp(BAR_FULL(s), ph) || !mbar_wait_warp(BAR_GS(s), ph)) { report(53); break; }
      tc_fence_after();
      const uint32_t q_s = sbase + s * C::STAGE, g_s = q_s + C::TILE;
      if (elect_one()) {
        // T[i][a] = sum_c gs_i[c] S1[a][c]: S1's rows a are K-major
        const uint32_t g_lo = desc_lo(g_s, 16), s_lo = desc_lo(sbase + C::OFF_S + mb * C::SMAT, 16);
#pragma unroll
        for (int sub = 0; sub < C::NSUB; ++sub)
          umma_ss_k64(tmem + (w.g & 1) * DD, g_lo + sub * (16384 >> 4), s_lo + sub * ((DD * 128) >> 4),
                      idesc_bf16(128, DD, 0, 0), sub > 0);
        // M = 128 feature rows; with D = 64 the second 64 are those of the tile that follows q, never read back
        umma_ss_mn_steps<8>(tmem + 2 * DD + mb * DD, desc_lo(q_s, 16384), desc_lo(g_s, 16384), idesc_bf16(128, DD, 1, 1),
                            w.t > 0 ? 1u : 0u);
        umma_commit(BAR_T(w.g & 1));       // of both products: grad_q is written over gs
        if (w.last()) {
          umma_commit(BAR_STATE(mb));
          umma_commit(BAR_SE(mb));
        }
      }
      __syncwarp();
    }
    __syncwarp();
  } else if (warp == 2) {
    // ================= TMA stores of grad_q: rows past the end are left out =================
    for (; w.live(); w.next()) {
      const int s = w.g % NS;
      if (!mbar_wait(BAR_DQ(s), (uint32_t)((w.g / NS) & 1))) { report(58); break; }
      if (lane == 0) {
        for (int sub = 0; sub < C::NSUB; ++sub)
          tma_store_3d(&tmO, sbase + s * C::STAGE + C::TILE + sub * 16384, sub * 64, w.token(), w.head);
        tma_store_wait_read();
        mbar_arrive(BAR_EMPTY(s));
      }
      __syncwarp();
    }
    if (lane == 0) tma_store_wait_all();
    __syncwarp();
  } else if (warp >= FG_FIRST) {
    constexpr int LPR = DD / 8, RPS = 32 * FG_WARPS / LPR, STEPS = 128 / RPS;   // 16-byte pieces of a row; rows per step
    const int te = tid - 32 * FG_FIRST, sub_r = te / LPR, piece = te % LPR;
    const uint32_t at0 = (uint32_t)((piece >> 3) * 16384 + sub_r * 128 + (((piece & 7) ^ (sub_r & 7)) << 4));   // in a tile
    const int qd = warp & 3, cols = (warp - FG_FIRST) >> 2;   // TMEM lane quarter; quarter of the features
    constexpr int HC = DD / 4;
    static_assert(RPS % 8 == 0 && STEPS <= LPR, "a thread's rows have one swizzle; a row's threads hold the rows' den");
    // all of these warps, in the same order; one that gave up is not waited for without a limit
    uint32_t met = 0;
    auto meet = [&]() -> bool {
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_MEET);
      if (mbar_wait(BAR_MEET, met++ & 1u)) return true;
      report(57);
      return false;
    };
    // its eight features summed over its rows: q e, gs; e
    uint64_t sq[4] = {0, 0, 0, 0}, sg[4] = {0, 0, 0, 0};
    float se = 0.f;
    uint4 o[STEPS];
    float den = 1.f;          // of this thread's row `piece`, if it has so many
    // out and den of a tile, asked for a tile ahead
    auto fetch = [&](const F1Walk& p) {
      const int tok = p.token() + sub_r;
      const size_t row = (size_t)p.head * a.n + tok;
#pragma unroll
      for (int st = 0; st < STEPS; ++st)
        o[st] = p.live() && tok + st * RPS < a.n ? __ldg((const uint4*)(a.out + (row + st * RPS) * DD) + piece)
                                                 : make_uint4(0u, 0u, 0u, 0u);
      den = p.live() && piece < STEPS && tok + piece * RPS < a.n ? __ldg(a.den + row + piece * RPS) : 1.f;
    };
    auto sts128 = [](uint32_t at, const uint32_t (&v)[4]) {
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
    };
    // grad_out -> gs in place, e = -dvec (as fm_gprep: dvec from the rounded values, so that both cancel alike)
    auto form = [&](const F1Walk& p) -> bool {
      const int s = p.g % NS;
      if (p.t == 0) {          // the run's normaliser column, once nobody reads that of two runs ago
        if (!meet()) return false;
        const float* src = a.total + (size_t)p.head * a.rows * a.dvp + (size_t)a.f_lin * a.dvp + DD;
        if (te < DD) ((float*)(smem + C::OFF_NCOL))[(p.m & 1) * DD + te] = __ldg(src + (size_t)te * a.dvp);
        if (!meet()) return false;
      }
      if (!mbar_wait(BAR_FULL(s), (uint32_t)((p.g / NS) & 1))) { report(54); return false; }
      const uint32_t qt = sbase + s * C::STAGE + at0, gt = qt + C::TILE;
      const float inv_own = 1.0f / den;
      float e[STEPS];
      uint32_t g[STEPS][4];
#pragma unroll
      for (int st = 0; st < STEPS; ++st) {
        const uint4 v = lds128u(gt + st * (RPS * 128));
        g[st][0] = v.x; g[st][1] = v.y; g[st][2] = v.z; g[st][3] = v.w;
      }
#pragma unroll
      for (int st = 0; st < STEPS; ++st) {
        const uint32_t ow[4] = {o[st].x, o[st].y, o[st].z, o[st].w};
        const float inv = __shfl_sync(0xffffffffu, inv_own, (lane & ~(LPR - 1)) | st);     // (past the end grad_out is 0)
        const uint64_t inv2 = pack2(inv, inv);
        uint64_t sum = 0ull;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          g[st][x] = pack_bf16_2(mul2(pack2u(g[st][x] << 16, g[st][x] & 0xFFFF0000u), inv2));
          const uint64_t gf = pack2u(g[st][x] << 16, g[st][x] & 0xFFFF0000u);
          sum = fma2(gf, pack2u(ow[x] << 16, ow[x] & 0xFFFF0000u), sum);
          sg[x] = add2(sg[x], gf);
        }
        float lo, hi;
        unpack2(sum, lo, hi);
        e[st] = -(lo + hi);
      }
#pragma unroll
      for (int k = LPR / 2; k >= 1; k >>= 1)
#pragma unroll
        for (int st = 0; st < STEPS; ++st) e[st] += __shfl_xor_sync(0xffffffffu, e[st], k);
#pragma unroll
      for (int st = 0; st < STEPS; ++st) {
        sts128(gt + st * (RPS * 128), g[st]);
        if (piece == 0) ((float*)(smem + C::OFF_E))[s * 128 + st * RPS + sub_r] = e[st];
      }
      fence_proxy_async();
      // (also orders this warp's earlier reads of the accumulators before the products that overwrite them)
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_GS(s));
      uint4 qv[STEPS];
#pragma unroll
      for (int st = 0; st < STEPS; ++st) qv[st] = lds128u(qt + st * (RPS * 128));
#pragma unroll
      for (int st = 0; st < STEPS; ++st) {
        const uint32_t qw[4] = {qv[st].x, qv[st].y, qv[st].z, qv[st].w};
        const uint64_t e2 = pack2(e[st], e[st]);
#pragma unroll
        for (int x = 0; x < 4; ++x) sq[x] = fma2(pack2u(qw[x] << 16, qw[x] & 0xFFFF0000u), e2, sq[x]);
        se += e[st];
      }
      return true;
    };
    // a run's vectors: column D and the constant row of its state
    auto write_vectors = [&](const F1Walk& p) -> bool {
      float* const mine = (float*)(smem + C::OFF_VEC) + (warp - FG_FIRST) * C::VROW;
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        float f[4];
        unpack2(sq[x], f[0], f[1]);
        unpack2(sg[x], f[2], f[3]);
#pragma unroll
        for (int k = LPR; k < 32; k <<= 1)          // the warp's other rows of the same features
#pragma unroll
          for (int y = 0; y < 4; ++y) f[y] += __shfl_xor_sync(0xffffffffu, f[y], k);
        if (lane < LPR) {
          *(float2*)(mine + piece * 8 + 2 * x) = make_float2(f[0], f[1]);
          *(float2*)(mine + DD + piece * 8 + 2 * x) = make_float2(f[2], f[3]);
        }
        sq[x] = sg[x] = 0ull;
      }
#pragma unroll
      for (int k = LPR; k < 32; k <<= 1) se += __shfl_xor_sync(0xffffffffu, se, k);
      if (lane == 0) mine[2 * DD] = se;
      se = 0.f;
      if (!meet()) return false;
      auto total = [&](int i) {
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < FG_WARPS; ++k) v += ((const float*)(smem + C::OFF_VEC))[k * C::VROW + i];
        return v;
      };
      float* st = a.states + (size_t)p.item * a.rows * a.dvp + (size_t)a.f_lin * a.dvp;
      if (te < DD) {
        st[(size_t)te * a.dvp + DD] = total(te);
        for (int x = DD + 1; x < a.dvp; ++x) st[(size_t)te * a.dvp + x] = 0.f;
      }
      for (int x = te; x < a.dvp; x += 32 * FG_WARPS) st[(size_t)DD * a.dvp + x] = x < DD ? total(DD + x) : (x == DD ? total(2 * DD) : 0.f);
      return meet();
    };
    float part = 0.f;
    F1Walk f(a);
    bool ok = true;
    auto form_next = [&]() {
      ok = form(f);
      if (ok && f.last()) ok = write_vectors(f);
      f.next();
      fetch(f);
    };
    fetch(f);
    if (C::AHEAD && f.live()) form_next();
    for (; ok && w.live(); w.next()) {
      if (f.live()) form_next();
      if (!ok) break;
      const int s = w.g % NS;
      // (the tile's e come from all the warps that form gs)
      if (!mbar_wait(BAR_GS(s), (uint32_t)((w.g / NS) & 1)) || !mbar_wait(BAR_T(w.g & 1), (uint32_t)((w.g >> 1) & 1))) {
        report(55);
        ok = false;
        break;
      }
      tc_fence_after();
      const float c = stat_scale(a.stat_q, w.head, a.lim) * stat_scale(a.stat_k, w.head, a.lim), A1 = a.a1 * c;
      const int r = qd * 32 + lane;
      const bool in = w.token() + r < a.n;
      const float e = ((const float*)(smem + C::OFF_E))[s * 128 + r];
      const int col = cols * HC;
      uint32_t tv[HC];
      const uint32_t t_at = tmem + ((uint32_t)(qd * 32) << 16) + (w.g & 1) * DD + col;
      if constexpr (HC == 32) tmem_ld32(t_at, tv);
      else tmem_ld16(t_at, tv);
      const uint32_t nc = sbase + C::OFF_NCOL + ((w.m & 1) * DD + col) * 4;
      const uint32_t qrow = sbase + s * C::STAGE + (col >> 6) * 16384 + r * 128, grow = qrow + C::TILE;
      tmem_wait_ld(tv);
#pragma unroll
      for (int b = 0; b < HC / 8; ++b) {
        const uint32_t pc = (((col & 63) / 8 + b) ^ (r & 7)) << 4;      // 16-byte piece of the row, swizzled
        const float4 n0 = lds128f(nc + 32 * b), n1 = lds128f(nc + 32 * b + 16);
        const float cv[8] = {n0.x, n0.y, n0.z, n0.w, n1.x, n1.y, n1.z, n1.w};
        float v[8];
        uint32_t ww[4];
#pragma unroll
        for (int x = 0; x < 8; ++x) v[x] = A1 * fmaf(e, cv[x], __uint_as_float(tv[8 * b + x]));
#pragma unroll
        for (int x = 0; x < 4; ++x) ww[x] = pack_bf16(v[2 * x], v[2 * x + 1]);
        sts128(grow + pc, ww);
        if (a.dots && in) {
          const uint4 xv = lds128u(qrow + pc);
          const uint32_t xw[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
          for (int x = 0; x < 4; ++x) {
            part = fmaf(v[2 * x], __uint_as_float(xw[x] << 16), part);
            part = fmaf(v[2 * x + 1], __uint_as_float(xw[x] & 0xFFFF0000u), part);
          }
        }
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_DQ(s));
      if (w.last()) {
        if (a.dots) {
#pragma unroll
          for (int k = 16; k >= 1; k >>= 1) part += __shfl_xor_sync(0xffffffffu, part, k);
          if (lane == 0) atomicAdd(a.dots + w.head, part);
          part = 0.f;
        }
        if (!mbar_wait(BAR_STATE(w.m & 1), (uint32_t)((w.m >> 1) & 1))) { report(56); ok = false; break; }
        tc_fence_after();
        if (qd * 32 < DD) {
          float* dst = a.states + (size_t)w.item * a.rows * a.dvp + (size_t)(a.f_lin + r) * a.dvp + col;
          uint32_t sv[HC];
          const uint32_t at = tmem + ((uint32_t)(qd * 32) << 16) + 2 * DD + (w.m & 1) * DD + col;
          if constexpr (HC == 32) tmem_ld32(at, sv);
          else tmem_ld16(at, sv);
          tmem_wait_ld(sv);
#pragma unroll
          for (int x = 0; x < HC / 4; ++x)
            ((float4*)dst)[x] = make_float4(__uint_as_float(sv[4 * x]), __uint_as_float(sv[4 * x + 1]),
                                            __uint_as_float(sv[4 * x + 2]), __uint_as_float(sv[4 * x + 3]));
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, 4 * DD);
  }
}

// Sum of a head's chunk states (the first-order rows, all there are when p = 1) and its bf16 first-order block.
// total: where the sum goes, or null.  Four elements a thread, eight chunks in flight.
__global__ void __launch_bounds__(256) first_total_kernel(const float* __restrict__ states, int nchunk, int per, int d, int dvp,
                                                          float* __restrict__ total, __nv_bfloat16* __restrict__ s1b) {
  const int e = (blockIdx.x * 256 + threadIdx.x) * 4, head = blockIdx.y;
  if (e >= per) return;
  const float* src = states + (size_t)head * nchunk * per + e;
  float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i0 = 0; i0 < nchunk; i0 += 8) {
    float4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      v[u] = i0 + u < nchunk ? __ldcs((const float4*)(src + (size_t)(i0 + u) * per)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < 8; ++u) { sum.x += v[u].x; sum.y += v[u].y; sum.z += v[u].z; sum.w += v[u].w; }
  }
  if (total) *(float4*)(total + (size_t)head * per + e) = sum;
  const int row = e / dvp, col = e % dvp;
  if (row < d && col < d)
    *(uint2*)(s1b + ((size_t)head * d + row) * d + col) = make_uint2(pack_bf16(sum.x, sum.y), pack_bf16(sum.z, sum.w));
}

}  // namespace

// ---- host side ---------------------------------------------------------------------------
// FASTMAX_B200_NO_TC_MOMENTS=1 keeps the moment family on the CUDA-core kernels (see fm_moments_tc.cu).
bool first_tc_supports(const fastmax_problem& p) {
  static const bool off = [] {
    const char* e = getenv("FASTMAX_B200_NO_TC_MOMENTS");
    return e && e[0] == '1';
  }();
  return !off && p.impl != FASTMAX_IMPL_MOMENTS_FFMA && p.dtype == FASTMAX_BF16 && (p.d == 64 || p.d == 128) && p.bh == p.bhkv;
}

size_t first_tc_copy_bytes(const fastmax_problem& p, int mats) { return (size_t)mats * p.d * p.d * 2; }

int first_tc_status(int* out, cudaStream_t stream) {
  FM_CUDA_TRY(cudaMemcpyFromSymbolAsync(out, g_ftc_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
int first_tc_status_reset(cudaStream_t stream) {
  const int zero = 0;
  FM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_ftc_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}

// First-order and constant rows of the chunk states of (y, z | e); e = 1 when dvec is null, else -dvec.
int first_tc_chunk_state(const Ctx& c, int heads, int n, int chunk, const void* y, const void* z,
                         const float* dvec, float* state) {
  if (heads == 0 || n == 0) return FASTMAX_OK;
  const fastmax_problem& p = c.p;
  const MomentDims m = moment_dims(p.d, p.p);
  const int nchunk = (n + chunk - 1) / chunk;
  CUtensorMap ty, tz;
  int rc;
  const int tok = p.d == 128 ? F1S<128>::TOK : F1S<64>::TOK;
  if ((rc = tma_map_bf16(&ty, y, heads, n, p.d, tok))) return rc;
  if ((rc = tma_map_bf16(&tz, z, heads, n, p.d, tok))) return rc;
  F1StateArgs a;
  a.y = y; a.z = z; a.dvec = dvec; a.state = state;
  a.n = n; a.chunk = chunk; a.nchunk = nchunk; a.dvp = m.dvp; a.rows = m.f; a.f_lin = p.d * p.d - m.f0;
  a.skip_chunk = c.skip_chunk;
  const unsigned grid = (unsigned)((size_t)heads * nchunk);
  if (p.d == 128) {
    FM_CUDA_TRY(cudaFuncSetAttribute(first_state_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, F1S<128>::SMEM));
    FM_LAUNCH("fm_first_tc_state", c.stream, (first_state_kernel<128><<<grid, F1_THREADS, F1S<128>::SMEM, c.stream>>>(ty, tz, a)));
  } else {
    FM_CUDA_TRY(cudaFuncSetAttribute(first_state_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, F1S<64>::SMEM));
    FM_LAUNCH("fm_first_tc_state", c.stream, (first_state_kernel<64><<<grid, F1_THREADS, F1S<64>::SMEM, c.stream>>>(ty, tz, a)));
  }
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

// Totals of a head's chunk states and their bf16 copies (p = 1: the states are the first-order rows).
int first_tc_total(const Ctx& c, int nchunk, const float* states, float* total, void* s1b) {
  const fastmax_problem& p = c.p;
  if (p.bh == 0) return FASTMAX_OK;
  const MomentDims m = moment_dims(p.d, p.p);
  const int per = m.f * m.dvp;
  dim3 grid((unsigned)((per + 1023) / 1024), p.bh);
  FM_LAUNCH("fm_first_total", c.stream,
            (first_total_kernel<<<grid, 256, 0, c.stream>>>(states, nchunk, per, p.d, m.dvp, total, (__nv_bfloat16*)s1b)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

// Tokens of a run of first_grad_kernel.  A run leaves a state behind (d = 128: 68 KB against 96 KB that a tile moves), and
// the CTAs, one per SM, each take the same number of runs but for one: the length with the least of both is taken.  At
// 512 tokens and more the states fit the room of gs (2 d bytes a token: 128 KB a run at d = 128) and one state more.
static int grad_run(const fastmax_problem& p) {
  int best = 0;
  double least = 0;
  for (int run = 512; run <= 8192; run *= 2) {
    const double t = (double)(((size_t)p.bh * ((p.nq + run - 1) / run) + 147) / 148) * ((run < p.nq ? run : p.nq) + 160);
    if (!best || t < least) {
      best = run;
      least = t;
    }
  }
  return best;
}

// Unmasked p = 1: grad_q from the key/value totals (and their bf16 copies), and the states of runs of (q, grad_out/den |
// -dvec) -- *nruns per head, at `states`, which has room for a state a head and 2 d bytes for every query row.
int first_tc_grad(const Ctx& c, const void* q, const void* out, const float* den, const void* grad_out, const float* total,
                  const void* s1b, const stat_t* stats, void* grad_q, float* dots, float* states, int* nruns) {
  const fastmax_problem& p = c.p;
  const MomentDims m = moment_dims(p.d, p.p);
  if ((((uintptr_t)grad_out | (uintptr_t)out) & 15) != 0)
    return fail(FASTMAX_E_ARG, "the tensor-core family needs 16-byte aligned tensors");
  CUtensorMap tq, tg, ts, to;
  int rc;
  if ((rc = tma_map_bf16(&tq, q, p.bh, p.nq, p.d, 128))) return rc;
  if ((rc = tma_map_bf16(&tg, grad_out, p.bh, p.nq, p.d, 128))) return rc;
  if ((rc = tma_map_bf16(&ts, s1b, p.bh, p.d, p.d, p.d))) return rc;
  if ((rc = tma_map_bf16(&to, grad_q, p.bh, p.nq, p.d, 128))) return rc;
  F1GradArgs a;
  a.out = (const __nv_bfloat16*)out; a.den = den; a.total = total; a.states = states; a.dots = dots;
  a.stat_q = p.normalize ? stats : nullptr;
  a.stat_k = p.normalize ? stats + p.bh : nullptr;
  a.a1 = p.a1; a.lim = p.lim;
  a.heads = p.bh; a.n = p.nq; a.dvp = m.dvp; a.rows = m.f; a.f_lin = p.d * p.d - m.f0;
  a.run = grad_run(p) / 128;
  a.runs = ((p.nq + 127) / 128 + a.run - 1) / a.run;
  *nruns = a.runs;
  const size_t items = (size_t)p.bh * a.runs;
  const unsigned grid = (unsigned)(items < 148 ? items : 148);
  if (p.d == 128) {
    FM_CUDA_TRY(cudaFuncSetAttribute(first_grad_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, F1G<128>::SMEM));
    FM_LAUNCH("fm_first_tc_grad", c.stream, (first_grad_kernel<128><<<grid, FG_THREADS, F1G<128>::SMEM, c.stream>>>(tq, tg, ts, to, a)));
  } else {
    FM_CUDA_TRY(cudaFuncSetAttribute(first_grad_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, F1G<64>::SMEM));
    FM_LAUNCH("fm_first_tc_grad", c.stream, (first_grad_kernel<64><<<grid, FG_THREADS, F1G<64>::SMEM, c.stream>>>(tq, tg, ts, to, a)));
  }
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

// bf16 copies of the first-order blocks of `mats` prefix (or total) states
int first_tc_convert(const Ctx& c, int mats, const float* state, void* s1b, int nchunk, const stat_t* stats) {
  if (mats == 0) return FASTMAX_OK;
  const fastmax_problem& p = c.p;
  const MomentDims m = moment_dims(p.d, p.p);
  FM_LAUNCH("fm_first_state_bf16", c.stream,
            (s1_to_bf16_kernel<<<mats, 256, 0, c.stream>>>(state, (__nv_bfloat16*)s1b, p.d, m.dvp, m.f,
                                                           p.d * p.d - m.f0, nchunk, p.normalize ? stats : nullptr,
                                                           p.normalize ? stats + p.bh : nullptr, p.a1, p.lim)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

// type A (type_b = 0): tile = x;  type B: tile = u (gs or v), uvec = dvec or null.  x is the token
// tensor itself (normaliser dot of type A).  Results overwrite o_add / den_add unless accumulate.
int first_tc_readout(const Ctx& c, int type_b, int heads, int n, int chunk, int per_chunk, const void* tile,
                     const void* x, const float* uvec, const float* state, const void* s1b,
                     const stat_t* stats, float* o_add, float* den_add, int accumulate, int final,
                     void* out_final, float* den_final, float* dots) {
  if (heads == 0 || n == 0) return FASTMAX_OK;
  const fastmax_problem& p = c.p;
  const MomentDims m = moment_dims(p.d, p.p);
  const int nchunk = (n + chunk - 1) / chunk;
  CUtensorMap tt, ts;
  int rc;
  if ((rc = tma_map_bf16(&tt, tile, heads, n, p.d, 128))) return rc;
  if ((rc = tma_map_bf16(&ts, s1b, (size_t)heads * (per_chunk ? nchunk : 1), p.d, p.d, p.d))) return rc;
  F1ReadArgs a;
  a.x = x; a.uvec = uvec; a.state = state; a.o_add = o_add; a.den_add = den_add;
  a.stat_q = p.normalize ? stats : nullptr;
  a.stat_k = p.normalize ? stats + p.bh : nullptr;
  a.a0 = p.a0; a.a1 = p.a1; a.lim = p.lim;
  a.n = n; a.chunk = chunk; a.nchunk = nchunk; a.per_chunk = per_chunk; a.dvp = m.dvp; a.rows = m.f;
  a.f_lin = p.d * p.d - m.f0; a.type_b = type_b; a.accumulate = accumulate;
  a.final = final; a.out_final = out_final; a.den_final = den_final; a.dots = dots;
  a.wide_io = (((uintptr_t)out_final | (uintptr_t)o_add | (uintptr_t)x) & 31) == 0;
  a.zero_chunk = (per_chunk && !final) ? c.zero_chunk : -1;
  // A CTA takes a run of tiles that share a state and pays for the copy, the vector terms and its own start once, as much
  // as two or three tiles; two CTAs run per SM.  The length that gives the shortest sum of waves is taken among those that do
  // not cross a chunk (256 heads x 16384 x 128: 32 tiles, in 3.5 waves, 409 us type A
  // and 373 type B; 16, in 6.9, 391 and 366).
  const int tiles = (n + 127) / 128;
  int run = 0;
  for (int r = per_chunk ? min(32, (chunk / 128) & -(chunk / 128)) : 32, least = 0; r >= 1; r >>= 1) {
    const long long waves = ((long long)heads * ((tiles + r - 1) / r) + 295) / 296, cost = waves * (r + 2);
    if (run == 0 || cost < least) {
      run = r;
      least = (int)(cost < 0x7FFFFFFF ? cost : 0x7FFFFFFF);
    }
  }
  a.run = run;
  const unsigned grid = (unsigned)((size_t)heads * ((tiles + run - 1) / run));
  const char* name = type_b ? "fm_first_tc_readout_b" : "fm_first_tc_readout_a";
  if (p.d == 128) {
    FM_CUDA_TRY(cudaFuncSetAttribute(first_readout_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, F1R<128>::SMEM));
    FM_LAUNCH(name, c.stream, (first_readout_kernel<128><<<grid, F1_THREADS, F1R<128>::SMEM, c.stream>>>(tt, ts, a)));
  } else {
    FM_CUDA_TRY(cudaFuncSetAttribute(first_readout_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, F1R<64>::SMEM));
    FM_LAUNCH(name, c.stream, (first_readout_kernel<64><<<grid, F1_THREADS, F1R<64>::SMEM, c.stream>>>(tt, ts, a)));
  }
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

}  // namespace fm
