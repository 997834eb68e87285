// Prompt processing for the decode state on the tcgen05 tensor cores (bf16 keys and values, d 64 or 128).
//
// What append_kernel of fm_decode.cu sums on the CUDA cores is a matrix product per head:
//   S[pair (a, b)][c] += sum_j (k_j[a] k_j[b]) (v_j, 1)[c]        rows: unordered feature pairs, K: tokens
// The product of two bf16 numbers has at most 16 significand bits, so it is EXACTLY the sum of two bf16 numbers;
// with the values as they are (bf16) every product the tensor core forms is exact, and what is rounded is the
// float32 summation only: the accumulators hold 64 tokens at a time and are then added to float32 registers,
// rounded to nearest.  (Finite keys and values: an infinite value times a low part that is exactly zero is NaN where a
// plain sum would stay infinite; a row of the state that holds either gives NaN when it is read.)  Measured, 2-norm error of the state against float64: 9.3e-7 after 4000 tokens where the
// CUDA-core kernel, token by token, has 2.8e-6; 0.9e-7 after 64.
//
// Rows.  128 lanes of tensor memory are one tile of pairs (b, b + s mod d) at a fixed distance s around the ring
// of features: d = 64 has two distances per tile (s = 0..32, every unordered pair once; half of s = 32 is left over),
// d = 128 one (s = 0..64).  The first-order rows are the pairs (b, one) and the constant row is (one, one), `one`
// being an extra feature row, so one code path makes every row of the state.
//
// One CTA = two tiles of one head and 64 value columns, 608 threads: two groups of eight warps, a tile each; warp 16
// loads the value tiles by TMA, warps 17 and 18 issue the products of the two tiles.  Per block of 64 tokens the
// sixteen warps write the keys transposed to shared memory (yT[feature][token]; 16-byte chunks XOR-swizzled so that
// the transposed stores and the row reads are both free of bank conflicts), then a thread forms its lane's 32 products
// (half of the block: two warps share a lane quarter), splits them and stores them as the A operand in tensor memory;
// B is the value tile as TMA delivered it.  The normaliser column is the sum of the thread's own products.
// 64 heads x 4000 tokens, d = 64, p = 2: 0.39 ms (append_kernel 2.22 ms; 0.57 ms with a block's 32 operand words held at
// once, which spilled).  Per block of 64 tokens the generator's chain -- transposed stores, barrier, row reads, products
// and splits, tcgen05.st -- takes some 3 000 cycles of which the two tiles' products need 520.
// The result goes through shared memory, because a lane is a row of 65 floats: whole rows are read, added and written
// to both places of the pair.
#include "fm_common.cuh"
#include "fm_sm100.cuh"

namespace fm {

__device__ int g_dec_status = 0;

namespace {
using namespace sm100;

constexpr int kHeader = 4;
constexpr int TB = 64;                                  // tokens per block
constexpr int kGenWarps = 16, kGenThreads = kGenWarps * 32;
constexpr int kProducerWarp = 16, kIssuerWarp = 17;     // and 18
constexpr int kThreads = 19 * 32;
constexpr int NS = 3;                                   // value stages

template <int D>
struct AT {
  static constexpr int ROWS = D + 2;                    // features, ones, zeros
  static constexpr int YT = ROWS * 128;                 // bytes of one transposed block (64 tokens)
  static constexpr int OFF_V = 0, OFF_Y = NS * 8192;    // the TMA tiles stay on 1024-byte boundaries
  static constexpr int OFF_EP = OFF_Y + 2 * YT;         // float ep[2][128][65], the last column: second part of e
  static constexpr int OFF_E = OFF_EP + 2 * 128 * 65 * 4;
  static constexpr int OFF_BAR = OFF_E + 2 * 128 * 4;
  static constexpr int NBAR = 2 * NS + 4;               // v_full, v_empty, a_full[2], done[2]
  static constexpr int OFF_MISC = OFF_BAR + NBAR * 8;   // TMEM address, max |k|^2 bits
  static constexpr int SMEM = OFF_MISC + 16 + 1024;
  static constexpr int TILES = (D == 64) ? 17 : 66;
  static constexpr int FIRST_ONLY = (D == 64) ? 16 : 64;   // p = 1: only the tiles with first-order rows
  static constexpr int CB = D / 64;                     // column blocks
};

struct AppArgs {
  const __nv_bfloat16* k;
  float* state;
  long long n_new, head_floats;
  int p, tile0, tiles;   // tiles tile0 .. tile0 + tiles - 1 exist
};

__device__ __forceinline__ void report(int code) { atomicCAS(&g_dec_status, 0, code); }

// Byte offset of token chunk c (8 tokens) of row f inside a transposed block.
__device__ __forceinline__ uint32_t yt_off(int f, int c) { return (uint32_t)(f * 128 + ((c ^ (f & 7) ^ ((f >> 3) & 7)) << 4)); }


template <int D>
__global__ void __launch_bounds__(kThreads, 1)
append_tc_kernel(const __grid_constant__ CUtensorMap tmV, const AppArgs a) {
  using C = AT<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + C::OFF_BAR;
  auto BAR_VF = [&](int s) { return bar0 + 8u * s; };
  auto BAR_VE = [&](int s) { return bar0 + 8u * (NS + s); };
  auto BAR_A = [&](int t) { return bar0 + 8u * (2 * NS + t); };
  auto BAR_DONE = [&](int t) { return bar0 + 8u * (2 * NS + 2 + t); };
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + C::OFF_MISC);
  int* kmax_bits = (int*)(smem + C::OFF_MISC + 4);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head = blockIdx.y, cb = blockIdx.x % C::CB, pair0 = (blockIdx.x / C::CB) * 2;
  const int active = min(2, a.tiles - pair0);            // tiles of this CTA
  float* hs = a.state + (long long)head * a.head_floats;
  const int nblk = (int)((a.n_new + TB - 1) / TB);

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) { mbar_init(BAR_VF(s), 1); mbar_init(BAR_VE(s), active); }
    for (int t = 0; t < 2; ++t) { mbar_init(BAR_A(t), kGenWarps / 2); mbar_init(BAR_DONE(t), 1); }
    mbar_fence_init();
    *kmax_bits = __float_as_int(hs[0]);
  }
  if (warp == kIssuerWarp) tmem_alloc(smem_u32((const void*)tmem_slot), 256);
  // the zero row of both buffers
  for (int i = tid; i < 2 * 32; i += kThreads) *(uint32_t*)(smem + C::OFF_Y + (i >> 5) * C::YT + (D + 1) * 128 + (i & 31) * 4) = 0u;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  bool ok = true;
  if (warp == kProducerWarp) {
    if (lane == 0) tma_prefetch_desc(&tmV);
    for (int j = 0; j < nblk; ++j) {
      const int s = j % NS;
      if (!mbar_wait(BAR_VE(s), (uint32_t)(((j / NS) & 1) ^ 1))) { report(61); break; }
      if (lane == 0) {
        mbar_expect_tx(BAR_VF(s), 8192);
        tma_load_3d(sbase + C::OFF_V + s * 8192, &tmV, BAR_VF(s), cb * 64, j * TB, head);
      }
    }
  } else if (warp >= kIssuerWarp) {
    const int t = warp - kIssuerWarp;
    if (t < active) {
      constexpr uint32_t idesc = idesc_bf16(128, 64, 0, 1);
      const uint32_t acc = tmem + t * 128, v_mn = desc_lo(sbase + C::OFF_V, 8192);
      for (int j = 0; j < nblk; ++j) {
        const int s = j % NS;
        if (!mbar_wait_warp(BAR_VF(s), (uint32_t)((j / NS) & 1))) { report(62); break; }
        if (!mbar_wait_warp(BAR_A(t), (uint32_t)(j & 1))) { report(63); break; }
        tc_fence_after();
        const uint32_t b = v_mn + (uint32_t)s * (8192 >> 4);
        if (elect_one()) {
          umma_ts_steps<TB / 16>(acc, acc + 96, b, idesc, 0u);     // low parts first
          umma_ts_steps<TB / 16>(acc, acc + 64, b, idesc, 1u);
          umma_commit(BAR_DONE(t));
          umma_commit(BAR_VE(s));
        }
        __syncwarp();
      }
    }
    __syncwarp();
  } else {
    const int t = warp >> 3, qd = warp & 3, hf = (warp >> 2) & 1;
    const int L = qd * 32 + lane, tile = a.tile0 + pair0 + t;
    const bool on = t < active;
    // this lane's two feature rows (D: ones, D + 1: zeros)
    int fx = D + 1, fy = D + 1;
    if (on) {
      const int b = (D == 64) ? (L & 63) : L, s = (D == 64) ? 2 * tile + (L >> 6) : tile;
      if (s < D / 2) { fx = b; fy = (b + s) & (D - 1); }
      else if (s == D / 2) {
        if (b < D / 2) { fx = b; fy = b + D / 2; }
        else if (b == D / 2) { fx = D; fy = D; }
      } else { fx = b; fy = D; }
      if (a.p == 1 && fx < D && fy < D) { fx = D + 1; fy = D + 1; }
    }
    const uint32_t tl = tmem + t * 128 + ((uint32_t)(qd * 32) << 16);
    uint64_t run[16], e2 = 0ull;
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
    // 16 bytes (8 features) of one token per thread and load; tokens past the end read as zero
    constexpr int VPT = D / 8, NLD = TB * VPT / kGenThreads;
    const __nv_bfloat16* kh = a.k + (long long)head * a.n_new * D;
    uint4 kr[NLD];
    auto fetch = [&](int j) {
#pragma unroll
      for (int i = 0; i < NLD; ++i) {
        const int idx = tid + i * kGenThreads;
        const long long tok = (long long)j * TB + idx / VPT;
        kr[i] = (j < nblk && tok < a.n_new) ? __ldg((const uint4*)(kh + tok * D) + idx % VPT) : make_uint4(0u, 0u, 0u, 0u);
      }
    };
    float kmax = 0.f;
    fetch(0);
    for (int j = 0; j < nblk; ++j) {
      uint8_t* yt = smem + C::OFF_Y + (j & 1) * C::YT;
      const uint32_t yt_s = sbase + C::OFF_Y + (j & 1) * C::YT;
#pragma unroll
      for (int i = 0; i < NLD; ++i) {
        const int idx = tid + i * kGenThreads, tok = idx / VPT, f0 = (idx % VPT) * 8;
        const uint32_t w[4] = {kr[i].x, kr[i].y, kr[i].z, kr[i].w};
        // the neighbouring token (VPT lanes away) gives the other half of every token pair: the even token's
        // thread writes features 0..3, the odd one's 4..7
        const bool odd = (tok & 1) != 0;
        uint32_t mine[2], theirs[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          mine[h] = odd ? w[2 + h] : w[h];
          theirs[h] = __shfl_xor_sync(0xffffffffu, odd ? w[h] : w[2 + h], VPT);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const uint32_t m = mine[e >> 1], o = theirs[e >> 1];
          const uint32_t lo = odd ? o : m, hi = odd ? m : o;          // even token in the low half
          const uint32_t word = __byte_perm(lo, hi, (e & 1) ? 0x7632 : 0x5410);
          const int f = f0 + (odd ? 4 : 0) + e;
          *(uint32_t*)(yt + yt_off(f, tok >> 3) + ((tok >> 1) & 3) * 4) = word;
        }
        if (blockIdx.x == 0) {
          float n2 = 0.f;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float lo = __uint_as_float(w[e] << 16), hi = __uint_as_float(w[e] & 0xFFFF0000u);
            n2 = fmaf(lo, lo, fmaf(hi, hi, n2));
          }
#pragma unroll
          for (int m = 1; m < VPT; m <<= 1) n2 += __shfl_xor_sync(0xffffffffu, n2, m);
          kmax = fmaxf(kmax, n2);
        }
      }
      if (tid < TB / 2) {     // the row of ones: nothing past the last token
        const long long tok = (long long)j * TB + 2 * tid;
        const uint32_t one = 0x3F80u;
        *(uint32_t*)(yt + yt_off(D, tid >> 2) + (tid & 3) * 4) =
            (tok < a.n_new ? one : 0u) | (tok + 1 < a.n_new ? one << 16 : 0u);
      }
      asm volatile("bar.sync 1, 512;" ::: "memory");
      fetch(j + 1);
      if (!on) continue;
      // two chunks of 8 tokens at a time: their 16 operand words and the 32 running sums fit the registers
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const ulonglong2 x = lds_v2(yt_s + yt_off(fx, hf * 4 + half * 2 + c)), y = lds_v2(yt_s + yt_off(fy, hf * 4 + half * 2 + c));
          const uint32_t xw[4] = {(uint32_t)x.x, (uint32_t)(x.x >> 32), (uint32_t)x.y, (uint32_t)(x.y >> 32)};
          const uint32_t yw[4] = {(uint32_t)y.x, (uint32_t)(y.x >> 32), (uint32_t)y.y, (uint32_t)(y.y >> 32)};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint64_t pr = mul2(pack2u(xw[q] << 16, xw[q] & 0xFFFF0000u), pack2u(yw[q] << 16, yw[q] & 0xFFFF0000u));
            e2 = add2(e2, pr);
            const uint32_t h = pack_bf16_2(pr);
            hi[4 * c + q] = h;
            lo[4 * c + q] = pack_bf16_2(fma2(pack2u(h << 16, h & 0xFFFF0000u), 0xBF800000BF800000ull, pr));
          }
        }
        if (half == 0 && j > 0) {     // the previous block's products are done: take its sums over, reuse the operand
          if (ok && !mbar_wait(BAR_DONE(t), (uint32_t)((j - 1) & 1))) { report(64); ok = false; }
          tc_fence_after();
          promote();
        }
        tmem_st8(tl + 64 + hf * 16 + half * 8, hi);
        tmem_st8(tl + 96 + hf * 16 + half * 8, lo);
      }
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_A(t));
    }
    if (on) {
      if (ok && !mbar_wait(BAR_DONE(t), (uint32_t)((nblk - 1) & 1))) { report(65); ok = false; }
      tc_fence_after();
      promote();
      float* ep = (float*)(smem + C::OFF_EP) + (t * 128 + L) * 65;
#pragma unroll
      for (int i = 0; i < 16; ++i) unpack2(run[i], ep[hf * 32 + 2 * i], ep[hf * 32 + 2 * i + 1]);
      float e0, e1;
      unpack2(e2, e0, e1);
      if (hf == 0) ep[64] = e0 + e1;
      else ((float*)(smem + C::OFF_E))[t * 128 + L] = e0 + e1;
    }
    if (blockIdx.x == 0 && kmax > 0.f) atomicMax(kmax_bits, __float_as_int(kmax));
  }
  tc_fence_before();
  ok = __syncthreads_and(ok);
  if (warp == kIssuerWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 256);
  }
  // a wait gave up: this CTA adds nothing, others of the head may have -- the state is undefined once the status word is set
  if (!ok) return;
  if (blockIdx.x == 0 && tid == 0) {
    hs[0] = __int_as_float(*kmax_bits);
    hs[1] = __int_as_float(__float_as_int(hs[1]) + (int)a.n_new);
  }
  // whole rows of the state: old values plus this call's sums, to both places of a pair
  constexpr int DV = D + 1;
  const int n2rows = (a.p == 2) ? D * D : 0;
  float* st = hs + kHeader;
  for (int rr = warp; rr < active * 128; rr += kThreads / 32) {
    const int t = rr >> 7, L = rr & 127, tile = a.tile0 + pair0 + t;
    const int b = (D == 64) ? (L & 63) : L, s = (D == 64) ? 2 * tile + (L >> 6) : tile;
    int row1, row2;
    if (s < D / 2 || (s == D / 2 && b < D / 2)) {
      if (a.p == 1) continue;
      const int o = (b + s) & (D - 1), x = min(b, o), y = max(b, o);
      row1 = x * D + y;
      row2 = y * D + x;
    } else if (s == D / 2) {
      if (b != D / 2) continue;
      row1 = row2 = n2rows + D;
    } else {
      row1 = row2 = n2rows + b;
    }
    const float* ep = (const float*)(smem + C::OFF_EP) + rr * 65;
    float* r1 = st + (long long)row1 * DV;
    float* r2 = st + (long long)row2 * DV;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int c = cb * 64 + h * 32 + lane;
      const float f = r1[c] + ep[h * 32 + lane];
      r1[c] = f;
      if (row2 != row1) r2[c] = f;
    }
    if (cb == 0 && lane == 0) {
      const float f = r1[D] + (ep[64] + ((const float*)(smem + C::OFF_E))[rr]);
      r1[D] = f;
      if (row2 != row1) r2[D] = f;
    }
  }
}

template <int D>
int launch(const fastmax_problem& p, const void* k, const void* v, long long n_new, float* state, cudaStream_t st) {
  using C = AT<D>;
  CUtensorMap tv;
  int rc;
  if ((rc = tma_map_bf16(&tv, v, p.bhkv, (size_t)n_new, D, TB))) return rc;
  const long long rows = 1 + D + (p.p == 2 ? (long long)D * D : 0);
  AppArgs a{(const __nv_bfloat16*)k, state, n_new, kHeader + rows * (D + 1), p.p, p.p == 1 ? C::FIRST_ONLY : 0,
            p.p == 1 ? C::TILES - C::FIRST_ONLY : C::TILES};
  dim3 grid((a.tiles + 1) / 2 * C::CB, p.bhkv);
  FM_CUDA_TRY(cudaFuncSetAttribute(append_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
  FM_LAUNCH("fm_decode_append", st, (append_tc_kernel<D><<<grid, kThreads, C::SMEM, st>>>(tv, a)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

}  // namespace

int decode_append_tc(const fastmax_problem& p, const void* k, const void* v, long long n_new, float* state,
                     cudaStream_t st) {
  return p.d == 64 ? launch<64>(p, k, v, n_new, state, st) : launch<128>(p, k, v, n_new, state, st);
}
int decode_tc_status(int* out, cudaStream_t stream) {
  FM_CUDA_TRY(cudaMemcpyFromSymbolAsync(out, g_dec_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
int decode_tc_status_reset(cudaStream_t stream) {
  const int zero = 0;
  FM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_dec_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}

}  // namespace fm
