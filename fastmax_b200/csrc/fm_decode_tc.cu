// Prompt processing for the decode state on the tcgen05 tensor cores (bf16 keys and values, d 64 or 128).
//
// What append_kernel of fm_decode.cu sums on the CUDA cores is a matrix product per head:
//   S[pair (a, b)][c] += sum_j (k_j[a] k_j[b]) (v_j, 1)[c]        rows: unordered feature pairs, K: tokens
// The product of two bf16 numbers has at most 16 significand bits, so it is EXACTLY the sum of two bf16 numbers, its
// rounding to bf16 and what that leaves, which one multiplication and one fused multiply-add on bf16 pairs deliver;
// with the values as they are (bf16) every product the tensor core forms is exact, and what is rounded is the
// float32 summation only: an accumulator holds 64 tokens and is then added to float32 registers, rounded to nearest.
// (Finite keys and values: an infinite value times a low part that is exactly zero is NaN where a
// plain sum would stay infinite; a row of the state that holds either gives NaN when it is read.)  Measured, 2-norm error
// of the state against float64, N(0,1) keys, d = 64: 0.9e-7 after 64 and 128 tokens, 1.1e-7 after 1000, 1.5e-7 after 4000, and of
// its normaliser column 0.4e-7 to 0.8e-7 (few_kernel, token by token: 0.9e-7 and 0.4e-7 after 28, append_kernel 2.8e-6 after 4000).
//
// Rows.  128 lanes of tensor memory are one tile of pairs (b, b + s mod d) at a fixed distance s around the ring
// of features: d = 64 has two distances per tile (s = 0..32, every unordered pair once; half of s = 32 is left over),
// d = 128 one (s = 0..64).  The first-order rows are the pairs (b, one) and the constant row is (one, one), `one`
// being an extra feature row, so one code path makes every row of the state.
//
// One CTA = two tiles of one head and 64 value columns, 608 threads: two groups of eight warps, a tile each; warp 16
// loads the value and key tiles by TMA, warps 17 and 18 issue the products of the two tiles.  Per block of 128 tokens the
// sixteen warps write the keys transposed to shared memory (yT[feature][token]; 16-byte chunks XOR-swizzled so that
// the transposed stores and the row reads are both free of bank conflicts), then a thread forms its lane's 64 products
// (half of the block's: two warps share a lane quarter), sixteen at a time, and stores their parts as the A operand in tensor
// memory; B is the value tile as TMA delivered it and, sixteen columns more, ones that make the normaliser: every K step's high
// parts have a column of their own there, and its low parts another, so that the tensor core adds sixteen numbers of eight bits
// to each and everything else is added in float32, rounded to nearest.  The two halves of a block have an accumulator each,
// because the tensor core truncates what it adds: 128 tokens in one had 1.2 to 2 times the error of 64 in prompts of 65 to 1000.
// There is no room for both beside the parts, so the second one lies over the parts of the first half, and its products wait for
// the first half's; the other tile's are issued meanwhile.
//   Measured, 64 heads, d = 64, p = 2: 4000 tokens 388 -> 284 us of kernel, 40 tokens 61 -> 40 (append_kernel: 2.22 ms for the
// former).  Of it: products as bf16 pairs instead of eleven instructions on unpacked float32 and the normaliser from the tensor core
// take off a ninth, blocks of 128 tokens instead of 64 8 %, keys by TMA 1 %, rows of the state asked for seven at a time 11 %; an
// accumulator to either half of a block costs 9 % (261 with one, at up to twice the error; 292 when both halves' sums are taken
// over before the parts are formed, 303 with the first half's products issued ahead of the second half's parts).  What bounds it: a
// block's chain -- transposed stores, barrier, row reads, products, tcgen05.st, sums -- 4 000 cycles, of which the shared-memory port
// is busy for some 2 200 (row reads 1 000, the tensor core's reads of B 640) and the tensor pipe for 1 300.  The transposition one
// block ahead with barriers of its own was slower by a tenth.
// The result goes through shared memory, because a lane is a row of 65 floats: whole rows are read, added and written
// to both places of the pair.
#include "fm_common.cuh"
#include "fm_sm100.cuh"

namespace fm {

__device__ int g_dec_status = 0;

namespace {
using namespace sm100;

constexpr int kHeader = 4;
constexpr int TB = 128;                                 // tokens per block
constexpr int kGenWarps = 16, kGenThreads = kGenWarps * 32;
constexpr int kProducerWarp = 16, kIssuerWarp = 17;     // and 18
constexpr int kThreads = 19 * 32;
constexpr int VT = TB * 128;                            // bytes of a tile of 64 columns
// TMEM columns of a tile: the accumulator of half h of a block is at 80 h (64 value columns, 16 of the normaliser), the parts of
// its K steps at 80 (h + 1).  So the second accumulator's value columns are where the first half's parts were: those of a lane
// quarter's two warps (32 columns each: two steps' low, two steps' high parts) under the columns that the same warp reads.
constexpr int kTileCols = 256, kHalfCols = 80, kHiOff = 16;
__device__ __forceinline__ constexpr int part_col(int half, int warp, int step) { return kHalfCols * (half + 1) + 32 * warp + 8 * step; }

template <int D>
struct AT {
  static constexpr int ROWS = D + 2;                    // features, ones, zeros
  static constexpr int YT = ROWS * TB * 2;              // bytes of one transposed block
  static constexpr int NS = D == 64 ? 3 : 2;            // stages: a value tile and the key tiles
  static constexpr int STAGE = VT + D / 64 * VT;
  static constexpr int OFF_ONE = NS * STAGE;            // the TMA tiles stay on 1024-byte boundaries
  static constexpr int OFF_Y = OFF_ONE + 2 * VT;
  static constexpr int OFF_EP = 0;                      // float ep[2][128][65], where the stages were
  static constexpr int OFF_E = 2 * 128 * 65 * 4;        // float e[2][128]: the second halves' part of the last column
  static constexpr int OFF_BAR = OFF_Y + 2 * YT;
  static_assert(NS * STAGE >= OFF_E + 2 * 128 * 4, "room for the results");
  static constexpr int NBAR = 2 * NS + 6;               // full, empty, a_full[2], first half done[2], done[2]
  static constexpr int OFF_MISC = OFF_BAR + NBAR * 8;   // TMEM address, max |k|^2 bits
  static constexpr int SMEM = OFF_MISC + 16 + 1024;
  static constexpr int TILES = (D == 64) ? 17 : 66;
  static constexpr int FIRST_ONLY = (D == 64) ? 16 : 64;   // p = 1: only the tiles with first-order rows
  static constexpr int CB = D / 64;                     // column blocks
};

struct AppArgs {
  float* state;
  long long n_new, head_floats;
  int p, tile0, tiles;   // tiles tile0 .. tile0 + tiles - 1 exist
};

__device__ __forceinline__ void report(int code) { atomicCAS(&g_dec_status, 0, code); }

__device__ __forceinline__ uint4 lds128(uint32_t saddr) {
  uint4 r;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(saddr));
  return r;
}
__device__ __forceinline__ __nv_bfloat162 as_bf162(uint32_t w) { return *reinterpret_cast<const __nv_bfloat162*>(&w); }
__device__ __forceinline__ uint32_t as_u32(__nv_bfloat162 v) { return *reinterpret_cast<const uint32_t*>(&v); }
// Byte offset of token chunk c (8 tokens) of row f inside a transposed block.
__device__ __forceinline__ uint32_t yt_off(int f, int c) { return (uint32_t)(f * (TB * 2) + ((c ^ (f & 7) ^ ((f >> 3) & 7)) << 4)); }


template <int D>
__global__ void __launch_bounds__(kThreads, 1)
append_tc_kernel(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmK, const AppArgs a) {
  using C = AT<D>;
  constexpr int NS = C::NS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + C::OFF_BAR;
  auto BAR_VF = [&](int s) { return bar0 + 8u * s; };
  auto BAR_VE = [&](int s) { return bar0 + 8u * (NS + s); };
  auto BAR_A = [&](int t) { return bar0 + 8u * (2 * NS + t); };
  auto BAR_HALF = [&](int t) { return bar0 + 8u * (2 * NS + 2 + t); };
  auto BAR_DONE = [&](int t) { return bar0 + 8u * (2 * NS + 4 + t); };
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + C::OFF_MISC);
  int* kmax_bits = (int*)(smem + C::OFF_MISC + 4);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head = blockIdx.y, cb = blockIdx.x % C::CB, pair0 = (blockIdx.x / C::CB) * 2;
  const int active = min(2, a.tiles - pair0);            // tiles of this CTA
  float* hs = a.state + (long long)head * a.head_floats;
  const int nblk = (int)((a.n_new + TB - 1) / TB);

  if (tid == 0) {
    for (int s = 0; s < NS; ++s) { mbar_init(BAR_VF(s), 1); mbar_init(BAR_VE(s), active + kGenWarps); }
    for (int t = 0; t < 2; ++t) {
      mbar_init(BAR_A(t), kGenWarps / 2);
      mbar_init(BAR_HALF(t), 1);
      mbar_init(BAR_DONE(t), 1);
    }
    mbar_fence_init();
    *kmax_bits = __float_as_int(hs[0]);
  }
  if (warp == kIssuerWarp) tmem_alloc(smem_u32((const void*)tmem_slot), 512);
  // the second block of B, for high and for low parts: sixteen columns (two 16-byte pieces, XOR-swizzled by the row), of which
  // one is one and the others zero -- the row's K step of its half, low parts four columns on; its other columns are not read
  for (int i = tid; i < 4 * TB; i += kThreads) {
    const int r = (i >> 1) % TB, low = i / (2 * TB), x = 4 * low + ((r >> 4) & 3);
    const uint32_t one = i & 1 ? 0u : 0x3F80u << (16 * (x & 1));
    *(uint4*)(smem + C::OFF_ONE + low * VT + r * 128 + (((i & 1) ^ (r & 7)) << 4)) =
        make_uint4(x >> 1 == 0 ? one : 0u, x >> 1 == 1 ? one : 0u, x >> 1 == 2 ? one : 0u, x >> 1 == 3 ? one : 0u);
  }
  fence_proxy_async();
  // the zero row of both buffers
  for (int i = tid; i < TB; i += kThreads)
    *(uint32_t*)(smem + C::OFF_Y + (i / (TB / 2)) * C::YT + (D + 1) * (TB * 2) + (i % (TB / 2)) * 4) = 0u;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  bool ok = true;
  if (warp == kProducerWarp) {
    if (lane == 0) { tma_prefetch_desc(&tmV); tma_prefetch_desc(&tmK); }
    for (int j = 0; j < nblk; ++j) {
      const int s = j % NS;
      if (!mbar_wait(BAR_VE(s), (uint32_t)(((j / NS) & 1) ^ 1))) { report(61); break; }
      if (lane == 0) {
        const uint32_t dst = sbase + s * C::STAGE;
        mbar_expect_tx(BAR_VF(s), C::STAGE);
        for (int sub = 0; sub < D / 64; ++sub) tma_load_3d(dst + VT + sub * VT, &tmK, BAR_VF(s), sub * 64, j * TB, head);
        tma_load_3d(dst, &tmV, BAR_VF(s), cb * 64, j * TB, head);
      }
    }
  } else if (warp >= kIssuerWarp) {
    const int t = warp - kIssuerWarp;
    if (t < active) {
      constexpr uint32_t idesc = idesc_bf16(128, 80, 0, 1);
      const uint32_t acc = tmem + t * kTileCols;
      for (int j = 0; j < nblk; ++j) {
        const int s = j % NS;
        if (!mbar_wait_warp(BAR_VF(s), (uint32_t)((j / NS) & 1))) { report(62); break; }
        if (!mbar_wait_warp(BAR_A(t), (uint32_t)(j & 1))) { report(63); break; }
        tc_fence_after();
        const uint32_t b_hi = desc_lo(sbase + s * C::STAGE, C::OFF_ONE - s * C::STAGE);   // the second block: the ones
        const uint32_t b_lo = desc_lo(sbase + s * C::STAGE, C::OFF_ONE + VT - s * C::STAGE);
        const int left = (int)(a.n_new - (long long)j * TB < TB ? a.n_new - (long long)j * TB : TB);
        // the K steps of half h that hold tokens, low parts first
        auto issue = [&](int h) {
          const int steps = min((left - h * (TB / 2) + 15) / 16, TB / 32);
#pragma unroll
          for (int x = 0; x < TB / 16; ++x) {
            const int ks = x % (TB / 32);
            if (ks < steps)
              umma_ts_1(acc + kHalfCols * h, acc + part_col(h, ks >> 1, ks & 1) + (x < TB / 32 ? 0 : kHiOff),
                        (x < TB / 32 ? b_lo : b_hi) + (h * (TB / 32) + ks) * 128, idesc, x > 0);
          }
        };
        const bool two = left > TB / 2;
        if (elect_one()) {
          issue(0);
          umma_commit(two ? BAR_HALF(t) : BAR_DONE(t));
          if (!two) umma_commit(BAR_VE(s));
        }
        __syncwarp();
        if (!two) continue;                              // (the last block)
        if (!mbar_wait_warp(BAR_HALF(t), (uint32_t)(j & 1))) { report(67); break; }
        tc_fence_after();
        if (elect_one()) {
          issue(1);
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
    const uint32_t tl = tmem + t * kTileCols + ((uint32_t)(qd * 32) << 16);
    uint64_t run[16];
    float run_e[4] = {0.f, 0.f, 0.f, 0.f};              // normaliser column: K steps of this warp's half of a block (0: the first)
#pragma unroll
    for (int i = 0; i < 16; ++i) run[i] = 0ull;
    // the sums of half h of a block: this warp's 32 value columns, and for one half the normaliser's K steps
    auto take = [&](int h) {
      const uint32_t from = tl + h * kHalfCols;
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        uint32_t v[16];
        tmem_ld16(from + hf * 32 + x * 16, v);
        tmem_wait_ld(v);
#pragma unroll
        for (int i = 0; i < 8; ++i) run[8 * x + i] = add2(run[8 * x + i], pack2u(v[2 * i], v[2 * i + 1]));
      }
      if (h == hf) {
        uint32_t e[8];
        tmem_ld8(from + 64, e);
        tmem_wait_ld(e);
#pragma unroll
        for (int i = 0; i < 4; ++i) run_e[i] += __uint_as_float(e[i]) + __uint_as_float(e[4 + i]);
      }
    };
    auto done = [&](uint32_t bar, int j) {
      if (ok && !mbar_wait(bar, (uint32_t)(j & 1))) { report(64); ok = false; }
      tc_fence_after();
    };
    // 16 bytes (8 features) of one token per thread and load, from the key tiles (16-byte pieces, XOR-swizzled by the row;
    // zeros past the end).  Read at the end of the block before: in global loads, the wait for the row reads below was one
    // for them too (700 of 3 700 cycles a block).
    constexpr int VPT = D / 8, NLD = TB * VPT / kGenThreads;
    uint4 kr[NLD];
    auto fetch = [&](int j) {
      if (j >= nblk) return;
      const int s = j % NS;
      if (ok && !mbar_wait(BAR_VF(s), (uint32_t)((j / NS) & 1))) { report(66); ok = false; }
#pragma unroll
      for (int i = 0; i < NLD; ++i) {
        const int idx = tid + i * kGenThreads, tok = idx / VPT, piece = idx % VPT;
        kr[i] = lds128(sbase + s * C::STAGE + VT + (piece >> 3) * VT + tok * 128 + (((piece & 7) ^ (tok & 7)) << 4));
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_VE(s));
    };
    float kmax = 0.f;
    fetch(0);
    // rows start on 256-byte boundaries, so a chunk of one is an exclusive or away (yt_off)
    const uint32_t x_row = sbase + C::OFF_Y + yt_off(fx, 0), y_row = sbase + C::OFF_Y + yt_off(fy, 0);
    for (int j = 0; j < nblk; ++j) {
      uint8_t* yt = smem + C::OFF_Y + (j & 1) * C::YT;
      const uint32_t xr = x_row + (j & 1) * C::YT, yr = y_row + (j & 1) * C::YT;
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
      if (!on) {
        fetch(j + 1);
        continue;
      }
      const long long left = a.n_new - (long long)j * TB;
      // Two K steps of either half of the block, those that hold tokens (the others are not multiplied); two chunks of 8 tokens
      // at a time: their 16 operand words and the 32 running sums fit the registers
#pragma unroll
      for (int step = 0; step < TB / 32; ++step) {
        const int half = step >> 1, tok0 = half * (TB / 2) + hf * 32 + (step & 1) * 16;
        if (step > 0 && tok0 >= left) break;
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint32_t at = (uint32_t)(tok0 / 8 + c) << 4;
          const ulonglong2 x = lds_v2(xr ^ at), y = lds_v2(yr ^ at);
          const uint32_t xw[4] = {(uint32_t)x.x, (uint32_t)(x.x >> 32), (uint32_t)x.y, (uint32_t)(x.y >> 32)};
          const uint32_t yw[4] = {(uint32_t)y.x, (uint32_t)(y.x >> 32), (uint32_t)y.y, (uint32_t)(y.y >> 32)};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const __nv_bfloat162 xv = as_bf162(xw[q]), yv = as_bf162(yw[q]), h = __hmul2(xv, yv);
            hi[4 * c + q] = as_u32(h);
            lo[4 * c + q] = as_u32(__hfma2(xv, yv, __hneg2(h)));      // exact: what rounding to eight bits left
          }
        }
        if (step == 0 && j > 0) {     // the previous block's products are done: take the second half's sums over, reuse the operands
          done(BAR_DONE(t), j - 1);
          take(1);
        }
        const uint32_t to = tl + part_col(half, hf, step & 1);
        tmem_st8(to + kHiOff, hi);
        tmem_st8(to, lo);
      }
      if (j > 0) take(0);             // the first half's, while the parts are on their way
      fetch(j + 1);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_A(t));
    }
    if (on) {
      done(BAR_DONE(t), nblk - 1);
      take(0);
      if (a.n_new - (long long)(nblk - 1) * TB > TB / 2) take(1);
    }
    asm volatile("bar.sync 1, 512;" ::: "memory");       // both tiles' products have read their stages
    if (on) {
      float* ep = (float*)(smem + C::OFF_EP) + (t * 128 + L) * 65;
#pragma unroll
      for (int i = 0; i < 16; ++i) unpack2(run[i], ep[hf * 32 + 2 * i], ep[hf * 32 + 2 * i + 1]);
      const float e = (run_e[0] + run_e[1]) + (run_e[2] + run_e[3]);
      if (hf == 0) ep[64] = e;
      else ((float*)(smem + C::OFF_E))[t * 128 + L] = e;
    }
    if (blockIdx.x == 0 && kmax > 0.f) atomicMax(kmax_bits, __float_as_int(kmax));
  }
  tc_fence_before();
  ok = __syncthreads_and(ok);
  if (warp == kIssuerWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  // a wait gave up: this CTA adds nothing, others of the head may have -- the state is undefined once the status word is set
  if (!ok) return;
  if (blockIdx.x == 0 && tid == 0) {
    hs[0] = __int_as_float(*kmax_bits);
    hs[1] = __int_as_float(__float_as_int(hs[1]) + (int)a.n_new);
  }
  // whole rows of the state: old values plus this call's sums, to both places of a pair
  constexpr int DV = D + 1, BATCH = 7, kWarps = kThreads / 32;
  const int n2rows = (a.p == 2) ? D * D : 0;
  float* st = hs + kHeader;
  auto rows_of = [&](int rr, int& row1, int& row2) -> bool {
    const int t = rr >> 7, L = rr & 127, tile = a.tile0 + pair0 + t;
    const int b = (D == 64) ? (L & 63) : L, s = (D == 64) ? 2 * tile + (L >> 6) : tile;
    if (s < D / 2 || (s == D / 2 && b < D / 2)) {
      const int o = (b + s) & (D - 1), x = min(b, o), y = max(b, o);
      row1 = x * D + y;
      row2 = y * D + x;
      return a.p == 2;
    }
    row1 = row2 = n2rows + (s == D / 2 ? D : b);
    return s != D / 2 || b == D / 2;
  };
  // a few rows of a warp at a time, so that their loads are under way together (64 heads, 40 tokens: 70 -> 43 us)
  for (int r0 = warp; r0 < active * 128; r0 += BATCH * kWarps) {
    int row1[BATCH], row2[BATCH];
    bool mine[BATCH];
    float old[BATCH][3];
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      const int rr = r0 + i * kWarps;
      mine[i] = rr < active * 128 && rows_of(rr, row1[i], row2[i]);
      if (mine[i]) {
        const float* r1 = st + (long long)row1[i] * DV;
        old[i][0] = r1[cb * 64 + lane];
        old[i][1] = r1[cb * 64 + 32 + lane];
        if (cb == 0 && lane == 0) old[i][2] = r1[D];
      }
    }
#pragma unroll
    for (int i = 0; i < BATCH; ++i) {
      if (!mine[i]) continue;
      const float* ep = (const float*)(smem + C::OFF_EP) + (r0 + i * kWarps) * 65;
      float* r1 = st + (long long)row1[i] * DV;
      float* r2 = st + (long long)row2[i] * DV;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = cb * 64 + h * 32 + lane;
        const float f = old[i][h] + ep[h * 32 + lane];
        r1[c] = f;
        if (row2[i] != row1[i]) r2[c] = f;
      }
      if (cb == 0 && lane == 0) {
        const float f = old[i][2] + (ep[64] + ((const float*)(smem + C::OFF_E))[r0 + i * kWarps]);
        r1[D] = f;
        if (row2[i] != row1[i]) r2[D] = f;
      }
    }
  }
}

template <int D>
int launch(const fastmax_problem& p, const void* k, const void* v, long long n_new, float* state, cudaStream_t st) {
  using C = AT<D>;
  CUtensorMap tv, tk;
  int rc;
  if ((rc = tma_map_bf16(&tv, v, p.bhkv, (size_t)n_new, D, TB))) return rc;
  if ((rc = tma_map_bf16(&tk, k, p.bhkv, (size_t)n_new, D, TB))) return rc;
  const long long rows = 1 + D + (p.p == 2 ? (long long)D * D : 0);
  AppArgs a{state, n_new, kHeader + rows * (D + 1), p.p, p.p == 1 ? C::FIRST_ONLY : 0,
            p.p == 1 ? C::TILES - C::FIRST_ONLY : C::TILES};
  dim3 grid((a.tiles + 1) / 2 * C::CB, p.bhkv);
  FM_CUDA_TRY(cudaFuncSetAttribute(append_tc_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
  FM_LAUNCH("fm_decode_append", st, (append_tc_kernel<D><<<grid, kThreads, C::SMEM, st>>>(tv, tk, a)));
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
