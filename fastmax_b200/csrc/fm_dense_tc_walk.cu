// Score form on the tcgen05 tensor cores, bf16, head dimension 64, equal head counts: the column loop of
// fm_dense_tc_wide.cu -- two groups of compute warps on alternate column tiles -- in CTAs that walk row tiles.
//
// fm_dense_tc_wide.cu takes 430 / 970 cycles for 128 x 64 scores of the forward / grad_k + grad_v, but a row tile's ends --
// launch, tensor memory, first loads and scores; last products, rows that are added, stores -- are another 8 000 to 10 000 that
// nothing covers.  fm_dense_tc_short.cu covers them with a second CTA on the SM, whose half of the tensor memory and registers
// leaves the loop at 730 / 1 550.  Here column tiles are counted through from one row tile to the next: operands of the next row
// tile are loaded meanwhile, its first scores follow the last ones of this, the float32 rows that a chunk adds to its result come
// by TMA while the columns pass, and the forward, which has room for two row tiles' accumulators, reads and stores a row tile's
// result when the next one's columns are done.  32 heads of 32768 in chunks of 2048, us, short-row kernels / this: forward
// 468 / 356, grad_k + grad_v 871 / 758; 240 heads of 2000, causal: forward 200 / 161.  A second buffer for the row operands and
// shorter rings pay in the forward (32 heads of 16384 in chunks of 2048 189 / 181, 160 heads of 1600 86 / 83) and not in DKDV
// (387 / 394).  What bounds it is the loop: TMEM loads,
// polynomial and TMEM stores of sixteen warps.  grad_q the same way was slower than its short kernel (0.78 to 0.98 of it):
// its S, W, E and two accumulators leave one set of each, so the warps wait for every tile's scores.
//
//   FWD   rows = queries (x = q), columns = keys (y = k, z = v):             P = f(x.y);  O += P Z,  out = O / row sum of P
//   DKDV  rows = keys (x = k, u = v), columns = queries (y = q, z = gs):     E = f'(x.y) (u.z - dvec_col), P = f(x.y);
//                                                                            grad_k += E Y,  grad_v += P Z
// Warps 0-7 are group 0 (even column tiles), 8-15 group 1 (odd ones); inside a group warp % 4 is the TMEM lane quarter and
// (warp / 4) % 2 one half of the tile's columns.  Warp 16 loads by TMA, warps 17 and 18 issue the score products of the two
// groups (forward: 17 all of them, 18 loads the Z tiles), warp 19 the accumulating products.  TMEM columns:
//   DKDV     S[2] 0 | W[2] 128 | E[2] 256 (bf16 pairs) | P[2] 320 | accumulators 384, 448
//   forward  three sets of 128 score columns at 0, 128, 256 (tile g in set g % 3), P over the S columns it came from;
//            accumulators of alternate row tiles 384, 448
// FIRST (DKDV): the first-order moment family's chunks, as in fm_dense_tc_short.cu: what a chunk's keys take from all tokens
// after it is one more product with the d x d state before the chunk's own, and its vectors are added at the end.  256 heads of
// 4096 in chunks of 512, us: 365 / 351; 64 of 2000 57.8 / 53.8; 80 of 600 31 / 27.  The forward of these chunks, tried in the
// same way, was slower than the short kernel's (232 / 247): its row tiles have 2.5 column
// tiles.
// All waits are bounded; a wait that gives up records a status and the CTA winds down.
#include <type_traits>

#include "fm_dense_tc_walk.cuh"
#include "fm_row_walk.cuh"
#include "fm_sm100.cuh"

namespace fm {

__device__ int g_walk_status = 0;

namespace {
using namespace sm100;
using namespace walk;

constexpr int D = 64;
constexpr int kThreads = 640, kComputeWarps = 16, kProducerWarp = 16, kIssuerWarp = 17, kAccIssuerWarp = 19;
constexpr int ROW_TILE = 128 * 128;
// registers a thread: at launch, and after the warpgroup that loads and issues has given some up
constexpr int kRegsLaunch = 96, kRegsCompute = 104, kRegsOther = 64;
static_assert(32 * kComputeWarps * kRegsCompute + (kThreads - 32 * kComputeWarps) * kRegsOther <= kThreads * kRegsLaunch,
              "the shares of the warpgroups add up to what the block is launched with");

template <int MODE, bool FIRST>
struct WK {
  static constexpr bool FWD = MODE == MODE_FWD, FUSED = MODE == MODE_DKDV;
  static constexpr int BN = FWD ? 128 : 64;                  // columns of a tile
  static constexpr int COL_TILE = BN * 128;
  static constexpr int ROWS = (FWD ? 1 : 2) * ROW_TILE;
  // Rings of Y and Z tiles.  DKDV: an even number, so that each barrier is waited on by one of the two groups' issuers, phase
  // after phase.
  static constexpr int NX = FUSED && !FIRST ? 1 : 2, NY = FWD ? 4 : 6, NZ = FWD ? 5 : 6;
  static constexpr int OFF_Y = NX * ROWS, OFF_Z = OFF_Y + NY * COL_TILE;
  static constexpr int ADD_HALF = 128 * 128;                 // 128 rows of 32 floats
  static constexpr int OFF_ADD = OFF_Z + NZ * COL_TILE, ADDS = (FUSED ? 2 : 1) * 2 * ADD_HALF;
  // FIRST, in place of rows to add: the state copy of the row tile's chunk, and of eight row tiles the state's normaliser column
  // (64) and constant row (65)
  static constexpr int S1_TILE = 8192, OFF_S1 = OFF_ADD, OFF_STV = OFF_S1 + NX * S1_TILE, STV = 132 * 4;
  // per compute warp 2 x 32 floats; FWD: row sums, [4][4][128]
  static constexpr int OFF_VEC = FIRST ? OFF_STV + 8 * STV : OFF_ADD + ADDS;
  static constexpr int OFF_ITEM = OFF_VEC + (FWD ? 4 * 4 * 128 : kComputeWarps * 64) * 4;   // eight row tiles (Item)
  static constexpr int OFF_BAR = OFF_ITEM + 8 * 32;
  static constexpr int NBAR = 15 + 2 * NY + 2 * NZ + 9;
  static constexpr int OFF_TMEM = OFF_BAR + NBAR * 8;
  static constexpr int SMEM = OFF_TMEM + 16 + 1024;
  static_assert(SMEM <= 227 * 1024, "shared memory");
  static constexpr int T_S = 0, T_W = 128, T_E = 256, T_P = 320, T_A = 384, SETS = 3, SET_COLS = 128;
  static constexpr int ACCS = FUSED ? 1 : 2;                 // row tiles whose accumulators there is room for
  static constexpr int FC = FUSED ? 32 : 16;                 // accumulator columns that a warp stores
  // readers of a row tile's operands: issuers; the compute warps have seen which row tile it is
  static constexpr int X_READERS = (FWD ? 1 : 2) + (FIRST ? 1 : 0) + kComputeWarps;
};

// A row tile as the producer hands it to the compute warps: also the coefficients of its head's polynomial (SQ: A2 is the
// root times the scale).
struct Item {
  int head, r0, tb, j;
  float A1, A2;
};

__device__ __forceinline__ void report(int code) { atomicCAS(&g_walk_status, 0, code); }

// SQ (DKDV): the polynomial as a square and a rest (fm_square.cuh).
template <int MODE, bool SQ, bool FIRST>
__global__ void __launch_bounds__(kThreads, 1)
walk_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmU,
            const __grid_constant__ CUtensorMap tmY, const __grid_constant__ CUtensorMap tmZ,
            const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const WalkArgs a) {
  using C = WK<MODE, FIRST>;
  constexpr bool FWD = C::FWD, FUSED = C::FUSED, rev = FUSED;
  constexpr int BN = C::BN, HB = BN / 2;         // HB: columns of one compute warp = packed columns of a group
  using Rows = RowWalk<WalkArgs, BN, rev>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + C::OFF_BAR;
  // barrier map: x[2] | x free[2] | rows to add | products of a row tile done[2] | accumulators read[2] | row sums[4] | y_full |
  // y_empty | z_full | z_empty | s_full[2] | s_free[2] | p_full[2] | pv_done[2]; forward: s_full[set] | p_full[set] |
  // set_free[set]
  constexpr int NY = C::NY, NZ = C::NZ;
  auto BAR_X = [&](int m) { return bar0 + 8u * (m % C::NX); };
  auto BAR_XE = [&](int m) { return bar0 + 8u * (2 + m % C::NX); };
  auto XPHASE = [&](int m) { return (uint32_t)(m / C::NX & 1); };
  const uint32_t BAR_ADD = bar0 + 32;
  auto BAR_DN = [&](int b) { return bar0 + 8u * (5 + b); };
  auto BAR_AF = [&](int b) { return bar0 + 8u * (7 + b); };
  auto BAR_RS = [&](int b) { return bar0 + 8u * (9 + b); };
  auto BAR_YF = [&](int s) { return bar0 + 8u * (13 + s); };
  auto BAR_YE = [&](int s) { return bar0 + 8u * (13 + NY + s); };
  auto BAR_ZF = [&](int s) { return bar0 + 8u * (13 + 2 * NY + s); };
  auto BAR_ZE = [&](int s) { return bar0 + 8u * (13 + 2 * NY + NZ + s); };
  const uint32_t bar1 = bar0 + 8u * (13 + 2 * NY + 2 * NZ);
  auto BAR_S = [&](int q) { return bar1 + 8u * q; };
  auto BAR_SFREE = [&](int q) { return bar1 + 8u * (2 + q); };
  auto BAR_P = [&](int q) { return bar1 + 8u * (4 + q); };
  auto BAR_PV = [&](int q) { return bar1 + 8u * (6 + q); };
  auto BAR_TS = [&](int t) { return bar1 + 8u * t; };
  auto BAR_TP = [&](int t) { return bar1 + 8u * (C::SETS + t); };
  auto BAR_TF = [&](int t) { return bar1 + 8u * (2 * C::SETS + t); };
  volatile uint32_t* tmem_slot = (volatile uint32_t*)(smem + C::OFF_TMEM);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (tid == 0) {
    for (int b = 0; b < C::NX; ++b) { mbar_init(BAR_X(b), 1); mbar_init(BAR_XE(b), C::X_READERS); }
    mbar_init(BAR_ADD, 1);
    for (int b = 0; b < 2; ++b) { mbar_init(BAR_DN(b), 1); mbar_init(BAR_AF(b), kComputeWarps); }
    for (int b = 0; b < 4; ++b) mbar_init(BAR_RS(b), kComputeWarps);
    for (int s = 0; s < NY; ++s) { mbar_init(BAR_YF(s), 1); mbar_init(BAR_YE(s), FUSED ? 2 : 1); }   // S, and DKDV's E Y
    for (int s = 0; s < NZ; ++s) { mbar_init(BAR_ZF(s), 1); mbar_init(BAR_ZE(s), FUSED ? 2 : 1); }   // P Z, and DKDV's W
    if constexpr (FWD) {
      for (int t = 0; t < C::SETS; ++t) {
        mbar_init(BAR_TS(t), 1);
        mbar_init(BAR_TP(t), kComputeWarps / 2);
        mbar_init(BAR_TF(t), 1);
      }
    } else {
      for (int q = 0; q < 2; ++q) {
        mbar_init(BAR_S(q), 1);
        mbar_init(BAR_SFREE(q), kComputeWarps / 2);
        mbar_init(BAR_P(q), kComputeWarps / 2);
        mbar_init(BAR_PV(q), 1);
      }
    }
    mbar_fence_init();
  }
  if (warp == kIssuerWarp) tmem_alloc(smem_u32((const void*)tmem_slot), 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // every role walks the same row tiles; g counts their column tiles
  auto has_state = [&](int r0) { return FIRST && r0 / a.chunk != a.zero_chunk; };
  Rows w;
  w.open(a);
  int g = 0;
  bool ok = true;
  if (warp >= kComputeWarps) {
    regs_down<kRegsOther>();
    // (row tile m's accumulators are read, and the rows that were added to them)
    auto read = [&](int m) { return mbar_wait(BAR_AF(m % C::ACCS), (uint32_t)((m / C::ACCS) & 1)); };
    if (warp == kProducerWarp) {
      // ================= TMA loads: row operands, Y tiles (DKDV: and Z tiles), rows to add =================
      if (lane == 0) {
        tma_prefetch_desc(&tmX);
        tma_prefetch_desc(&tmY);
        if (!FWD) { tma_prefetch_desc(&tmU); tma_prefetch_desc(&tmZ); }
      }
      // the fp32 rows to add to the result of row tile x, once those of the one before have been read
      auto load_add = [&](int m, int r0, int head) -> bool {
        if (!a.o_add) return true;
        if (m > 0 && !read(m - 1)) { report(13); return false; }
        if (lane == 0) {
          mbar_expect_tx(BAR_ADD, C::ADDS);
          for (int b = 0; b < (FUSED ? 4 : 2); ++b)
            tma_load_3d(sbase + C::OFF_ADD + b * C::ADD_HALF, b < 2 ? &tmA : &tmB, BAR_ADD, (b & 1) * 32, r0, head);
        }
        return true;
      };
      stat_t st_q = 0, st_k = 0;
      auto ask = [&](int head) {
        if (!a.stat_q) return;
        st_q = __ldg(a.stat_q + head);
        st_k = __ldg(a.stat_k + head);
      };
      if (w.live(a)) ask(w.head);
      // FIRST: the state's vectors, asked for with the row tile
      auto vectors = [&](int m, int r0, int head) {
        const float* st = a.st + (size_t)(head * a.nchunk + r0 / a.chunk) * (D + 1) * a.dvp;
        float x[5];
        const bool some = has_state(r0);
#pragma unroll
        for (int i = 0; i < 5; ++i) {
          const int e = lane + 32 * i;
          x[i] = !some || e > 128 ? 0.f : (e < 64 ? __ldg(st + (size_t)e * a.dvp + D) : __ldg(st + (size_t)D * a.dvp + (e - 64)));
        }
        float* to = (float*)(smem + C::OFF_STV + (m & 7) * C::STV);
#pragma unroll
        for (int i = 0; i < 5; ++i)
          if (lane + 32 * i <= 128) to[lane + 32 * i] = x[i];
        __syncwarp();
      };
      int last_r0 = 0, last_head = 0;
      for (; ok && w.live(a); w.next(a)) {
        const float c = a.stat_q ? stat_scale(&st_q, 0, a.lim) * stat_scale(&st_k, 0, a.lim) : 1.f;
        if (!mbar_wait(BAR_XE(w.m), XPHASE(w.m) ^ 1u)) { report(1); break; }
        if constexpr (FIRST) vectors(w.m, w.r0, w.head);
        if (lane == 0) {
          const Item it = {w.head, w.r0, w.tb, w.j, a.a1 * c, SQ ? a.sq.root * c : a.a2 * c * c};
          *(Item*)(smem + C::OFF_ITEM + (w.m & 7) * 32) = it;
          const uint32_t bar = BAR_X(w.m), to = sbase + w.m % C::NX * C::ROWS;
          mbar_expect_tx(bar, C::ROWS + (has_state(w.r0) ? C::S1_TILE : 0));
          if (has_state(w.r0))
            tma_load_3d(sbase + C::OFF_S1 + w.m % C::NX * C::S1_TILE, &tmA, bar, 0, 0, w.head * a.nchunk + w.r0 / a.chunk);
          tma_load_3d(to, &tmX, bar, 0, w.r0, w.head);
          if (!FWD) tma_load_3d(to + ROW_TILE, &tmU, bar, 0, w.r0, w.head);
        }
        {
          Rows x = w;
          x.next(a);
          if (x.live(a)) ask(x.head);
        }
        for (int i = 0; i < w.j; ++i, ++g) {
          const int s = g % NY;
          if (!mbar_wait(BAR_YE(s), (uint32_t)(((g / NY) & 1) ^ 1))) { report(1); ok = false; break; }
          if (lane == 0) {
            mbar_expect_tx(BAR_YF(s), C::COL_TILE);
            tma_load_3d(sbase + C::OFF_Y + s * C::COL_TILE, &tmY, BAR_YF(s), 0, (w.tb + i) * BN, w.head);
          }
          if (FUSED) {
            if (!mbar_wait(BAR_ZE(s), (uint32_t)(((g / NZ) & 1) ^ 1))) { report(1); ok = false; break; }
            if (lane == 0) {
              mbar_expect_tx(BAR_ZF(s), C::COL_TILE);
              tma_load_3d(sbase + C::OFF_Z + s * C::COL_TILE, &tmZ, BAR_ZF(s), 0, (w.tb + i) * BN, w.head);
            }
          }
          // some columns ahead of it: DKDV's result is stored at the end of its row tile, the forward's at that of the next
          if (i == min(2, w.j - 1)) {
            if (FUSED) ok = load_add(w.m, w.r0, w.head);
            else if (w.m > 0) ok = load_add(w.m - 1, last_r0, last_head);
            if (!ok) break;
          }
        }
        last_r0 = w.r0;
        last_head = w.head;
      }
      // no more row tiles
      if (ok && mbar_wait(BAR_XE(w.m), XPHASE(w.m) ^ 1u) && lane == 0) {
        ((Item*)(smem + C::OFF_ITEM + (w.m & 7) * 32))->j = 0;
        mbar_arrive(BAR_X(w.m));
      }
      __syncwarp();
      if (ok && FWD && w.m > 0) load_add(w.m - 1, last_r0, last_head);
      __syncwarp();
    } else if (FWD && warp == kIssuerWarp + 1) {
      // ================= TMA loads of the forward's Z tiles =================
      if (lane == 0) tma_prefetch_desc(&tmZ);
      for (; ok && w.live(a); w.next(a))
        for (int i = 0; i < w.j; ++i, ++g) {
          const int s = g % NZ;
          if (!mbar_wait(BAR_ZE(s), (uint32_t)(((g / NZ) & 1) ^ 1))) { report(14); ok = false; break; }
          if (lane == 0) {
            mbar_expect_tx(BAR_ZF(s), C::COL_TILE);
            tma_load_3d(sbase + C::OFF_Z + s * C::COL_TILE, &tmZ, BAR_ZF(s), 0, (w.tb + i) * BN, w.head);
          }
        }
    } else if (warp == kIssuerWarp || warp == kIssuerWarp + 1) {
      // ================= issuers of the S / W products (whole warp, one elected lane issues) =================
      constexpr uint32_t idescS = idesc_bf16(128, BN, 0, 0);
      const uint32_t y_k = desc_lo(sbase + C::OFF_Y, 16), z_k = desc_lo(sbase + C::OFF_Z, 16);      // K-major views
      const int q = warp - kIssuerWarp;
      for (; ok && w.live(a); g += w.j, w.next(a)) {
        if (!mbar_wait_warp(BAR_X(w.m), XPHASE(w.m))) { report(2); break; }
        const uint32_t x_lo = desc_lo(sbase + w.m % C::NX * C::ROWS, 16), u_lo = x_lo + (ROW_TILE >> 4);
        for (int gi = FWD ? g : g + ((g ^ q) & 1); gi < g + w.j; gi += FWD ? 1 : 2) {
          const int s = gi % NY;
          // the tiles have normally been loaded long ago: checking them first keeps that check out of the way from the score
          // region's release to the next scores
          if (!mbar_wait_warp(BAR_YF(s), (uint32_t)((gi / NY) & 1))) { report(3); ok = false; break; }
          if (FUSED && !mbar_wait_warp(BAR_ZF(s), (uint32_t)((gi / NZ) & 1))) { report(3); ok = false; break; }
          if (FWD) {
            // S of tile g goes to set g % 3 once the accumulating product of tile g - 3 has read that set's P
            if (gi >= C::SETS && !mbar_wait_warp(BAR_TF(gi % C::SETS), (uint32_t)((gi / C::SETS - 1) & 1))) {
              report(4);
              ok = false;
              break;
            }
          } else {
            if (gi >= 2 && !mbar_wait_warp(BAR_SFREE(q), (uint32_t)(((gi >> 1) - 1) & 1))) { report(4); ok = false; break; }
          }
          tc_fence_after();
          const uint32_t y_lo = y_k + (uint32_t)s * (C::COL_TILE >> 4);
          if (elect_one()) {
            if constexpr (FWD) {
              umma_ss_k64(tmem + gi % C::SETS * C::SET_COLS, x_lo, y_lo, idescS);
              umma_commit(BAR_TS(gi % C::SETS));
              umma_commit(BAR_YE(s));
            } else {
              umma_ss_k64(tmem + C::T_S + q * BN, x_lo, y_lo, idescS);
              umma_ss_k64(tmem + C::T_W + q * BN, u_lo, z_k + (uint32_t)s * (C::COL_TILE >> 4), idescS);
              umma_commit(BAR_S(q));
              umma_commit(BAR_YE(s));
              umma_commit(BAR_ZE(s));
            }
          }
          __syncwarp();
        }
        if (ok && elect_one()) umma_commit(BAR_XE(w.m));
        __syncwarp();
      }
      __syncwarp();
    } else if (warp == kAccIssuerWarp) {
      // ================= issuer of the accumulating products =================
      constexpr uint32_t idescO = idesc_bf16(128, D, 0, 1);
      const uint32_t y_mn = desc_lo(sbase + C::OFF_Y, C::COL_TILE), z_mn = desc_lo(sbase + C::OFF_Z, C::COL_TILE);   // MN-major
      for (; ok && w.live(a); w.next(a)) {
        if (w.m >= C::ACCS && !__all_sync(0xffffffffu, read(w.m - C::ACCS))) { report(6); break; }
        const uint32_t acc = tmem + C::T_A + w.m % C::ACCS * D;
        const uint32_t state = has_state(w.r0) ? 1u : 0u;
        if constexpr (FIRST) {
          // what the chunk's keys take from all tokens after it: u S1^T and x S1
          if (state) {
            if (!mbar_wait_warp(BAR_X(w.m), XPHASE(w.m))) { report(6); break; }
            tc_fence_after();
            const uint32_t s1 = sbase + C::OFF_S1 + w.m % C::NX * C::S1_TILE;
            const uint32_t x_lo = desc_lo(sbase + w.m % C::NX * C::ROWS, 16), s_mn = desc_lo(s1, 8192);
            if (elect_one()) {
              umma_ss_k64(acc, x_lo + (ROW_TILE >> 4), desc_lo(s1, 16), idesc_bf16(128, D, 0, 0));
              umma_ss_kmn_steps<4>(acc + D, x_lo, s_mn, idescO, 0u);
              umma_commit(BAR_XE(w.m));
            }
          } else if (elect_one()) {
            mbar_arrive(BAR_XE(w.m));
          }
          __syncwarp();
        }
        for (int i = 0; i < w.j; ++i, ++g) {
          const int s = g % NZ, q = g & 1, set = g % C::SETS;
          if (!mbar_wait_warp(BAR_ZF(s), (uint32_t)((g / NZ) & 1)) ||
              (FUSED && !mbar_wait_warp(BAR_YF(s), (uint32_t)((g / NY) & 1))) ||
              !mbar_wait_warp(FWD ? BAR_TP(set) : BAR_P(q), (uint32_t)((FWD ? g / C::SETS : g >> 1) & 1))) {
            report(5);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t z_lo = z_mn + (uint32_t)s * (C::COL_TILE >> 4);
          if (elect_one()) {
            if constexpr (FWD) {
              // the warp that read columns [32 c, 32 c + 32) of the set left 16 packed columns at 32 c
#pragma unroll
              for (int ks = 0; ks < BN / 16; ++ks)
                umma_ts_1(acc, tmem + set * C::SET_COLS + (ks >> 1) * 32 + (ks & 1) * 8, z_lo + ks * 128, idescO,
                          (i > 0 || ks > 0) ? 1u : state);
              umma_commit(BAR_TF(set));
            } else {
              umma_ts_steps<BN / 16>(acc, tmem + C::T_E + q * HB, y_mn + (uint32_t)s * (C::COL_TILE >> 4), idescO,
                                     i > 0 ? 1u : state);
              umma_ts_steps<BN / 16>(acc + D, tmem + C::T_P + q * HB, z_lo, idescO, i > 0 ? 1u : state);
              umma_commit(BAR_PV(q));
              umma_commit(BAR_YE(s));
            }
            umma_commit(BAR_ZE(s));
            if (i + 1 == w.j) umma_commit(BAR_DN(w.m % C::ACCS));
          }
          __syncwarp();
        }
      }
      __syncwarp();
    }
  } else {
    // ================= compute warps =================
    regs_up<kRegsCompute>();
    const int gp = warp >> 3, cpart = (warp >> 2) & 1, qd = warp & 3, part4 = warp >> 2, rl = qd * 32 + lane;
    const uint32_t tl = tmem + ((uint32_t)(qd * 32) << 16);
    float* myvec = (float*)(smem + C::OFF_VEC) + warp * 64;
    const uint32_t myvec_s = sbase + C::OFF_VEC + warp * 256;
    const uint64_t A0v = pack2(a.a0, a.a0);
    // dvec of this lane's column in a column tile
    auto fetch_vec = [&](int tile, int head) -> float {
      const int col = tile * BN + cpart * 32 + lane;
      return col < a.ncols ? __ldg(a.dvec + (size_t)head * a.ncols + col) : 0.f;
    };
    // row tile m, written by the producer before its operands are loaded; waits for it
    auto item = [&](int m) -> Item {
      const uint32_t at = sbase + C::OFF_ITEM + (m & 7) * 32;
      const ulonglong2 v = lds_v2(at), f = lds_v2(at + 16);
      return {(int)(uint32_t)v.x, (int)(v.x >> 32), (int)(uint32_t)v.y, (int)(v.y >> 32), __uint_as_float((uint32_t)f.x),
              __uint_as_float((uint32_t)(f.x >> 32))};
    };
    auto open = [&](int m, Item& it) -> bool {
      if (!mbar_wait(BAR_X(m), XPHASE(m))) { report(11); return false; }
      it = item(m);
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_XE(m));
      return true;
    };
    // The result of a row tile: this warp's FC accumulator columns.
    auto finish = [&](int m, int head, int r0, float pre, float A1) -> bool {
      const int ab = m % C::ACCS, row = r0 + rl;
      const bool row_ok = row < a.nrows, second = FUSED && part4 >= 2;
      const int cc = FUSED ? (part4 & 1) * 32 : part4 * 16;
      const size_t grow = (size_t)head * a.nrows + (row_ok ? row : 0);
      const size_t orow = FWD ? out_row(head, row_ok ? row : 0, a.nrows, a.o_heads) : grow;
      const __nv_bfloat16* xr = FUSED && !second && a.dots && row_ok ? (const __nv_bfloat16*)a.x + grow * D + cc : nullptr;
      __nv_bfloat16* dst = (__nv_bfloat16*)(second ? a.o2 : a.o) + orow * D + cc;
      const bool wide = (((uintptr_t)dst | (uintptr_t)xr) & 31) == 0;
      uint32_t xw[C::FC / 16][8];                   // asked for before the waits
      if (xr) {
#pragma unroll
        for (int h = 0; h < C::FC / 16; ++h) ldg32(xr + 16 * h, xw[h], wide);
      }
      float rowsum = FWD && a.den_add && row_ok ? __ldg(a.den_add + grow) : 0.f, scale = pre;
      if (!mbar_wait(BAR_DN(ab), (uint32_t)((m / C::ACCS) & 1))) { report(10); return false; }
      if (a.o_add && !mbar_wait(BAR_ADD, (uint32_t)(m & 1))) { report(12); return false; }
      if constexpr (FWD) {
        if (!mbar_wait(BAR_RS(m & 3), (uint32_t)((m >> 2) & 1))) { report(12); return false; }
        const float* sums = (const float*)(smem + C::OFF_VEC) + (m & 3) * 512 + rl;
        rowsum += (sums[0] + sums[128]) + (sums[256] + sums[384]);
        scale = 1.0f / rowsum;
        if (part4 == 0 && row_ok) a.den_out[grow] = rowsum;
      }
      tc_fence_after();
      uint32_t ov[C::FC];
      const uint32_t at = tl + C::T_A + ab * D + (second ? D : 0) + cc;
      if constexpr (FUSED) tmem_ld32(at, ov);
      else tmem_ld16(at, ov);
      tmem_wait_ld(ov);
      // (accumulator * factor left out of E' + row to add), forward: (accumulator + row to add) / row sum
      float f[C::FC];
#pragma unroll
      for (int e = 0; e < C::FC; ++e) f[e] = FUSED ? __uint_as_float(ov[e]) * pre : __uint_as_float(ov[e]);
      if constexpr (FIRST) {
        // grad_k: normaliser column, grad_v: constant row
        const uint32_t vec = sbase + C::OFF_STV + (m & 7) * C::STV + (second ? 256 : 0) + cc * 4;
        const float mul = second ? a.a0 : A1;
#pragma unroll
        for (int e = 0; e < C::FC / 4; ++e) {
          const ulonglong2 v = lds_v2(vec + 16 * e);
          float x[4];
          unpack2(v.x, x[0], x[1]);
          unpack2(v.y, x[2], x[3]);
#pragma unroll
          for (int i = 0; i < 4; ++i) f[4 * e + i] = fmaf(mul, x[i], f[4 * e + i]);
        }
      } else if (a.o_add) {
        const uint32_t row_s = sbase + C::OFF_ADD + (second ? 2 * C::ADD_HALF : 0) + (cc >> 5) * C::ADD_HALF + rl * 128;
#pragma unroll
        for (int p = 0; p < C::FC / 4; ++p) {
          const ulonglong2 v = lds_v2(row_s + (((((cc & 31) >> 2) + p) ^ (rl & 7)) << 4));
          float x[4];
          unpack2(v.x, x[0], x[1]);
          unpack2(v.y, x[2], x[3]);
#pragma unroll
          for (int e = 0; e < 4; ++e) f[4 * p + e] += x[e];
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(BAR_AF(ab));
      float part = 0.f;
      if (row_ok) {
#pragma unroll
        for (int h = 0; h < C::FC / 16; ++h) {
          uint32_t v[8];
          if (FWD) {
#pragma unroll
            for (int e = 0; e < 16; ++e) f[16 * h + e] *= scale;
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = pack_bf16(f[16 * h + 2 * e], f[16 * h + 2 * e + 1]);
          stg32(dst + 16 * h, v, wide);
          if (xr) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              part = fmaf(f[16 * h + 2 * e], __uint_as_float(xw[h][e] << 16), part);
              part = fmaf(f[16 * h + 2 * e + 1], __uint_as_float(xw[h][e] & 0xFFFF0000u), part);
            }
          }
        }
      }
      if (FUSED && !second && a.dots) {
#pragma unroll
        for (int k = 16; k >= 1; k >>= 1) part += __shfl_xor_sync(0xffffffffu, part, k);
        if (lane == 0) atomicAdd(a.dots + head, part);
      }
      return true;
    };
    Item it;
    ok = open(0, it);
    int m = 0;
    float nxt_raw = 0.f;                          // dvec of this lane's column in the group's first column tile
    if (ok && rev && gp < it.j) nxt_raw = fetch_vec(it.tb + gp, it.head);
    while (ok && it.j > 0) {
      const int first = (g ^ gp) & 1;              // the group's first column tile of this row tile
      const float A1 = it.A1, A2 = it.A2;
      const uint64_t A1v = pack2(A1, A1), A2v = pack2(A2, A2), A2d = pack2(2.f * A2, 2.f * A2);
      const uint64_t Bv = a.sq.shift, Cv = a.sq.rest;
      const int row = it.r0 + rl;
      int limcol = a.ncols - 1, lowcol = 0;        // columns kept for this row: lowcol <= col <= limcol
      if (a.mask) {
        if (rev) lowcol = row - a.off;
        else limcol = min(limcol, row + a.off);
      }
      const int wrow_lo = it.r0 + qd * 32, wrow_hi = wrow_lo + 31;
      float nxt = nxt_raw;
      uint64_t rs2[4] = {0ull, 0ull, 0ull, 0ull};  // forward: row sums
      for (int i = first; i < it.j; i += 2) {
        const int gi = g + i, n = gi >> 1, set = gi % C::SETS;
        const float cur = -nxt;
        if (rev && i + 2 < it.j) nxt = fetch_vec(it.tb + i + 2, it.head);
        const uint32_t tset = tl + set * C::SET_COLS;
        if (!mbar_wait(FWD ? BAR_TS(set) : BAR_S(gp), (uint32_t)((FWD ? gi / C::SETS : n) & 1))) { report(7); ok = false; break; }
        tc_fence_after();
        const uint32_t vec_s = myvec_s + (n & 1) * 128;
        if (rev) {
          myvec[(n & 1) * 32 + lane] = cur;
          __syncwarp();
        }
        // the warp's HB columns in passes of 32
#pragma unroll
        for (int ps = 0; ps < HB / 32; ++ps) {
          uint32_t sv[32], wv[FWD ? 1 : 32];
          tmem_ld32(FWD ? tset + cpart * HB + ps * 32 : tl + C::T_S + gp * BN + cpart * HB + ps * 32, sv);
          if constexpr (!FWD) {
            tmem_ld32(tl + C::T_W + gp * BN + cpart * HB + ps * 32, wv);
            tmem_wait_ld(sv, wv);
            // S and W of this tile are in registers: the group's next tile may be issued
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR_SFREE(gp));
          } else {
            tmem_wait_ld(sv);
          }
          const int c0 = (it.tb + i) * BN + cpart * HB + ps * 32;    // first of these 32 columns
          bool need_mask = (c0 + 32 > a.ncols);
          if (a.mask) need_mask = need_mask || (rev ? (c0 < wrow_hi - a.off) : (c0 + 31 > wrow_lo + a.off));
          // the mask test stays outside the element loops so that each loop is one basic block of independent pairs; E and
          // P of a pair are formed together so that S and W die pair by pair
          uint32_t pe[16], pp[FUSED ? 16 : 1];
          ulonglong2 nd2 = make_ulonglong2(0ull, 0ull);
          auto element = [&](int e, auto masked) {
            const uint64_t s2 = pack2u(sv[2 * e], sv[2 * e + 1]);
            bool z0 = false, z1 = false;
            if constexpr (decltype(masked)::value) {
              const int col = c0 + 2 * e;
              z0 = col > limcol || col < lowcol;
              z1 = col + 1 > limcol || col + 1 < lowcol;
            }
            auto round2 = [&](uint64_t v) -> uint32_t {
              if constexpr (!decltype(masked)::value) return pack_bf16_2(v);
              float v0, v1;
              unpack2(v, v0, v1);
              return pack_bf16(z0 ? 0.f : v0, z1 ? 0.f : v1);
            };
            if constexpr (FWD) {
              const uint64_t p2 = fma2(fma2(A2v, s2, A1v), s2, A0v);
              pe[e] = round2(p2);
              // Tiles on the causal diagonal (and ragged last tiles) hold most of what an early row sees, so their share
              // of the row sum is taken from the ROUNDED values the product will use: numerator and denominator then carry
              // the same rounding, and a row with one key returns its value exactly.
              rs2[e & 3] = add2(rs2[e & 3], decltype(masked)::value ? pack2u(pe[e] << 16, pe[e] & 0xFFFF0000u) : p2);
            } else {
              if ((e & 1) == 0) nd2 = lds_v2(vec_s + (e >> 1) * 16);   // four column values per load
              const uint64_t ndl = (e & 1) ? nd2.y : nd2.x;
              const uint64_t t2 = SQ ? fma2(s2, A2v, Bv) : fma2(A2d, s2, A1v);
              pe[e] = round2(mul2(t2, add2(pack2u(wv[2 * e], wv[2 * e + 1]), ndl)));
              pp[e] = round2(SQ ? fma2(t2, t2, Cv) : fma2(fma2(A2v, s2, A1v), s2, A0v));
            }
          };
          if (!need_mask) {
#pragma unroll
            for (int e = 0; e < 16; ++e) element(e, std::false_type());
          } else {
#pragma unroll
            for (int e = 0; e < 16; ++e) element(e, std::true_type());
          }
          // the group's previous products must have consumed E and P before they are overwritten
          if (FUSED && n > 0) {
            if (!mbar_wait(BAR_PV(gp), (uint32_t)((n - 1) & 1))) { report(9); ok = false; break; }
            tc_fence_after();
          }
          // forward: P over the first 16 of the 32 S columns this pass has just read
          tmem_st16(FWD ? tset + cpart * HB + ps * 32 : tl + C::T_E + gp * HB + cpart * (HB / 2), pe);
          if constexpr (FUSED) tmem_st16(tl + C::T_P + gp * HB + cpart * (HB / 2), pp);
        }
        if (!ok) break;
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(FWD ? BAR_TP(set) : BAR_P(gp));
      }
      if (!ok) break;
      if constexpr (FWD) {
        float lo, hi;
        unpack2(add2(add2(rs2[0], rs2[1]), add2(rs2[2], rs2[3])), lo, hi);
        ((float*)(smem + C::OFF_VEC))[(m & 3) * 512 + part4 * 128 + rl] = lo + hi;
        __syncwarp();
        if (lane == 0) mbar_arrive(BAR_RS(m & 3));
      }
      Item next;
      if (!(ok = open(m + 1, next))) break;
      if (rev && (((g + it.j) ^ gp) & 1) < next.j) nxt_raw = fetch_vec(next.tb + (((g + it.j) ^ gp) & 1), next.head);
      // SQ: the factor left out of E'
      if (FUSED) {
        ok = finish(m, it.head, it.r0, SQ && part4 < 2 ? 2.f * A2 : 1.f, A1);
      } else if (m > 0) {
        const Item before = item(m - 1);
        ok = finish(m - 1, before.head, before.r0, 1.f, 0.f);
      }
      g += it.j;
      it = next;
      ++m;
    }
    if (ok && !FUSED && m > 0) {
      const Item before = item(m - 1);
      finish(m - 1, before.head, before.r0, 1.f, 0.f);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kIssuerWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// the compute warps wait for registers that the block must have been launched with
template <int MODE, bool SQ, bool FIRST>
bool has_registers() {
  static std::atomic<int> regs{0};
  return launch_registers(walk_kernel<MODE, SQ, FIRST>, &regs) >= kRegsLaunch;
}

template <int MODE, bool SQ, bool FIRST>
int start(const Ctx& c, const char* name, unsigned grid, const CUtensorMap& tx, const CUtensorMap& tu, const CUtensorMap& ty,
          const CUtensorMap& tz, const CUtensorMap& ta, const CUtensorMap& tb, const WalkArgs& a) {
  using C = WK<MODE, FIRST>;
  FM_CUDA_TRY(cudaFuncSetAttribute(walk_kernel<MODE, SQ, FIRST>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
  FM_LAUNCH(name, c.stream, (walk_kernel<MODE, SQ, FIRST><<<grid, kThreads, C::SMEM, c.stream>>>(tx, tu, ty, tz, ta, tb, a)));
  FM_CUDA_TRY(cudaGetLastError());
  return FASTMAX_OK;
}

template <int MODE>
int launch(const Ctx& c, const char* name, const void* x, const void* u, const void* y, const void* z, int nrows, int ncols,
           WalkArgs a, const FirstState* fs) {
  const fastmax_problem& p = c.p;
  if (p.bh == 0 || nrows == 0) return FASTMAX_OK;
  CUtensorMap tx, tu, ty, tz, ta, tb;
  int rc;
  if ((rc = tma_map_bf16(&tx, x, p.bh, nrows, D, 128))) return rc;
  if ((rc = tma_map_bf16(&tu, u ? u : x, p.bh, nrows, D, 128))) return rc;
  if ((rc = tma_map_bf16(&ty, y, p.bh, ncols, D, WK<MODE, false>::BN))) return rc;
  if ((rc = tma_map_bf16(&tz, z, p.bh, ncols, D, WK<MODE, false>::BN))) return rc;
  ta = tb = tx;
  if (a.o_add && (rc = tma_map_f32_rows(&ta, a.o_add, p.bh, nrows))) return rc;
  if (a.o2_add && (rc = tma_map_f32_rows(&tb, a.o2_add, p.bh, nrows))) return rc;
  if (fs) {
    // the first-order chunks come here without passing dense_tc_forward / _backward, which check this for the others
    const uintptr_t bases = (uintptr_t)x | (uintptr_t)u | (uintptr_t)y | (uintptr_t)z | (uintptr_t)a.o | (uintptr_t)a.o2;
    if (bases & 15) return fail(FASTMAX_E_ARG, "the tensor-core family needs 16-byte aligned tensors");
    a.nchunk = (nrows + a.chunk - 1) / a.chunk;
    a.st = fs->states;
    a.dvp = moment_dims(D, 1).dvp;
    a.zero_chunk = fs->zero_chunk;
    if ((rc = tma_map_bf16(&ta, fs->s1b, (size_t)p.bh * a.nchunk, D, D, D))) return rc;
  }
  a.x = x;
  a.heads = p.bh;
  a.nrows = nrows;
  a.ncols = ncols;
  a.ntr = (nrows + 127) / 128;
  a.ratio = 1;
  a.off = p.nk - p.nq;
  a.mask = p.mask;
  a.a0 = p.a0;
  a.a1 = p.a1;
  a.a2 = p.p == 2 ? p.a2 : 0.f;
  a.lim = p.lim;
  a.order = row_order(p, a.heads, a.ntr, 1, a.chunk);
  const long long blocks = (long long)a.heads * a.ntr;
  if (blocks > 0x7FFF0000LL) return fail(FASTMAX_E_ARG, "heads x row tiles = %lld exceeds the grid limit", blocks);
  const unsigned grid = (unsigned)(blocks < 148 ? blocks : 148);
  if (fs) return start<MODE, false, MODE == MODE_DKDV>(c, name, grid, tx, tu, ty, tz, ta, tb, a);
  if (MODE == MODE_DKDV && square_form(a.a0, a.a1, a.a2, &a.sq)) return start<MODE, MODE == MODE_DKDV, false>(c, name, grid, tx, tu, ty, tz, ta, tb, a);
  return start<MODE, false, false>(c, name, grid, tx, tu, ty, tz, ta, tb, a);
}

}  // namespace

bool dense_tc_walk_runs(bool forward) {
  if (forward) return has_registers<MODE_FWD, false, false>();
  return has_registers<MODE_DKDV, false, false>() && has_registers<MODE_DKDV, true, false>() && has_registers<MODE_DKDV, false, true>();
}

int dense_tc_walk_forward(const Ctx& c, const void* q, const void* k, const void* v, const WalkArgs& a) {
  return launch<MODE_FWD>(c, "fm_dense_tc_fwd", q, nullptr, k, v, c.p.nq, c.p.nk, a, nullptr);
}
int dense_tc_walk_dkdv(const Ctx& c, const void* k, const void* v, const void* q, const void* gs, const WalkArgs& a,
                       const FirstState* fs) {
  return launch<MODE_DKDV>(c, "fm_dense_tc_dkdv", k, v, q, gs, c.p.nk, c.p.nq, a, fs);
}

int tc_walk_status(int* out, cudaStream_t stream) {
  FM_CUDA_TRY(cudaMemcpyFromSymbolAsync(out, g_walk_status, sizeof(int), 0, cudaMemcpyDeviceToHost, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}
int tc_walk_status_reset(cudaStream_t stream) {
  const int zero = 0;
  FM_CUDA_TRY(cudaMemcpyToSymbolAsync(g_walk_status, &zero, sizeof(int), 0, cudaMemcpyHostToDevice, stream));
  FM_CUDA_TRY(cudaStreamSynchronize(stream));
  return FASTMAX_OK;
}

}  // namespace fm
