// Host-side orchestration of the moment-state form: which kernels run, in which
// order, on which slices of the caller's workspace.  The same stages serve a
// whole sequence on one GPU and one contiguous shard of a sequence split over
// several GPUs; in the sharded case the caller exchanges the per-shard totals
// between the stages (see include/fastmax_b200.h).
#include "fm_common.cuh"

namespace fm {

static size_t up256(size_t x) { return (x + 255) / 256 * 256; }

// Tokens per chunk of causal first-order problems, for the kernels it was measured with; 0 for the others (tensor cores
// switched off, float32 operands too large for the split kernels), which keep 2048 and the rate model of moments_faster.
// What a token costs is its own chunk in score form, so short chunks win.  Measured, ms per step at 256 / 512 / 1024 / 2048:
//   bf16 on the tensor cores, 256 heads x 4096: d = 64 1.30, 1.30, 1.97, 2.41 (the last two with separate read-outs); d = 128
//   4.19, 3.65, 3.79, 4.60.  float32 with the split score kernels, d = 32, 8 heads x 4096: 0.31, 0.42, 0.64, 1.06.
//   Everything on the CUDA cores, 256 heads x 2000: float32 d = 16 2.39, 3.21, 4.96, 8.19; d = 128 20.8, 25.6, 35.8, 55.7;
//   bf16 d = 32 3.81, 5.10, 7.67, 12.8.
int first_order_chunk(const fastmax_problem& p) {
  if (p.p != 1 || !p.mask) return 0;
  if (p.dtype == FASTMAX_BF16) return first_tc_supports(p) ? 512 : (p.d <= 32 ? 256 : 0);
  return dense_split_supports(p) || (p.d != 32 && p.d != 64) ? 256 : 0;
}

// Tokens per chunk.  Second order: 2048, measured best for the tensor-core kernels (ms per step at 1024 / 1536 / 2048 / 3072 /
// 4096: 8 heads x 65536 3.63, 3.07, 3.07, 3.36, 3.49; 512 x 10 000 28.3, 24.1, 24.0, 25.9, 26.7): a chunk's state is as large as
// its tokens, so larger chunks mean fewer states to build, scan and convert, and more in-chunk score work.  First order, causal: first_order_chunk; unmasked: there is no
// in-chunk part and every chunk only adds a state to sum.
int moments_chunk(const fastmax_problem& p) {
  int L = p.chunk > 0 ? p.chunk : first_order_chunk(p);
  if (L == 0) L = 2048;
  L = (L + 255) / 256 * 256;
  return L;
}

size_t moment_state_bytes(const fastmax_problem& p, int n) {
  const MomentDims m = moment_dims(p.d, p.p);
  const int L = moments_chunk(p);
  return up256(sizeof(float) * (size_t)p.bh * ((n + L - 1) / L) * m.f * m.dvp);
}
size_t moment_total_bytes(const fastmax_problem& p) {
  const MomentDims m = moment_dims(p.d, p.p);
  return up256(sizeof(float) * (size_t)p.bh * m.f * m.dvp);
}

// bf16 copies of the chunk states that the tensor-core read-outs multiply: second order, in one layout for read-outs of type
// A and one for type B, or first order.  The room for them holds one layout.
static size_t copies_a_bytes(const fastmax_problem& p, int mats) {
  return moments_tc_supports(p) ? up256(moments_tc_copy_a_bytes(mats)) : 0;
}
static size_t copies_b_bytes(const fastmax_problem& p, int mats) {
  return moments_tc_supports(p) ? up256(moments_tc_copy_b_bytes(mats)) : 0;
}
// Where the copies of `mats` states go that are read out in one kind (mode 0: A, 1: B) or both (2): `s16`, and for both kinds
// the type B ones lie in the rows of n tokens that the type A read-out will write, which therefore comes second.  Chunks
// that are too short for that (of less than 1216 tokens) use s16 for one kind after the other: c.a == c.b.
static StateCopies copies_at(const fastmax_problem& p, int mode, void* s16, float* rows_a, int n, int mats) {
  StateCopies c;
  if (mode != 1) c.a = s16;
  if (mode != 0) c.b = s16;
  if (mode == 2 && copies_b_bytes(p, mats) <= sizeof(float) * (size_t)p.bh * n * p.d) c.b = rows_a;
  return c;
}
// the layouts of `c` that can be written at once
static StateCopies at_once(StateCopies c) {
  if (c.a == c.b) c.a = nullptr;
  return c;
}
size_t state16_bytes(const fastmax_problem& p, int n) {
  const int L = moments_chunk(p);
  const int mats = p.bh * ((n + L - 1) / L);
  const size_t a = copies_a_bytes(p, mats), b = copies_b_bytes(p, mats);
  if (a > 0) return a > b ? a : b;
  return first_tc_supports(p) ? up256(first_tc_copy_bytes(p, mats)) : 0;
}

// the type B copies of the key/value chunk prefixes, which a causal forward leaves for the backward's grad_q
size_t moment_kept16_bytes(const fastmax_problem& p) {
  const int L = moments_chunk(p);
  return copies_b_bytes(p, p.bh * ((p.nk + L - 1) / L));
}

bool moments_all_tc(const fastmax_problem& p) {
  return dense_tc_supports(p) && first_tc_supports(p) && (p.p == 1 || moments_tc_supports(p));
}

// Heads are the y or z dimension of several of the family's grids, which ends at 65535; the score families have
// one-dimensional grids.
bool moments_supports(const fastmax_problem& p) {
  return p.bh == p.bhkv && p.bh <= 65535 && (!p.mask || p.nq == p.nk);
}

// Causal p = 1 at d = 64: the score kernels of the chunks read the states themselves, so there is no read-out pass
// and no fp32 rows between two kernels.
static bool first_fused(const fastmax_problem& p) {
  return p.p == 1 && p.mask && p.d == 64 && p.nq == p.nk && first_tc_supports(p) && dense_tc_wide_supports(p);
}

// Workspace of the one-call forward: [states][total][o_add][den_add][bf16 copies][float32 operand parts].  The fused
// first-order path has no fp32 rows between two kernels and no total (256 heads x 2048, bf16: 27 MB instead of 167).
MomFwdWs moments_fwd_layout(const fastmax_problem& p) {
  MomFwdWs w;
  w.states = 0;
  w.total = w.states + moment_state_bytes(p, p.nk);
  const size_t rows = first_fused(p) ? 0 : (size_t)p.bh * p.nq;
  w.o_add = w.total + (rows ? moment_total_bytes(p) : 0);
  w.den_add = w.o_add + up256(sizeof(float) * rows * p.d);
  w.s16 = w.den_add + up256(sizeof(float) * rows);
  w.split = w.s16 + state16_bytes(p, p.nk);
  w.bytes = w.split + (p.mask && dense_split_supports(p) ? dense_split_fwd_bytes(p) : 0);
  return w;
}
// Workspace of the one-call backward:
// [dots][delta][dvec][gs][states][total][gq_add][gk_add][gv_add][bf16 copies][float32 operand parts]
MomBwdWs moments_bwd_layout(const fastmax_problem& p) {
  MomBwdWs w;
  w.dots = 0;
  w.delta = up256(sizeof(float) * (size_t)(p.bh + p.bhkv));
  w.dvec = w.delta + up256(sizeof(float) * (size_t)p.bh * p.nq);
  w.gs = w.dvec + up256(sizeof(float) * (size_t)p.bh * p.nq);
  w.states = w.gs + (dense_tc_supports(p) ? up256((size_t)2 * p.bh * p.nq * p.d) : 0);
  w.total = w.states + moment_state_bytes(p, p.nk > p.nq ? p.nk : p.nq);
  const bool fused = first_fused(p);    // as in the forward: 98 MB instead of 505
  w.gq_add = w.total + (fused ? 0 : moment_total_bytes(p));
  w.gk_add = w.gq_add + (fused ? 0 : up256(sizeof(float) * (size_t)p.bh * p.nq * p.d));
  w.gv_add = w.gk_add + (fused ? 0 : up256(sizeof(float) * (size_t)p.bhkv * p.nk * p.d));
  w.s16 = w.gv_add + (fused ? 0 : up256(sizeof(float) * (size_t)p.bhkv * p.nk * p.d));
  w.split = w.s16 + state16_bytes(p, p.nk > p.nq ? p.nk : p.nq);
  w.bytes = w.split + (p.mask && dense_split_supports(p) ? dense_split_bwd_bytes(p) : 0);
  return w;
}

int moments_build_states(const Ctx& c, int n, const void* y, const void* z, const float* den,
                         const float* delta, int ext, const void* gs, const float* dvec, float* states) {
  const fastmax_problem& p = c.p;
  const int L = moments_chunk(p);
  const bool tc2 = moments_tc_supports(p), tc1 = first_tc_supports(p);
  int rc;
  // second-order rows: tensor cores where built, else everything on the CUDA cores
  if (p.p == 2) {
    if (!tc2) return moments_chunk_state(c, p.bh, n, L, y, z, den, delta, ext, states);
    if ((rc = moments_tc_chunk_state(c, p.bh, n, L, y, ext ? gs : z, ext ? dvec : nullptr, states))) return rc;
  }
  // first-order and constant rows
  if (tc1) return first_tc_chunk_state(c, p.bh, n, L, y, ext ? gs : z, ext ? dvec : nullptr, states);
  return moments_chunk_state(c, p.bh, n, L, y, z, den, delta, ext, states, 1);
}

// read-out of prefix (or total) states for n tokens; mode 0: type A, 1: type B, 2: both on x
// ready (may be null): second-order copies that exist already (prefix_states, or kept by the forward)
static int read_states(const Ctx& c, int mode, int n, int per_chunk, const void* x, const void* u,
                       const float* den, const float* delta, int ext, const void* gs, const float* dvec,
                       const float* states, void* s16, const stat_t* stats, float* out_a, float* den_a,
                       float* out_b, const StateCopies* ready = nullptr) {
  const fastmax_problem& p = c.p;
  const int L = moments_chunk(p);
  int rc;
  const bool tc2 = moments_tc_supports(p);
  const bool tc1 = first_tc_supports(p) && (p.p == 1 || tc2);
  const int mats = p.bh * (per_chunk ? (n + L - 1) / L : 1);
  if (tc2) {
    // both kinds come out complete: the first-order and constant terms ride along
    const StateCopies cp = ready ? *ready : copies_at(p, mode, s16, out_a, n, mats);
    if (!ready && (rc = moments_tc_convert(c, mats, states, at_once(cp)))) return rc;
    if (mode != 0 && (rc = moments_tc_readout_b(c, p.bh, n, L, per_chunk, x, ext ? gs : u, ext ? dvec : nullptr, cp.b,
                                                stats, states, out_b)))
      return rc;
    if (!ready && mode == 2 && cp.a == cp.b) {
      StateCopies then;
      then.a = cp.a;
      if ((rc = moments_tc_convert(c, mats, states, then))) return rc;
    }
    if (mode != 1 && (rc = moments_tc_readout_a(c, p.bh, n, L, per_chunk, x, cp.a, stats, states, out_a, den_a)))
      return rc;
    return FASTMAX_OK;
  }
  if (tc1) {
    // first-order part on tensor cores; it adds to the second-order part when there is one
    if ((rc = first_tc_convert(c, mats, states, s16))) return rc;
    if ((mode == 0 || mode == 2) && !tc2)
      if ((rc = first_tc_readout(c, 0, p.bh, n, L, per_chunk, x, x, nullptr, states, s16, stats, out_a, den_a,
                                 tc2)))
        return rc;
    if (mode == 1 || mode == 2)
      if ((rc = first_tc_readout(c, 1, p.bh, n, L, per_chunk, ext ? gs : u, x, ext ? dvec : nullptr, states,
                                 s16, stats, out_b, nullptr, tc2)))
        return rc;
    return FASTMAX_OK;
  }
  if ((mode == 0 || mode == 2) && !tc2)
    if ((rc = moments_readout(c, 0, p.bh, n, L, per_chunk, x, nullptr, nullptr, nullptr, 0, states, stats,
                              out_a, den_a, tc2)))
      return rc;
  if (mode == 1 || mode == 2)
    if ((rc = moments_readout(c, 1, p.bh, n, L, per_chunk, x, u, den, delta, ext, states, stats, out_b,
                              nullptr, tc2)))
      return rc;
  return FASTMAX_OK;
}

// p = 1 on tensor cores without a score-form part: the read-out of the total state is the
// result, so it is divided / rounded in the read-out kernel itself; s16: the bf16 copies of the totals (first_tc_total)
static bool first_is_whole(const fastmax_problem& p) { return p.p == 1 && !p.mask && first_tc_supports(p); }
static int read_first_final(const Ctx& c, int type_b, int n, const void* tile, const void* x, const float* uvec,
                            const float* total, const void* s16, const stat_t* stats, int final, void* out,
                            float* den_out, float* dots) {
  return first_tc_readout(c, type_b, c.p.bh, n, moments_chunk(c.p), 0, tile, x, uvec, total, s16, stats, nullptr,
                          nullptr, 0, final, out, den_out, dots);
}

// grad_k and grad_v from the query/gradient totals
static int read_first_dkdv(const Ctx& c, const void* k, const void* v, const float* total, const void* s16, const stat_t* stats,
                           float* dots, void* grad_k, void* grad_v) {
  int rc;
  if ((rc = read_first_final(c, 1, c.p.nk, v, k, nullptr, total, s16, stats, 2, grad_k, nullptr, dots))) return rc;
  return read_first_final(c, 0, c.p.nk, k, k, nullptr, total, s16, stats, 2, grad_v, nullptr, nullptr);
}
static int plain_layout(const fastmax_problem& p, const FwdOut& o) {
  if (!o.out_f32 && o.o_stride == p.d) return FASTMAX_OK;
  return fail(FASTMAX_E_UNSUPPORTED, "the moment family writes the plain output layout only");
}

// Exclusive running sums over the chunks of every head (per-chunk mode).  With `fuse` and the tensor-core second-order
// part, the second-order rows go straight to the bf16 copies `to` in one pass over the raw states and stay raw in
// `states` (nothing else reads them); only the first-order rows are summed in place.  *ready tells whether `to` holds
// the copies.
static int prefix_states(const Ctx& c, int nchunk, float* states, const float* base, int reverse, bool fuse,
                         const StateCopies& to, bool* ready) {
  const fastmax_problem& p = c.p;
  *ready = fuse && p.p == 2 && moments_tc_supports(p);
  if (!*ready) return moments_prefix(c, p.bh, nchunk, states, base, nullptr, reverse, 1);
  int rc;
  // first the first-order rows in place: the copies carry them too
  if ((rc = moments_prefix(c, p.bh, nchunk, states, base, nullptr, reverse, 1, p.d * p.d))) return rc;
  return moments_tc_prefix_convert(c, p.bh, nchunk, states, base, reverse, to);
}

// Copies of the context that tell the tensor-core moment kernels which chunk's state nothing will read,
// and whose tokens read an empty running sum (see Ctx).
// (the states that skipping() builds go to prefix_states with `fuse`)
static Ctx skipping(const Ctx& c, int chunk) { Ctx r = c; r.skip_chunk = chunk; r.lower_rows = true; return r; }
static Ctx zeroing(const Ctx& c, int chunk) { Ctx r = c; r.zero_chunk = chunk; return r; }

// ---- forward -----------------------------------------------------------------------
// kv_states: raw chunk states of (k, v) for this shard (already built); s_base: sum of the
// totals of all earlier shards or null.  Turns the states into prefixes in place.
int moments_forward_finish(const Ctx& c, const void* q, const void* k, const void* v,
                           const stat_t* stats, float* kv_states, const float* s_base,
                           float* o_add, float* den_add, void* s16, const FwdOut& o, bool fuse, void* keep_b) {
  const fastmax_problem& p = c.p;
  const int L = moments_chunk(p);
  const int nchunk = (p.nk + L - 1) / L;
  int rc;
  // fuse: the caller does not need the fp32 second-order prefixes (see prefix_states); the type A copies are used up
  // here, type B ones are written at keep_b when the backward will want them
  bool ready;
  StateCopies cp;
  cp.a = s16;
  cp.b = keep_b;
  if ((rc = prefix_states(c, nchunk, kv_states, s_base, 0, fuse, cp, &ready))) return rc;
  if (first_fused(p) && !o.out_f32) {
    if ((rc = first_tc_convert(c, p.bh * nchunk, kv_states, s16, nchunk, stats))) return rc;
    ChunkAdd own;
    own.chunk = L;
    const FirstState fs = {kv_states, s16, s_base ? -1 : 0};
    return dense_tc_short_forward(c, q, k, v, stats, o.out, o.den, &own, &fs);
  }
  // without a base the tokens of the first chunk have nothing before them
  if ((rc = read_states(zeroing(c, s_base ? -1 : 0), 0, p.nq, 1, q, nullptr, nullptr, nullptr, 0, nullptr, nullptr,
                        kv_states, s16, stats, o_add, den_add, nullptr, ready ? &cp : nullptr)))
    return rc;
  ChunkAdd ca;
  ca.chunk = L;
  ca.out_add = o_add;
  ca.den_add = den_add;
  if (dense_tc_supports(p) && !o.out_f32) return dense_tc_forward(c, q, k, v, stats, o.out, o.den, &ca);
  if (c.split_ws) return dense_split_forward(c, q, k, v, stats, o, c.split_ws, &ca);
  return dense_ffma_forward(c, q, k, v, stats, o, ca);
}

// total_keep (may be null): where the forward leaves what the backward would otherwise rebuild from k and v --
// unmasked: the total key/value state; causal: the chunk states of the keys and values (first-order rows as
// exclusive prefixes; with the tensor-core second-order part those rows stay raw and their prefixes follow
// as bf16 transposed copies, moment_kept16_bytes)
int moments_forward(const Ctx& c, const void* q, const void* k, const void* v, const stat_t* stats,
                    const FwdOut& o, void* workspace, float* total_keep) {
  const fastmax_problem& p = c.p;
  const int L = moments_chunk(p);
  const MomFwdWs w = moments_fwd_layout(p);
  char* ws = (char*)workspace;
  float* states = (p.mask && total_keep) ? total_keep : (float*)(ws + w.states);
  float* total = (!p.mask && total_keep) ? total_keep : (float*)(ws + w.total);
  float* o_add = (float*)(ws + w.o_add);
  float* den_add = (float*)(ws + w.den_add);
  int rc;
  void* s16 = ws + w.s16;
  // causal: nothing comes after the last chunk, so its state is not built
  const int last = (p.nk + L - 1) / L - 1;
  if ((rc = moments_build_states(p.mask ? skipping(c, last) : c, p.nk, k, v, nullptr, nullptr, 0, nullptr, nullptr,
                                 states)))
    return rc;
  if (p.mask) {
    // second-order prefixes go straight to their bf16 copies; those for the backward lie behind the kept fp32 states
    void* keep_b = total_keep ? (void*)((char*)total_keep + moment_state_bytes(p, p.nk)) : nullptr;
    return moments_forward_finish(c, q, k, v, stats, states, nullptr, o_add, den_add, s16, o, true, keep_b);
  }
  // unmasked: every query reads the total of all keys
  const int nchunk = (p.nk + L - 1) / L;
  if (first_is_whole(p)) {
    if ((rc = plain_layout(p, o)) || (rc = first_tc_total(c, nchunk, states, total, s16))) return rc;
    return read_first_final(c, 0, p.nq, q, q, nullptr, total, s16, stats, 1, o.out, o.den, nullptr);
  }
  if ((rc = moments_prefix(c, p.bh, nchunk, states, nullptr, total, 0, 0))) return rc;
  return moments_forward_total(c, q, stats, total, o_add, den_add, s16, o);
}

// What moments_forward leaves at total_keep, for a forward of another family.  The tensor-core state kernels read k and
// v by TMA, so unaligned tensors take the CUDA-core ones.  Unmasked, the chunk states need a workspace; without one
// the total is summed as a single chunk, in less parallel but next to a forward that is quadratic in the length.
int moments_leave_states(const Ctx& c, const void* k, const void* v, bool aligned, void* workspace,
                         size_t workspace_bytes, float* total_keep) {
  const fastmax_problem& p = c.p;
  const int L = moments_chunk(p), nchunk = (p.nk + L - 1) / L;
  const size_t need = moment_state_bytes(p, p.nk);
  const bool room = workspace && workspace_bytes >= need && ((uintptr_t)workspace & 15) == 0;
  if (!p.mask && !room) return moments_chunk_state(c, p.bh, p.nk, p.nk, k, v, nullptr, nullptr, 0, total_keep);
  float* states = p.mask ? total_keep : (float*)workspace;
  int rc;
  if (aligned)
    rc = moments_build_states(p.mask ? skipping(c, nchunk - 1) : c, p.nk, k, v, nullptr, nullptr, 0, nullptr, nullptr, states);
  else
    rc = moments_chunk_state(c, p.bh, p.nk, L, k, v, nullptr, nullptr, 0, states);
  if (rc) return rc;
  if (!p.mask) return moments_prefix(c, p.bh, nchunk, states, nullptr, total_keep, 0, 0);
  bool ready;
  StateCopies cp;
  cp.b = (char*)total_keep + need;
  return prefix_states(c, nchunk, states, nullptr, 0, true, cp, &ready);
}

// Unmasked forward from a given total state (this device's keys, or the sum over all shards).
int moments_forward_total(const Ctx& c, const void* q, const stat_t* stats, const float* total, float* o_add,
                          float* den_add, void* s16, const FwdOut& o) {
  const fastmax_problem& p = c.p;
  int rc;
  if ((rc = plain_layout(p, o))) return rc;
  if (first_is_whole(p)) {
    if ((rc = first_tc_total(c, 1, total, nullptr, s16))) return rc;
    return read_first_final(c, 0, p.nq, q, q, nullptr, total, s16, stats, 1, o.out, o.den, nullptr);
  }
  if ((rc = read_states(c, 0, p.nq, 0, q, nullptr, nullptr, nullptr, 0, nullptr, nullptr, total, s16, stats,
                        o_add, den_add, nullptr)))
    return rc;
  return moments_finalize(c, p.bh, p.nq, o_add, den_add, nullptr, o.out, o.den, nullptr, 0);
}

// ---- backward ----------------------------------------------------------------------
// What grad_k and grad_v take from the tokens after a chunk: the states of (q, gradient) become suffix sums (r_base: those
// of later shards, or null) and are read out in both kinds.  zero_chunk has nothing after it.  Nothing reads r_states after
// this, so their second-order rows may stay raw (prefix_states).
static int read_suffix_sums(const Ctx& c, int nchunk, float* r_states, const float* r_base, int zero_chunk, const void* k,
                            const void* v, const stat_t* stats, void* s16, float* gk_add, float* gv_add) {
  const fastmax_problem& p = c.p;
  const StateCopies cp = copies_at(p, 2, s16, gv_add, p.nk, p.bh * nchunk);
  const Ctx z = zeroing(c, zero_chunk);
  auto read = [&](int mode, const StateCopies* ready) {
    return read_states(z, mode, p.nk, 1, k, v, nullptr, nullptr, 0, nullptr, nullptr, r_states, s16, stats, gv_add, nullptr,
                       gk_add, ready);
  };
  bool ready;
  int rc = prefix_states(c, nchunk, r_states, r_base, 1, true, at_once(cp), &ready);
  if (rc) return rc;
  if (!ready) return read(2, nullptr);
  if (cp.a != cp.b) return read(2, &cp);
  StateCopies then;
  then.a = cp.a;
  if ((rc = read(1, &cp)) || (rc = moments_tc_prefix_convert(c, p.bh, nchunk, r_states, r_base, 1, then))) return rc;
  return read(0, &cp);
}

// The part of grad_q that reads the key/value prefixes (everything before a token's own chunk).  It
// depends on nothing from later shards, so a sequence shard issues it while the query/gradient
// totals are being exchanged.
int moments_backward_dq_far(const Ctx& c, const void* q, const float* den, const stat_t* stats,
                            const void* grad_out, const float* delta, const float* dvec, const void* gs,
                            const float* s_states, float* gq_add, void* s16) {
  return read_states(c, 1, c.p.nq, 1, q, grad_out, den, delta, 1, gs, dvec, s_states, s16, stats, nullptr,
                     nullptr, gq_add);
}

// s_states: exclusive prefixes of the (k, v) chunk states (as left by the forward finish);
// r_states: raw chunk states of (q, grad_out/den | -delta/den); r_base: sum of the totals of
// all later shards or null.  Writes the three gradients without the normalisation row fix.
int moments_backward_finish(const Ctx& c, const void* q, const void* k, const void* v,
                            const float* den, const stat_t* stats, const void* grad_out,
                            const float* delta, const float* dvec, const void* gs,
                            const float* s_states, float* r_states, const float* r_base,
                            float* gq_add, float* gk_add, float* gv_add, void* s16, float* dots,
                            void* grad_q, void* grad_k, void* grad_v, bool dq_far_done) {
  const fastmax_problem& p = c.p;
  const int L = moments_chunk(p);
  const int nchunk = (p.nq + L - 1) / L;
  int rc;
  // grad_q reads the key/value prefixes with u = [grad_out/den | -delta/den]
  if (!dq_far_done &&
      (rc = moments_backward_dq_far(c, q, den, stats, grad_out, delta, dvec, gs, s_states, gq_add, s16)))
    return rc;
  // grad_k and grad_v read the suffix sums of the query/gradient states
  if ((rc = read_suffix_sums(c, nchunk, r_states, r_base, r_base ? -1 : nchunk - 1, k, v, stats, s16, gk_add, gv_add)))
    return rc;
  ChunkAdd ca;
  ca.chunk = L;
  ca.gq_add = gq_add;
  ca.gk_add = gk_add;
  ca.gv_add = gv_add;
  if (dense_tc_supports(p))
    return dense_tc_backward(c, q, k, v, gs, dvec, stats, dots, grad_q, grad_k, grad_v, &ca);
  return dense_ffma_backward(c, q, k, v, den, stats, grad_out, delta, dots, grad_q, grad_k, grad_v, ca);
}

// kv_total_kept (may be null): what the forward left behind (unmasked: the total key/value state; causal: the
// exclusive prefixes of the key/value chunk states); without it the states are rebuilt from k and v
int moments_backward(const Ctx& c, const void* q, const void* k, const void* v, const void* out,
                     const float* den, const stat_t* stats, const void* grad_out, void* grad_q,
                     void* grad_k, void* grad_v, void* workspace, const float* kv_total_kept) {
  const fastmax_problem& p = c.p;
  const int L = moments_chunk(p);
  const MomBwdWs w = moments_bwd_layout(p);
  char* ws = (char*)workspace;
  float* dots = (float*)(ws + w.dots);
  float* delta = (float*)(ws + w.delta);
  float* dvec = (float*)(ws + w.dvec);
  void* gs = ws + w.gs;
  float* states = (float*)(ws + w.states);
  float* total = (float*)(ws + w.total);
  float* gq_add = (float*)(ws + w.gq_add);
  float* gk_add = (float*)(ws + w.gk_add);
  float* gv_add = (float*)(ws + w.gv_add);
  void* s16 = ws + w.s16;
  int rc;
  if (p.normalize)
    FM_CUDA_TRY(cudaMemsetAsync(dots, 0, sizeof(float) * (size_t)(p.bh + p.bhkv), c.stream));
  const bool tc = dense_tc_supports(p);
  // the plain row dots feed the CUDA-core kernels only; when every stage runs on tensor cores they
  // all read gs / dvec and the pass over grad_out and out is skipped
  const bool all_tc = moments_all_tc(p);
  if (!all_tc && (rc = launch_delta(c, grad_out, out, delta))) return rc;
  // unmasked p = 1: no score kernel reads gs, and the kernel of grad_q forms it itself
  const bool whole = first_is_whole(p) && p.nq > 0;
  if (tc && !whole && (rc = launch_gprep(c, grad_out, out, den, gs, dvec))) return rc;
  const int nck = (p.nk + L - 1) / L, ncq = (p.nq + L - 1) / L;
  if (p.mask) {
    // the key/value prefixes are rebuilt (the forward does not keep them), used for grad_q,
    // then the buffer is reused for the query/gradient states
    bool ready = false;
    StateCopies kv;               // second-order bf16 copies of the key/value prefixes, where they exist already
    if (!kv_total_kept) {
      if ((rc = moments_build_states(skipping(c, nck - 1), p.nk, k, v, nullptr, nullptr, 0, nullptr, nullptr, states)))
        return rc;
      kv.b = s16;
      if ((rc = prefix_states(c, nck, states, nullptr, 0, true, kv, &ready))) return rc;
    } else if (moment_kept16_bytes(p) > 0) {
      kv.b = (char*)const_cast<float*>(kv_total_kept) + moment_state_bytes(p, p.nk);
      ready = true;
    }
    if (first_fused(p)) {
      const float* sums = kv_total_kept ? kv_total_kept : states;
      ChunkAdd own;
      own.chunk = L;
      if ((rc = first_tc_convert(c, p.bh * nck, sums, s16, nck, stats))) return rc;
      const FirstState before = {sums, s16, 0};
      if ((rc = dense_tc_short_dq(c, q, k, v, gs, dvec, stats, dots, grad_q, &own, &before))) return rc;
      if ((rc = moments_build_states(skipping(c, 0), p.nq, q, grad_out, den, delta, 1, gs, dvec, states))) return rc;
      if ((rc = prefix_states(c, ncq, states, nullptr, 1, true, kv, &ready))) return rc;
      if ((rc = first_tc_convert(c, p.bh * ncq, states, s16, ncq, stats))) return rc;
      const FirstState after = {states, s16, ncq - 1};
      if ((rc = dense_tc_first_dkdv(c, q, k, v, gs, dvec, stats, dots, grad_k, grad_v, own, after))) return rc;
      return p.normalize ? launch_norm_fixup(c, q, k, stats, dots, grad_q, grad_k) : FASTMAX_OK;
    }
    // grad_q: the first chunk's tokens have no keys before their chunk; grad_k, grad_v: the last chunk's
    // tokens no queries after theirs, and nothing reads the query/gradient state of the first chunk
    if ((rc = read_states(zeroing(c, 0), 1, p.nq, 1, q, grad_out, den, delta, 1, gs, dvec,
                          kv_total_kept ? kv_total_kept : states, s16, stats, nullptr, nullptr, gq_add,
                          ready ? &kv : nullptr)))
      return rc;
    if ((rc = moments_build_states(skipping(c, 0), p.nq, q, grad_out, den, delta, 1, gs, dvec, states))) return rc;
    if ((rc = read_suffix_sums(c, ncq, states, nullptr, ncq - 1, k, v, stats, s16, gk_add, gv_add))) return rc;
    ChunkAdd ca;
    ca.chunk = L;
    ca.gq_add = gq_add;
    ca.gk_add = gk_add;
    ca.gv_add = gv_add;
    if (tc) rc = dense_tc_backward(c, q, k, v, gs, dvec, stats, dots, grad_q, grad_k, grad_v, &ca);
    else if (c.split_ws)
      rc = dense_split_backward(c, q, k, v, out, den, stats, grad_out, dots, grad_q, grad_k, grad_v, c.split_ws, &ca);
    else rc = dense_ffma_backward(c, q, k, v, den, stats, grad_out, delta, dots, grad_q, grad_k, grad_v, ca);
    if (rc) return rc;
  } else {
    // unmasked: totals only, no score-form part.  The two totals share one buffer, so grad_q is
    // read out before the query/gradient total replaces the key/value total.
    if (!kv_total_kept) {
      if ((rc = moments_build_states(c, p.nk, k, v, nullptr, nullptr, 0, nullptr, nullptr, states))) return rc;
      if ((rc = moments_prefix(c, p.bh, nck, states, nullptr, total, 0, 0))) return rc;
    }
    if (whole) {
      // one kernel reads the query side; the room for gs and the states behind it take those it leaves, s16 the copies of
      // either total
      const float* kv = kv_total_kept ? kv_total_kept : total;
      int nruns;
      if ((rc = first_tc_total(c, 1, kv, nullptr, s16))) return rc;
      if ((rc = first_tc_grad(c, q, out, den, grad_out, kv, s16, stats, grad_q, p.normalize ? dots : nullptr, (float*)gs, &nruns)))
        return rc;
      if ((rc = first_tc_total(c, nruns, (const float*)gs, total, s16))) return rc;
      if ((rc = read_first_dkdv(c, k, v, total, s16, stats, p.normalize ? dots + p.bh : nullptr, grad_k, grad_v))) return rc;
      return p.normalize ? launch_norm_fixup(c, q, k, stats, dots, grad_q, grad_k) : FASTMAX_OK;
    }
    if ((rc = moments_backward_total(c, q, k, v, den, stats, grad_out, delta, dvec, gs,
                                     kv_total_kept ? kv_total_kept : total, nullptr, gq_add,
                                     gk_add, gv_add, s16, dots, grad_q, nullptr, nullptr)))
      return rc;
    if ((rc = moments_build_states(c, p.nq, q, grad_out, den, delta, 1, gs, dvec, states))) return rc;
    if ((rc = moments_prefix(c, p.bh, ncq, states, nullptr, total, 0, 0))) return rc;
    if ((rc = moments_backward_total(c, q, k, v, den, stats, grad_out, delta, dvec, gs, nullptr, total, gq_add,
                                     gk_add, gv_add, s16, dots, nullptr, grad_k, grad_v)))
      return rc;
  }
  if (p.normalize) return launch_norm_fixup(c, q, k, stats, dots, grad_q, grad_k);
  return FASTMAX_OK;
}

// Unmasked gradients from given total states (this device's, or the sums over all shards): grad_q
// from the key/value total when kv_total and grad_q are given, grad_k and grad_v from the
// query/gradient total when qg_total and grad_k are given.  Without the normalisation row fix.
int moments_backward_total(const Ctx& c, const void* q, const void* k, const void* v, const float* den,
                           const stat_t* stats, const void* grad_out, const float* delta, const float* dvec,
                           const void* gs, const float* kv_total, const float* qg_total, float* gq_add,
                           float* gk_add, float* gv_add, void* s16, float* dots, void* grad_q, void* grad_k,
                           void* grad_v) {
  const fastmax_problem& p = c.p;
  int rc;
  if (kv_total && grad_q) {
    if (first_is_whole(p)) {
      if ((rc = first_tc_total(c, 1, kv_total, nullptr, s16))) return rc;
      if ((rc = read_first_final(c, 1, p.nq, gs, q, dvec, kv_total, s16, stats, 2, grad_q, nullptr,
                                 p.normalize ? dots : nullptr)))
        return rc;
    } else {
      if ((rc = read_states(c, 1, p.nq, 0, q, grad_out, den, delta, 1, gs, dvec, kv_total, s16, stats, nullptr,
                            nullptr, gq_add)))
        return rc;
      if ((rc = moments_finalize(c, p.bh, p.nq, gq_add, nullptr, q, grad_q, nullptr,
                                 p.normalize ? dots : nullptr, 1)))
        return rc;
    }
  }
  if (qg_total && grad_k) {
    if (first_is_whole(p)) {
      if ((rc = first_tc_total(c, 1, qg_total, nullptr, s16))) return rc;
      if ((rc = read_first_dkdv(c, k, v, qg_total, s16, stats, p.normalize ? dots + p.bh : nullptr, grad_k, grad_v))) return rc;
    } else {
      if ((rc = read_states(c, 2, p.nk, 0, k, v, nullptr, nullptr, 0, nullptr, nullptr, qg_total, s16, stats,
                            gv_add, nullptr, gk_add)))
        return rc;
      if ((rc = moments_finalize(c, p.bh, p.nk, gk_add, nullptr, k, grad_k, nullptr,
                                 p.normalize ? dots + p.bh : nullptr, 1)))
        return rc;
      if ((rc = moments_finalize(c, p.bh, p.nk, gv_add, nullptr, nullptr, grad_v, nullptr, nullptr, 1)))
        return rc;
    }
  }
  return FASTMAX_OK;
}

}  // namespace fm
