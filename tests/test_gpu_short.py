"""GPU parity of the short-row score kernels (bf16, d = 64, two row tiles per SM) against the CPU oracle: enough heads
that the dispatch picks them (checked by kernel name in a test of its own, since launches of the short and the wide
kernels carry the same labels), row and column tile edges, grouped heads, more keys than queries, both orders, and the
chunks of the moment family.  Tolerance: the bf16 one of the other tests (2e-2 of the largest value)."""
import pytest
import torch

from gpu_util import assert_close, oracle, run_cabi

from fastmax_b200 import _cabi

pytestmark = pytest.mark.gpu


def randn(*shape, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=g)


# bh, nq, nk, mask, p, normalize; bh * row tiles > 148
CASES = [(150, 1, 1, 1, 2, 1), (150, 63, 63, 1, 2, 1), (150, 65, 65, 0, 2, 1), (150, 128, 128, 1, 1, 1),
         (75, 129, 129, 1, 2, 0), (75, 191, 193, 1, 2, 1), (75, 130, 450, 0, 2, 1), (50, 300, 300, 1, 2, 1)]


@pytest.mark.parametrize("cfg", CASES, ids=[f"bh{c[0]}nq{c[1]}nk{c[2]}m{c[3]}p{c[4]}z{c[5]}" for c in CASES])
def test_short_rows_against_dense_oracle(cfg):
    bh, nq, nk, mask, p, norm = cfg
    q, go = randn(1, bh, nq, 64, seed=nq), randn(1, bh, nq, 64, seed=nq + 1)
    k, v = randn(1, bh, nk, 64, seed=nk + 2), randn(1, bh, nk, 64, seed=nk + 3)
    if not norm:
        q, k = q / 8, k / 8
    kw = dict(mask=mask, normalize=norm, p=p, a0=1.0, a1=1.0, a2=0.5, lim=1.0)
    got, _ = run_cabi(q, k, v, go, torch.bfloat16, impl="dense_tc", **kw)
    assert _cabi.device_status() == 0
    ref = oracle(q, k, v, go, torch.bfloat16, dense=True, **kw)
    assert_close(got, ref, torch.bfloat16, str(cfg), floor=1.0 if nk == 1 else 1e-2)


def kernel_names(call):
    """Functions of the kernels that ``call`` launches, from the CUDA activity trace."""
    call()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return [e.key for e in prof.key_averages()]


def test_sizes_of_these_tests_reach_the_short_kernels():
    kw = dict(mask=True, normalize=True, p=2)

    def step(heads, kv, n, **more):
        q, go = [torch.randn(heads, n, 64, device="cuda").bfloat16() for _ in range(2)]
        k, v = [torch.randn(kv, n, 64, device="cuda").bfloat16() for _ in range(2)]

        def call():
            out, den, st = _cabi.forward(q, k, v, **{**kw, **more})
            _cabi.backward(q, k, v, out, den, st, go, **{**kw, **more})
        return kernel_names(call)

    seen = {"score": step(150, 150, 65, impl="dense_tc"), "two row tiles": step(75, 75, 129, impl="dense_tc"),
            "grouped": step(180, 60, 150, impl="dense_tc"), "chunks": step(40, 40, 520, impl="moments", chunk=256),
            "first order": step(40, 40, 700, impl="moments", chunk=256, p=1)}
    if not any(seen.values()):
        pytest.skip("no CUDA activity trace on this machine")
    for what, names in seen.items():
        short = [n_ for n_ in names if "short_kernel<" in n_]
        # grouped: the 120 row tiles of 60 key/value heads are fewer than the SMs, so that pass stays on the wide kernel
        assert len(short) == (2 if what == "grouped" else 3), (what, names)
        assert any("dense_tc_wide_kernel" in n_ for n_ in names) == (what == "grouped"), (what, names)


@pytest.mark.parametrize("p,chunk,n", [(1, 256, 700), (1, 512, 1537), (2, 256, 520), (1, 0, 1100)])
def test_chunks_of_the_moment_family(p, chunk, n):
    bh = 40
    q, k, v, go = [randn(1, bh, n, 64, seed=s + n) for s in range(4)]
    kw = dict(mask=1, normalize=1, p=p, a0=0.8, a1=1.2, a2=0.4, lim=1.1)
    got, _ = run_cabi(q, k, v, go, torch.bfloat16, impl="moments", **{**kw, **({"chunk": chunk} if chunk else {})})
    assert _cabi.device_status() == 0
    ref = oracle(q, k, v, go, torch.bfloat16, dense=True, **kw)
    assert_close(got, ref, torch.bfloat16, f"p={p} chunk={chunk} n={n}")


@pytest.mark.parametrize("mask", [0, 1])
def test_grouped_heads_against_expanded_heads(mask):
    g = torch.Generator(device="cuda").manual_seed(3)
    kv, r, n = 60, 3, 150
    mk = lambda h: torch.randn(h, n, 64, generator=g, device="cuda").bfloat16()  # noqa: E731
    q, k, v, go = mk(kv * r), mk(kv), mk(kv), mk(kv * r)
    kw = dict(mask=bool(mask), normalize=True, p=2)
    res = {}
    for impl in ("dense_tc", "dense_ffma"):
        out, den, st = _cabi.forward(q, k, v, impl=impl, **kw)
        res[impl] = (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, impl=impl, **kw))
    assert _cabi.device_status() == 0
    for a, b, name in zip(res["dense_tc"], res["dense_ffma"], ("out", "dq", "dk", "dv")):
        assert float((a.float() - b.float()).abs().max() / b.float().abs().max()) < 2e-2, name


def test_first_order_shards_read_the_base_of_earlier_shards():
    """Two sequence shards one after the other: the second one's chunks start from the first one's total."""
    from fastmax_b200.sharded import CudaShardBackend
    g = torch.Generator(device="cuda").manual_seed(5)
    bh, nl = 3, 640
    q, k, v = [torch.randn(bh, 2 * nl, 64, generator=g, device="cuda").bfloat16() for _ in range(3)]
    want, wden, _ = _cabi.forward(q, k, v, mask=True, normalize=True, p=1, impl="dense_ffma")
    be = CudaShardBackend(normalize=True, a0=1.0, a1=1.0, a2=0.5, lim=1.0, p=1, chunk=256)
    sh = lambda t, r: t[:, r * nl:(r + 1) * nl].contiguous()  # noqa: E731
    st = torch.stack([be.rowmax(sh(q, r), sh(k, r), r * nl) for r in range(2)]).max(0).values
    kv = [be.kv_state(sh(k, r), sh(v, r)) for r in range(2)]
    outs = [be.forward(sh(q, r), sh(k, r), sh(v, r), st, kv[r][0], kv[0][1] if r else None) for r in range(2)]
    assert _cabi.device_status() == 0
    out, den = torch.cat([o for o, _ in outs], 1), torch.cat([d for _, d in outs], 1)
    assert float((out.float() - want.float()).abs().max() / want.float().abs().max()) < 2e-2
    assert float((den - wden).abs().max() / wden.abs().max()) < 1e-2


def test_first_order_chunks_refuse_unaligned_results():
    """Forced onto the moment family (AUTO takes such tensors elsewhere), and as a sequence shard: an argument error before
    the kernel that would write the rows, forward and backward."""
    bh, n = 3, 600
    size = bh * n * 64
    q, k, v, go = [torch.randn(bh, n, 64, device="cuda").bfloat16() for _ in range(4)]
    odd = lambda: torch.empty(size + 1, dtype=torch.bfloat16, device="cuda")[1:].view(bh, n, 64)  # noqa: E731
    kw = dict(mask=True, normalize=True, p=1, impl="moments", chunk=256)
    fwd, bwd, stats = _cabi.workspace_bytes(q, k, **kw)
    scratch = lambda m: torch.empty(m, dtype=torch.uint8, device="cuda")  # noqa: E731
    with pytest.raises(ValueError, match="16-byte aligned"):
        _cabi.forward(q, k, v, buffers=dict(out=odd(), den=torch.empty(bh, n, device="cuda"), stats=scratch(stats),
                                            workspace=scratch(fwd)), **kw)
    out, den, st = _cabi.forward(q, k, v, **kw)
    want = _cabi.backward(q, k, v, out, den, st, go, **kw)
    for name in ("grad_q", "grad_k", "grad_v"):
        grads = {g: torch.empty_like(q) for g in ("grad_q", "grad_k", "grad_v")}
        with pytest.raises(ValueError, match="16-byte aligned"):
            _cabi.backward(q, k, v, out, den, st, go, buffers={**grads, name: odd(), "workspace": scratch(bwd)}, **kw)
    got = _cabi.backward(q, k, v, out, den, st, go, **kw)
    assert all(torch.equal(a, b) for a, b in zip(got[2:], want[2:]))     # no atomics behind grad_v
    L = _cabi.lib()
    prob = _cabi.make_problem(q, k, True, False, 1.0, 1.0, 1.0, 0.5, 1.0, 1, "auto", 256)
    states = torch.empty(L.fastmax_b200_moment_state_bytes(prob), dtype=torch.uint8, device="cuda")
    total = torch.empty(L.fastmax_b200_moment_total_bytes(prob), dtype=torch.uint8, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    assert L.fastmax_b200_shard_kv_state(prob, k.data_ptr(), v.data_ptr(), states.data_ptr(), total.data_ptr(), stream) == 0
    ws = scratch(L.fastmax_b200_shard_forward_workspace_bytes(prob))
    rc = L.fastmax_b200_shard_forward(prob, q.data_ptr(), k.data_ptr(), v.data_ptr(), None, states.data_ptr(), None,
                                      odd().data_ptr(), den.data_ptr(), ws.data_ptr(), ws.numel(), stream)
    assert rc == -1 and b"16-byte aligned" in L.fastmax_b200_last_error()
    torch.cuda.synchronize()
    assert _cabi.device_status() == 0


@pytest.mark.parametrize("d,heads,n", [(64, 96, 1700), (128, 16, 4300)])
@pytest.mark.parametrize("back_aligned", [False, True], ids=["unaligned backward", "aligned backward"])
def test_unaligned_tensors_at_lengths_of_the_moment_family(d, heads, n, back_aligned):
    """AUTO serves causal first-order tensors that TMA cannot read on the CUDA cores; a backward on aligned copies runs on the
    moment family and finds the states it expects behind the statistics (filled with NaN before)."""
    g = torch.Generator(device="cuda").manual_seed(d)
    size = heads * n * d
    flat = [torch.randn(size + 1, generator=g, device="cuda").bfloat16() for _ in range(4)]
    q, k, v, go = [t[1:].view(heads, n, d) for t in flat]
    assert q.data_ptr() % 16
    kw = dict(mask=True, normalize=True, p=1)
    assert _cabi.selected_impl(_cabi.make_problem(q, k, True, True, 1.0, 1.0, 1.0, 0.5, 1.0, 1)) == "moments"
    aligned = [t.clone() for t in (q, k, v, go)]
    out, den, st = _cabi.forward(*aligned[:3], **kw)
    want = (out,) + tuple(_cabi.backward(*aligned[:3], out, den, st, aligned[3], **kw))
    fwd, _, stats = _cabi.workspace_bytes(q, k, **kw)
    bufs = dict(out=torch.empty_like(aligned[0]), den=torch.empty_like(den),
                stats=torch.full((stats,), 255, dtype=torch.uint8, device="cuda"),
                workspace=torch.empty(fwd, dtype=torch.uint8, device="cuda"))
    _cabi.profile(True)
    out, den, st = _cabi.forward(q, k, v, buffers=bufs, **kw)
    t = aligned if back_aligned else (q, k, v, go)
    got = (out,) + tuple(_cabi.backward(*t[:3], out, den, st, t[3], **kw))
    names = {n_ for n_, _ in _cabi.profile_records()}
    _cabi.profile(False)
    assert "fm_dense_ffma_fwd" in names and ("fm_dense_ffma_dq" in names) != back_aligned, names
    for a, b, name in zip(got, want, ("out", "dq", "dk", "dv")):
        assert float((a.float() - b.float()).abs().max() / b.float().abs().max()) < 2e-2, name
