"""GPU parity of the float32 score kernels on the tensor cores (operands as three bf16 parts) against the CPU
oracle: tile edges (128 rows, 64 columns), grouped heads, more keys than queries, both polynomial orders.

Bound: every product is exact to 2^-26 of itself, sums of 64 columns are accumulated by the tensor core and added
in float32, so a result is as exact as the CUDA-core family's, 1e-5 relative for these lengths; the tests ask for
2e-5 (max |x - ref| / max |ref|) where the other float32 tests ask for 1e-4."""
import pytest
import torch

from gpu_util import oracle, run_cabi

from fastmax_b200 import _cabi

pytestmark = pytest.mark.gpu
BOUND = 2e-5

# bh, nq, nk, d, mask, p, normalize
CASES = [(1, 1, 1, 32, 1, 2, 0), (2, 2, 2, 64, 1, 2, 1), (3, 63, 63, 32, 1, 2, 1), (2, 64, 64, 64, 0, 2, 1),
         (2, 65, 65, 32, 0, 1, 0), (2, 127, 127, 64, 1, 1, 1), (3, 128, 128, 32, 1, 2, 1), (2, 129, 129, 64, 1, 2, 0),
         (2, 257, 257, 32, 0, 2, 1), (2, 70, 300, 32, 1, 2, 1), (2, 200, 457, 64, 0, 2, 1), (5, 1000, 1000, 32, 1, 2, 1),
         (1, 1500, 1500, 64, 0, 2, 0)]


def randn(*shape, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.randn(*shape, generator=g)


@pytest.mark.parametrize("cfg", CASES, ids=[f"bh{c[0]}nq{c[1]}nk{c[2]}d{c[3]}m{c[4]}p{c[5]}z{c[6]}" for c in CASES])
def test_split_kernels_against_dense_oracle(cfg):
    bh, nq, nk, d, mask, p, norm = cfg
    q, go = randn(1, bh, nq, d, seed=nq), randn(1, bh, nq, d, seed=nq + 1)
    k, v = randn(1, bh, nk, d, seed=nk + 2), randn(1, bh, nk, d, seed=nk + 3)
    if not norm:
        q, k = q * d ** -0.5, k * d ** -0.5
    kw = dict(mask=mask, normalize=norm, p=p, a0=1.0, a1=1.0, a2=0.5, lim=1.0)
    _cabi.profile(True)
    got, _ = run_cabi(q, k, v, go, torch.float32, **kw)
    names = {n for n, _ in _cabi.profile_records()}
    _cabi.profile(False)
    assert {"fm_dense_split_fwd", "fm_dense_split_dq", "fm_dense_split_dkdv"} <= names, names
    assert _cabi.device_status() == 0
    ref = oracle(q, k, v, go, torch.float32, dense=True, **kw)
    for x, r, name in zip(got, ref, ("out", "dq", "dk", "dv")):
        # at one key the gradients of q and k are zeros made of terms of size one
        err = float((x.double() - r).abs().max() / r.abs().max().clamp_min(1.0 if nk == 1 else 1e-2))
        assert err < BOUND, (name, err)


@pytest.mark.parametrize("d,ratio,n", [(32, 4, 190), (64, 2, 321)])
def test_grouped_heads_match_expanded_heads(d, ratio, n):
    g = torch.Generator(device="cuda").manual_seed(n)
    mk = lambda h: torch.randn(h, n, d, generator=g, device="cuda")  # noqa: E731
    q, k, v, go = mk(2 * ratio), mk(2), mk(2), mk(2 * ratio)
    kw = dict(mask=True, normalize=True, p=2)
    out, den, st = _cabi.forward(q, k, v, **kw)
    got = (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, **kw))
    out, den, st = _cabi.forward(q, k, v, impl="dense_ffma", **kw)
    want = (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, impl="dense_ffma", **kw))
    for x, r, name in zip(got, want, ("out", "dq", "dk", "dv")):
        assert float((x - r).abs().max() / r.abs().max()) < BOUND, name


def test_less_workspace_or_unaligned_tensors_run_on_the_cuda_cores():
    """A call that the split kernels cannot serve is served as before: no forward workspace, and 4-byte alignment."""
    n, d = 150, 32
    kw = dict(mask=True, normalize=True, p=2)
    flat = [torch.randn(2 * n * d + 1, device="cuda") for _ in range(3)]
    q, k, v = [t[1:].view(2, n, d) for t in flat]
    assert q.data_ptr() % 16 and q.is_contiguous()
    out, _, _ = _cabi.forward(q, k, v, **kw)
    want, _, _ = _cabi.forward(q, k, v, impl="dense_ffma", **kw)
    assert torch.equal(out, want)
    q, k, v = [t.clone() for t in (q, k, v)]
    prob = _cabi.make_problem(q, k, True, True, 1.0, 1.0, 1.0, 0.5, 1.0, 2)
    out, den = torch.empty_like(q), torch.empty(2, n, device="cuda")
    stats = torch.empty(64, dtype=torch.uint8, device="cuda")
    rc = _cabi.lib().fastmax_b200_forward(prob, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), den.data_ptr(),
                                          stats.data_ptr(), None, 0, torch.cuda.current_stream().cuda_stream)
    assert rc == 0 and torch.equal(out, want)


@pytest.mark.parametrize("p", [1, 2])
def test_no_room_for_the_operand_parts(p):
    """Where the device has no room for the operand parts, a call runs on the CUDA cores in the least workspace."""
    bh, n, d = 512, 4096, 32
    q, k, v, go = [torch.randn(bh, n, d, device="cuda") for _ in range(4)]
    kw = dict(mask=True, normalize=True, p=p)
    tensor = q.numel() * 4
    total = torch.cuda.get_device_properties(0).total_memory

    def run(room_fwd=None, room_bwd=None):
        def leave(room):
            torch.cuda.empty_cache()
            if room is not None:
                torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room * tensor) / total)
        _cabi.profile(True)
        try:
            leave(room_fwd)
            out, den, st = _cabi.forward(q, k, v, **kw)
            leave(room_bwd)
            got = (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, **kw))
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        names = {n_ for n_, _ in _cabi.profile_records()}
        _cabi.profile(False)
        return got, names

    want, names = run()
    assert any("split" in n_ for n_ in names), names
    # forward: the result, and either 4.5 tensors of parts or none (first order: one of fp32 rows); backward: three
    # gradients, and 6 tensors of parts or none (first order: three of fp32 rows)
    got, names = run(3, 7.5)
    assert not any("split" in n_ for n_ in names), names
    for x, r, name in zip(got, want, ("out", "dq", "dk", "dv")):
        assert float((x - r).abs().max() / r.abs().max()) < BOUND, name


@pytest.mark.parametrize("bh,n,d,mask,chunk", [(40, 700, 32, 1, 0), (200, 900, 32, 1, 0), (420, 640, 32, 1, 0), (500, 641, 32, 1, 0),
                                               (75, 513, 32, 0, 0), (160, 1000, 64, 1, 0), (330, 520, 64, 1, 0), (60, 650, 64, 0, 0),
                                               (150, 1100, 32, 1, 256), (600, 600, 32, 1, 256), (40, 900, 64, 1, 256), (16, 1281, 64, 1, 512),
                                               (30, 500, 64, 1, 512), (370, 500, 64, 1, 0), (370, 512, 32, 1, 0), (740, 512, 32, 1, 0),
                                               (30, 1500, 32, 1, 0), (34, 1000, 64, 1, 0), (20, 2100, 64, 0, 0),
                                               (80, 212, 32, 0, 0), (80, 212, 32, 1, 0), (37, 1000, 32, 0, 0), (80, 212, 64, 1, 0), (72, 474, 64, 0, 0)])
def test_row_walks_match_the_cuda_cores(bh, n, d, mask, chunk):
    """Several row tiles to a CTA, in every order they are taken in: head by head, tile by tile, in pairs (even and odd
    numbers of tiles).  Both families' bounds against float64 add up to 2e-5 of the largest value at these lengths."""
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v, go = [torch.randn(bh, n, d, generator=g, device="cuda") for _ in range(4)]
    kw = dict(mask=bool(mask), normalize=True, p=1 if chunk else 2)
    impl = dict(impl="moments", chunk=chunk) if chunk else {}
    out, den, st = _cabi.forward(q, k, v, **kw, **impl)
    got = (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, **kw, **impl))
    out, den, st = _cabi.forward(q, k, v, impl="dense_ffma", **kw)
    want = (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, impl="dense_ffma", **kw))
    assert _cabi.device_status() == 0
    for x, r, name in zip(got, want, ("out", "dq", "dk", "dv")):
        # per head, so that a row tile that is left out or taken twice shows whatever the other heads' values are
        err = float(((x - r).abs().amax((1, 2)) / r.abs().amax((1, 2))).max())
        assert err < BOUND, (name, err)
