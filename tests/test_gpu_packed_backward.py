"""The packed forward and the library's backward as a pair (what a binding of the reference's forwardpass and backwardpass
calls), at lengths where the backward runs on the moment family and reads states behind the statistics: the packed
forward has to have left them.  The statistics buffer is filled with NaN first, so that what nobody wrote shows.

The gradients are compared with the plain-layout pair of the same problem; tolerances are those of the other tests, bf16
2e-2 and float32 1e-4 of the largest value."""
import pytest
import torch

from fastmax_b200 import _cabi

pytestmark = pytest.mark.gpu


def pair(q, k, v, go, out_dtype, with_workspace, **kw):
    L, (bh, n, d) = _cabi.lib(), q.shape
    prob = _cabi.make_problem(q, k, kw["mask"], kw["normalize"], 1.0, 1.0, 1.0, 0.5, 1.0, kw["p"])
    assert _cabi.selected_impl(prob) == "moments"
    o = torch.empty(bh, n, d + 1, device="cuda")
    stats = torch.full((L.fastmax_b200_stats_bytes(prob),), 255, dtype=torch.uint8, device="cuda")
    wsb = L.fastmax_b200_forward_workspace_bytes(prob) if with_workspace else 0
    ws = torch.empty(max(wsb, 1), dtype=torch.uint8, device="cuda")
    rc = L.fastmax_b200_forward_packed(prob, q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), stats.data_ptr(),
                                       ws.data_ptr() if wsb else None, wsb, torch.cuda.current_stream().cuda_stream)
    _cabi._check(rc, "forward_packed")
    out, den = o[:, :, :d].to(out_dtype).contiguous(), o[:, :, d].contiguous()
    q, k, v = [t.clone() for t in (q, k, v)]                      # aligned, whatever the forward was given
    return (out,) + tuple(_cabi.backward(q, k, v, out, den, stats, go, **kw))


# dtype, d, p, mask, heads, n: float32 and bf16 states on the CUDA cores, first and second order on the tensor cores
CASES = [(torch.bfloat16, 64, 1, True, 96, 1700), (torch.bfloat16, 64, 1, True, 24, 4096), (torch.bfloat16, 128, 1, True, 16, 4300),
         (torch.bfloat16, 64, 2, True, 2, 10000), (torch.bfloat16, 64, 2, False, 3, 6500), (torch.bfloat16, 64, 1, False, 3, 6500),
         (torch.float32, 16, 1, True, 8, 2400), (torch.float32, 32, 1, True, 32, 4100), (torch.float32, 16, 2, False, 3, 2500),
         (torch.bfloat16, 32, 1, False, 3, 2500)]


@pytest.mark.parametrize("with_workspace", [False, True], ids=["no workspace", "workspace"])
@pytest.mark.parametrize("dtype,d,p,mask,heads,n", CASES,
                         ids=[f"{str(c[0])[6:]}d{c[1]}p{c[2]}m{int(c[3])}bh{c[4]}n{c[5]}" for c in CASES])
def test_backward_after_packed_forward(dtype, d, p, mask, heads, n, with_workspace):
    g = torch.Generator(device="cuda").manual_seed(n + d)
    q, k, v, go = [torch.randn(heads, n, d, generator=g, device="cuda").to(dtype) for _ in range(4)]
    kw = dict(mask=mask, normalize=True, p=p)
    got = pair(q, k, v, go, dtype, with_workspace, **kw)
    out, den, st = _cabi.forward(q, k, v, **kw)
    want = (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, **kw))
    assert _cabi.device_status() == 0
    for a, b, name in zip(got, want, ("out", "dq", "dk", "dv")):
        assert float((a.float() - b.float()).abs().max() / b.float().abs().max()) < (1e-4 if dtype == torch.float32 else 2e-2), name


@pytest.mark.parametrize("p,heads,n", [(1, 96, 1700), (2, 2, 10000)])
def test_states_of_unaligned_keys_and_values(p, heads, n):
    """k and v that TMA cannot read: the states come from the CUDA-core kernels, in the layout the backward expects."""
    g = torch.Generator(device="cuda").manual_seed(n)
    size = heads * n * 64
    flat = [torch.randn(size + 1, generator=g, device="cuda").bfloat16() for _ in range(3)]
    q, k, v = [t[1:].view(heads, n, 64) for t in flat]
    assert k.data_ptr() % 16
    go = torch.randn(heads, n, 64, generator=g, device="cuda").bfloat16()
    kw = dict(mask=True, normalize=True, p=p)
    got = pair(q, k, v, go, torch.bfloat16, False, **kw)
    q, k, v = [t.clone() for t in (q, k, v)]
    out, den, st = _cabi.forward(q, k, v, **kw)
    want = (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, **kw))
    assert _cabi.device_status() == 0
    for a, b, name in zip(got, want, ("out", "dq", "dk", "dv")):
        assert float((a.float() - b.float()).abs().max() / b.float().abs().max()) < 2e-2, name


def test_statistics_at_eight_byte_alignment():
    """The statistic words need no more than 8 bytes; a buffer placed like that keeps no states, forward or backward."""
    g = torch.Generator(device="cuda").manual_seed(8)
    heads, n, d = 96, 1700, 64
    q, k, v, go = [torch.randn(heads, n, d, generator=g, device="cuda").bfloat16() for _ in range(4)]
    kw = dict(mask=True, normalize=True, p=1)
    out, den, st = _cabi.forward(q, k, v, **kw)
    want = (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, **kw))
    odd = torch.full((st.numel() + 8,), 255, dtype=torch.uint8, device="cuda")[8:]
    bufs = dict(out=torch.empty_like(q), den=torch.empty_like(den), stats=odd,
                workspace=torch.empty(_cabi.workspace_bytes(q, k, **kw)[0], dtype=torch.uint8, device="cuda"))
    out, den, st = _cabi.forward(q, k, v, buffers=bufs, **kw)
    got = (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, **kw))
    for a, b, name in zip(got, want, ("out", "dq", "dk", "dv")):
        assert float((a.float() - b.float()).abs().max() / b.float().abs().max()) < 2e-2, name
