"""The `fastmax_cuda` extension at lengths where the library's own calls run on the moment family, while both directions
of the extension are of the score form: normalised gradients must not depend on what lies behind the statistics, the
result carries no moment states, and float32 gets its tensor-core kernels."""
import pytest
import torch

import fastmax_b200
from fastmax_b200 import _cabi

fastmax_cuda = pytest.importorskip("fastmax_cuda", reason="build with python -m fastmax_b200.build --torch-ext")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,d,heads,n,mask", [(torch.bfloat16, 64, 32, 2304, True), (torch.float32, 32, 24, 3600, True),
                                                  (torch.bfloat16, 64, 4, 3000, False)])
def test_normalised_backward_of_long_first_order_sequences(dtype, d, heads, n, mask):
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v, go = [torch.randn(heads, n, d, generator=g, device="cuda").to(dtype) for _ in range(4)]
    torch.full((64 << 20,), 7.0, device="cuda")            # what freed memory holds is not zero
    _cabi.profile(True)
    o = fastmax_cuda.forwardpass(q, k, v, None, mask, 0.0, True, 1.0, 1.0, 1.0, 0.5, 1.0, 1)
    names = {n_ for n_, _ in _cabi.profile_records()}
    _cabi.profile(False)
    assert not any("moments" in n_ or "first" in n_ for n_ in names), names
    assert ("fm_dense_split_fwd" in names) == (dtype == torch.float32)
    assert o.untyped_storage().nbytes() <= 4 * o.numel() + 256 + 8 * 2 * heads + 256
    got = [o[:, :, :d]] + list(fastmax_cuda.backwardpass(q, k, v, o, go, mask, 1.0, 1.0, 0.5, 1))
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out = fastmax_b200.FASTMultiHeadAttention()(*leaves, mask=mask, normalize=True, p=1)
    want = [out.detach()] + list(torch.autograd.grad(out, leaves, go))
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    for a, b, name in zip(got, want, ("out", "dq", "dk", "dv")):
        assert float((a.float() - b.float()).abs().max() / b.float().abs().max()) < tol, name


def test_no_room_for_the_operand_parts():
    """float32 on a device that has room for the results but not for 6 bytes per operand element."""
    bh, n, d = 256, 4096, 32
    q, k, v, go = [torch.randn(bh, n, d, device="cuda") for _ in range(4)]
    total, tensor = torch.cuda.get_device_properties(0).total_memory, q.numel() * 4

    def run(room_fwd=None, room_bwd=None):
        def leave(room):
            torch.cuda.empty_cache()
            if room is not None:
                torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + room * tensor) / total)
        _cabi.profile(True)
        try:
            leave(room_fwd)
            o = fastmax_cuda.forwardpass(q, k, v, None, True, 0.0, True, 1.0, 1.0, 1.0, 0.5, 1.0, 2)
            leave(room_bwd)
            got = [o[:, :, :d]] + list(fastmax_cuda.backwardpass(q, k, v, o, go, True, 1.0, 1.0, 0.5, 2))
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        names = {n_ for n_, _ in _cabi.profile_records()}
        _cabi.profile(False)
        return got, names

    want, names = run()
    assert any("split" in n_ for n_ in names), names
    got, names = run(2.5, 6)     # forward: the result and 4.5 tensors; backward: a copy of out, three gradients and 6
    assert not any("split" in n_ for n_ in names), names
    for a, b, name in zip(got, want, ("out", "dq", "dk", "dv")):
        assert float((a - b).abs().max() / b.abs().max()) < 2e-5, name
