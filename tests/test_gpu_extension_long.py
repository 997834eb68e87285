"""The `fastmax_cuda` extension at lengths where the library's own backward would read moment states that the packed
forward does not leave: normalised gradients must not depend on what lies behind the statistics."""
import pytest
import torch

import fastmax_b200

fastmax_cuda = pytest.importorskip("fastmax_cuda", reason="build with python -m fastmax_b200.build --torch-ext")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,d,heads,n,mask", [(torch.bfloat16, 64, 32, 2304, True), (torch.float32, 32, 24, 3600, True),
                                                  (torch.bfloat16, 64, 4, 3000, False)])
def test_normalised_backward_of_long_first_order_sequences(dtype, d, heads, n, mask):
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v, go = [torch.randn(heads, n, d, generator=g, device="cuda").to(dtype) for _ in range(4)]
    torch.full((64 << 20,), 7.0, device="cuda")            # what freed memory holds is not zero
    o = fastmax_cuda.forwardpass(q, k, v, None, mask, 0.0, True, 1.0, 1.0, 1.0, 0.5, 1.0, 1)
    got = [o[:, :, :d]] + list(fastmax_cuda.backwardpass(q, k, v, o, go, mask, 1.0, 1.0, 0.5, 1))
    leaves = [t.clone().requires_grad_(True) for t in (q, k, v)]
    out = fastmax_b200.FASTMultiHeadAttention()(*leaves, mask=mask, normalize=True, p=1)
    want = [out.detach()] + list(torch.autograd.grad(out, leaves, go))
    tol = 1e-4 if dtype == torch.float32 else 2e-2
    for a, b, name in zip(got, want, ("out", "dq", "dk", "dv")):
        assert float((a.float() - b.float()).abs().max() / b.float().abs().max()) < tol, name
