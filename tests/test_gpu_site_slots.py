"""Split and merge of the packed projection at the shapes where the lanes' slots can go wrong: head sizes whose slots do
not divide a warp or exceed it, token counts around a warp's, rotated widths of every kind, few and many vectors."""
import pytest
import torch

from oracle.call_site_oracle import split_heads

from fastmax_b200 import _cabi

pytestmark = pytest.mark.gpu

# batch, tokens, heads, groups, head size, rotated features
SHAPES = [(2, 9, 2, 1, 24, 8), (1, 7, 3, 3, 40, 24), (1, 8, 1, 1, 544, 544), (2, 33, 2, 2, 528, 16), (1, 1, 4, 2, 64, 64),
          (3, 17, 40, 8, 64, 48), (1, 3, 300, 100, 16, 16), (1, 1001, 2, 1, 128, 64), (2, 5, 2, 2, 8, 8),
          # odd numbers of 16-byte pieces in bf16, one slot more than a warp among them; vectors taken in pairs, an odd number of them
          (1, 13, 2, 1, 24, 16), (3, 70, 4, 2, 72, 16), (2, 33, 3, 3, 88, 64), (1, 5, 1, 1, 520, 16), (1, 37, 5, 5, 8, 8),
          (2, 300, 3, 1, 8, 8), (2, 70, 3, 1, 16, 16)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["fp32", "bf16"])
@pytest.mark.parametrize("b,t,heads,groups,hs,r", SHAPES)
def test_split_and_merge_slots(b, t, heads, groups, hs, r, dtype):
    g = torch.Generator().manual_seed(hs + t)
    qkv = torch.randn(b, t, (heads + 2 * groups) * hs, generator=g).to(dtype)
    cos, sin = torch.randn(t, r, generator=g), torch.randn(t, r, generator=g)
    x = qkv.double().requires_grad_(True)
    ref = split_heads(x, cos.double(), sin.double(), heads, groups, hs, r, expand=False)
    got = _cabi.qkv_split_rope(qkv.cuda().view(b, t, groups, heads // groups + 2, hs), cos, sin, r)
    # two products and a sum in fp32, then one rounding to the result's type; |x|, |cos|, |sin| < 5
    tol = 50 * 2.0 ** (-23 if dtype == torch.float32 else -8)
    for a, e in zip(got, ref):
        assert float((a.cpu().double() - e.detach().reshape(a.shape)).abs().max()) < tol
    grads = [torch.randn(a.shape, generator=g).to(dtype) for a in got]
    want, = torch.autograd.grad(ref, (x,), [w.double().reshape(e.shape) for w, e in zip(grads, ref)])
    merged = _cabi.qkv_merge_rope_grad(*[w.cuda() for w in grads], cos, sin, r, b)
    assert float((merged.cpu().double().reshape(want.shape) - want).abs().max()) < tol
