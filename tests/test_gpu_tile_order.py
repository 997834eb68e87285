"""Causal grids of a few waves start tile by tile over all heads, longer and shorter ones head by head.  The order must not
change a bit of the result: each problem is run whole (tile by tile) and in slices of its heads that the same kernels
take head by head.  Without normalisation no sum depends on the order in which CTAs finish."""
import pytest
import torch

from fastmax_b200 import _cabi

pytestmark = pytest.mark.gpu

# dtype, d, heads, heads per slice, nq, nk: row tiles of the whole / of a slice against the 148 (short rows: 296) CTAs that run
# at once.  Two row tiles of d = 128 share a CTA of the forward.
CASES = [(torch.float32, 32, 24, 12, 1000, 1000), (torch.float32, 64, 24, 12, 900, 1100), (torch.float32, 32, 150, 75, 130, 130),
         (torch.bfloat16, 64, 6, 3, 4000, 4000), (torch.bfloat16, 64, 40, 20, 1000, 1000), (torch.bfloat16, 64, 160, 80, 140, 300),
         (torch.bfloat16, 64, 350, 175, 200, 400), (torch.bfloat16, 128, 20, 5, 2000, 2000), (torch.bfloat16, 128, 40, 8, 700, 1000)]


@pytest.mark.parametrize("dtype,d,heads,part,nq,nk", CASES, ids=[f"{str(c[0])[6:]}d{c[1]}bh{c[2]}nq{c[4]}nk{c[5]}" for c in CASES])
def test_order_of_row_tiles_changes_nothing(dtype, d, heads, part, nq, nk):
    g = torch.Generator(device="cuda").manual_seed(nq + d)
    mk = lambda n, s: (s * torch.randn(heads, n, d, generator=g, device="cuda")).to(dtype)  # noqa: E731
    q, k, v, go = mk(nq, d ** -0.5), mk(nk, d ** -0.5), mk(nk, 1.0), mk(nq, 1.0)
    kw = dict(mask=True, normalize=False, p=2)

    def run(*t):
        out, den, st = _cabi.forward(*t[:3], **kw)
        return (out, den) + tuple(_cabi.backward(*t[:3], out, den, st, t[3], **kw))

    whole = run(q, k, v, go)
    for lo in range(0, heads, part):
        s = slice(lo, lo + part)
        for a, b, name in zip(whole, run(*[t[s].contiguous() for t in (q, k, v, go)]), ("out", "den", "dq", "dk", "dv")):
            assert torch.equal(a[s], b), (lo, name)
    assert _cabi.device_status() == 0
    # the last head against float64, so that both orders are not wrong together
    x, y, z = [t[-1].double().requires_grad_(True) for t in (q, k, v)]
    sc = x @ y.T
    f = (1 + sc + 0.5 * sc * sc).tril(nk - nq)
    ref = (f @ z) / f.sum(-1, keepdim=True)
    want = (ref.detach(),) + torch.autograd.grad(ref, (x, y, z), go[-1].double())
    for a, b, name in zip((whole[0],) + whole[2:], want, ("out", "dq", "dk", "dv")):
        assert float((a[-1].double() - b).abs().max() / b.abs().max()) < (1e-4 if dtype == torch.float32 else 2e-2), name
