"""Second-order read-outs of the bf16 moment family (d = 64): both kinds, walked by persistent CTAs in groups of 256
tokens, against the CPU oracle.  Sizes at the edges: last groups of one row, of half a group, of a row short of one, one
group per chunk and several, chunk counts around one, and more groups than SMs, so that a CTA takes several in turn."""
import pytest
import torch

from gpu_util import assert_close, oracle, run_cabi

from fastmax_b200 import _cabi

pytestmark = pytest.mark.gpu


def _problem(bh, n, seed, mask, a1=1.0, a2=0.5):
    g = torch.Generator().manual_seed(seed)
    t = [torch.randn(1, bh, n, 64, generator=g) for _ in range(4)]
    return t, dict(mask=mask, normalize=1, p=2, a0=1.0, a1=a1, a2=a2, lim=1.0)


# bh, n, mask, chunk
SIZES = [(1, 257, 1, 256), (2, 511, 1, 256), (2, 513, 1, 256), (3, 640, 1, 512), (2, 1025, 1, 512), (1, 2049, 1, 2048),
         (40, 1300, 1, 256), (1, 1, 0, 256), (2, 255, 0, 256), (3, 385, 0, 256), (80, 700, 0, 512),
         # either side of where the copies for grad_k fit into the rows of grad_v: 1216 tokens a state
         (2, 2431, 1, 2048), (2, 2432, 1, 2048), (3, 1215, 0, 1024), (3, 1216, 0, 1024)]


@pytest.mark.parametrize("bh,n,mask,chunk", SIZES)
def test_readouts_at_the_edges_of_their_groups(bh, n, mask, chunk):
    t, kw = _problem(bh, n, 900 + n, mask)
    got, _ = run_cabi(*t, torch.bfloat16, impl="moments", chunk=chunk, **kw)
    assert _cabi.device_status() == 0
    ref = oracle(*t, torch.bfloat16, dense=True, **kw)
    what = f"{bh} x {n}, chunk {chunk}"
    if n > 1:
        assert_close(got, ref, torch.bfloat16, what)
        return
    # one token: grad_q and grad_k are zero, the difference of two terms of |g| |v| = 64 with bf16 operands (2^-9 each)
    for t, floor in ((0, 1e-2), (1, 8.0), (2, 8.0), (3, 1e-2)):
        assert_close(got[t:t + 1], ref[t:t + 1], torch.bfloat16, f"{what}, tensor {t}", floor=floor)


def test_readouts_without_a_second_order_coefficient():
    """a2 = 0: the factors of the second-order sums vanish, the first-order terms must not go with them."""
    t, kw = _problem(2, 700, 77, 1, a1=0.7, a2=0.0)
    got, _ = run_cabi(*t, torch.bfloat16, impl="moments", chunk=256, **kw)
    ref = oracle(*t, torch.bfloat16, dense=True, **kw)
    assert_close(got, ref, torch.bfloat16, "a2 = 0")


@pytest.mark.parametrize("bh,n,mask,chunk", [(2, 2431, 1, 2048), (2, 2432, 1, 2048), (3, 1215, 0, 1024), (3, 1216, 0, 1024),
                                             (2, 700, 1, 256), (1, 5000, 1, 2048)])
@pytest.mark.parametrize("keep", [True, False])
def test_workspaces_are_not_overrun(bh, n, mask, chunk, keep):
    """Forward and backward in workspaces of exactly the sizes asked for, the bytes behind them untouched; with the states kept
    beside the statistics, and in a statistics buffer whose alignment leaves no room for them."""
    L, dev = _cabi.lib(), "cuda"
    q, k, v, go = [torch.randn(bh, n, 64, device=dev, generator=torch.Generator(device=dev).manual_seed(i)).bfloat16()
                   for i in range(4)]
    prob = _cabi.Problem(dtype=_cabi.BF16, bh=bh, bhkv=bh, nq=n, nk=n, d=64, mask=mask, normalize=1, p=2, impl=3, a0=1, a1=1,
                         a2=0.5, lim=1, temperature=1, chunk=chunk)
    out, gq, gk, gv = [torch.empty_like(q) for _ in range(4)]
    den = torch.empty(bh, n, device=dev)
    stats = torch.full((L.fastmax_b200_stats_bytes(prob) + 4096,), 0x5A, dtype=torch.uint8, device=dev)
    sp = stats.data_ptr() + (0 if keep else 8)
    stream = torch.cuda.current_stream().cuda_stream

    def scratch(size):
        return torch.full((size + 4096,), 0x5A, dtype=torch.uint8, device=dev), size

    ws, size = scratch(L.fastmax_b200_forward_workspace_bytes(prob))
    _cabi._check(L.fastmax_b200_forward(prob, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), den.data_ptr(), sp,
                                        ws.data_ptr(), size, stream), "forward")
    assert (ws[size:] == 0x5A).all() and (stats[-4096 + 8:] == 0x5A).all()
    ws, size = scratch(L.fastmax_b200_backward_workspace_bytes(prob))
    _cabi._check(L.fastmax_b200_backward(prob, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), den.data_ptr(), sp,
                                         go.data_ptr(), gq.data_ptr(), gk.data_ptr(), gv.data_ptr(), ws.data_ptr(), size,
                                         stream), "backward")
    assert (ws[size:] == 0x5A).all() and _cabi.device_status() == 0
    kw = dict(mask=mask, normalize=1, p=2, a0=1.0, a1=1.0, a2=0.5, lim=1.0)
    ref = oracle(*[t.float().cpu()[None] for t in (q, k, v, go)], torch.bfloat16, dense=True, **kw)
    assert_close([t.float().cpu()[None] for t in (out, gq, gk, gv)], ref, torch.bfloat16, f"{bh} x {n}, chunk {chunk}")
