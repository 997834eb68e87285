"""The bf16 score kernels that walk row tiles (d = 64, equal head counts): several row tiles to a CTA in every order they are
taken in, ragged rows and columns, more keys than queries, chunks with a shorter last one, one and two rounds of row tiles and
many, against the float32 score kernels on the CUDA cores.  Tolerance: the bf16 one of the other tests (2e-2 of a head's
largest value)."""
import pytest
import torch

from fastmax_b200 import _cabi

pytestmark = pytest.mark.gpu

# bh, nq, nk, mask, p, normalize, chunk, walking kernels (forward; grad_k and grad_v)
CASES = [(38, 1000, 1000, 1, 2, 1, 0, 1), (34, 1150, 1150, 1, 1, 0, 0, 1), (20, 1030, 1030, 1, 1, 0, 0, 0), (38, 1900, 2029, 1, 2, 1, 0, 1),
         (55, 690, 650, 0, 2, 1, 0, 2), (44, 900, 930, 0, 2, 1, 0, 2), (60, 650, 520, 0, 1, 1, 0, 2), (200, 650, 640, 0, 1, 0, 0, 2),
         (75, 515, 515, 1, 2, 1, 256, 2), (34, 1281, 1281, 1, 2, 0, 512, 2), (240, 641, 641, 1, 2, 1, 256, 2), (150, 1031, 1031, 1, 2, 1, 0, 1),
         (75, 515, 515, 1, 1, 1, 512, 1), (34, 1281, 1281, 1, 1, 0, 512, 1), (240, 641, 641, 1, 1, 1, 512, 1),
         # in pairs: even and odd numbers of row tiles, whole chunks, a shorter last one
         (185, 1024, 1024, 1, 2, 1, 0, 1), (185, 1900, 1900, 1, 2, 1, 0, 1), (185, 1024, 1024, 1, 2, 1, 512, 2), (560, 1281, 1281, 1, 2, 0, 512, 2)]


@pytest.mark.parametrize("cfg", CASES, ids=["bh%dnq%dnk%dm%dp%dz%dc%dw%d" % c for c in CASES])
def test_row_walks_match_the_cuda_cores(cfg):
    bh, nq, nk, mask, p, norm, chunk, walking = cfg
    g = torch.Generator(device="cuda").manual_seed(nq + nk)
    q, k, v, go = [torch.randn(bh, n, 64, generator=g, device="cuda") for n in (nq, nk, nk, nq)]
    if not norm:
        q, k = q / 8, k / 8
    q, k, v, go = [t.bfloat16() for t in (q, k, v, go)]
    kw = dict(mask=bool(mask), normalize=bool(norm), p=p)
    impl = dict(impl="moments", chunk=chunk) if chunk else dict(impl="dense_tc")

    def run(q, k, v, go, **impl):
        out, den, st = _cabi.forward(q, k, v, **kw, **impl)
        return (out,) + tuple(_cabi.backward(q, k, v, out, den, st, go, **kw, **impl))

    run(q, k, v, go, **impl)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        for _ in range(2):               # the trace may miss the very first launch
            got = run(q, k, v, go, **impl)
        torch.cuda.synchronize()
    names = [e.key for e in prof.key_averages()]
    assert sum("walk_kernel<" in n for n in names) == walking, names
    assert _cabi.device_status() == 0
    want = run(*[t.float() for t in (q, k, v, go)], impl="dense_ffma")
    for x, r, name in zip(got, want, ("out", "dq", "dk", "dv")):
        # per head, so that a row tile that is left out or taken twice shows whatever the other heads' values are
        err = float(((x.float() - r).abs().amax((1, 2)) / r.abs().amax((1, 2))).max())
        assert err < 2e-2, (name, err)
    bt, _, _ = _cabi.forward_bt(q, k, v, bh // 2 if bh % 2 == 0 else bh, **kw, **impl)
    if chunk and p == 2:         # (two issuers add the halves of a block to these chunks' states, in the order they come)
        torch.testing.assert_close(bt.transpose(1, 2).reshape(got[0].shape), got[0], rtol=2 ** -7, atol=2e-3)
    else:
        assert torch.equal(bt.transpose(1, 2).reshape(got[0].shape), got[0])
