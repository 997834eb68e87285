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
         (40, 1300, 1, 256), (1, 1, 0, 256), (2, 255, 0, 256), (3, 385, 0, 256), (80, 700, 0, 512)]


@pytest.mark.parametrize("bh,n,mask,chunk", SIZES)
def test_readouts_at_the_edges_of_their_groups(bh, n, mask, chunk):
    t, kw = _problem(bh, n, 900 + n, mask)
    got, _ = run_cabi(*t, torch.bfloat16, impl="moments", chunk=chunk, **kw)
    assert _cabi.device_status() == 0
    ref = oracle(*t, torch.bfloat16, dense=True, **kw)
    # one token: grad_q and grad_k are zero, the difference of two terms of |g| |v| = 64 with bf16 operands (2^-9 each)
    assert_close(got, ref, torch.bfloat16, f"{bh} x {n}, chunk {chunk}", floor=8.0 if n == 1 else 1e-2)


def test_readouts_without_a_second_order_coefficient():
    """a2 = 0: the factors of the second-order sums vanish, the first-order terms must not go with them."""
    t, kw = _problem(2, 700, 77, 1, a1=0.7, a2=0.0)
    got, _ = run_cabi(*t, torch.bfloat16, impl="moments", chunk=256, **kw)
    ref = oracle(*t, torch.bfloat16, dense=True, **kw)
    assert_close(got, ref, torch.bfloat16, "a2 = 0")
