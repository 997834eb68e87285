"""Prompt processing of the decode state at the sizes where its kernels change: the tensor-core kernel's blocks of 128
tokens and their K steps of 16 (bf16, d 64 and 128), the CUDA-core kernel's batches, and the few-token kernel (below 24
tokens at p = 1; at p = 2 below 28 for those, else 40); onto an empty and onto a filled state, against float64 sums.

Bound: products are exact (bf16) or rounded once (float32) and sums of up to n terms are accumulated in float32, so
the error of an element is within n * 2^-24 of the sum of its terms' magnitudes; elements of a state of N(0,1) keys
stay within sqrt(n) of that sum's share, for which 2e-5 relative to the largest element leaves a factor of ten."""
import pytest
import torch

import fastmax_b200

pytestmark = pytest.mark.gpu


def want(k, v, p):
    k, vt = k.double(), torch.cat([v.double(), torch.ones_like(v[..., :1], dtype=torch.float64)], -1)
    h, n, d = k.shape
    rows = [k.transpose(1, 2) @ vt, vt.sum(1, keepdim=True)]
    if p == 2:
        rows.insert(0, (k.unsqueeze(3) * k.unsqueeze(2)).flatten(2).transpose(1, 2) @ vt)
    return torch.cat(rows, 1)


def rows_of(state, heads, d, p):
    f = d + 1 + (d * d if p == 2 else 0)
    s = state.view(heads, 4 + f * (d + 1))
    return s[:, :4].cpu(), s[:, 4:].view(heads, f, d + 1).double().cpu()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("heads,d,p,pieces", [
    (2, 64, 2, (1, 63)), (3, 64, 2, (64,)), (2, 64, 2, (65, 64, 127)), (2, 64, 1, (200, 3)), (1, 128, 2, (129, 70)),
    (2, 128, 1, (64, 65)), (2, 32, 2, (300, 31)), (1, 32, 1, (90,)), (5, 64, 2, (1000,))])
def test_append_matches_float64_sums(heads, d, p, pieces, dtype):
    g = torch.Generator().manual_seed(d + sum(pieces))
    n = sum(pieces)
    k, v = [torch.randn(heads, n, d, generator=g).to(dtype) for _ in range(2)]
    st = fastmax_b200.FastmaxDecodeState(heads, heads, d, dtype=dtype, device="cuda:0", p=p)
    lo = 0
    for m in pieces:
        st.append(k[:, lo:lo + m].contiguous().cuda(), v[:, lo:lo + m].contiguous().cuda())
        lo += m
    head, got = rows_of(st.state, heads, d, p)
    ref = want(k, v, p)
    assert float((got - ref).abs().max() / ref.abs().max()) < 2e-5
    assert head[:, 1].contiguous().view(torch.int32).tolist() == [n] * heads
    assert torch.allclose(head[:, 0].double(), (k.double() ** 2).sum(-1).amax(1), rtol=1e-6)
    assert not head[:, 2:].any()
    if p == 2:       # both places of a pair hold the same bits
        s2 = got[:, :d * d].view(heads, d, d, d + 1)
        assert torch.equal(s2, s2.transpose(1, 2))


@pytest.mark.parametrize("heads,d,p,pieces", [
    (2, 64, 2, (28, 27)), (2, 64, 2, (112, 113)), (3, 64, 2, (128, 127)), (2, 128, 2, (28, 144)), (2, 128, 2, (129, 240)),
    (2, 64, 1, (14, 128)), (2, 128, 1, (13, 257, 16)), (4, 64, 2, (3000,))])
def test_append_at_the_edges_of_blocks_and_steps(heads, d, p, pieces):
    test_append_matches_float64_sums(heads, d, p, pieces, torch.bfloat16)


@pytest.mark.parametrize("n", [64, 65, 100, 128, 200, 1000])
def test_sums_of_a_prompt_stay_short_in_the_tensor_core(n):
    """Its accumulators cut off what they add, by 2^-23 of the partial sum at most and by a third of that on average, always
    towards zero.  With keys and values of one sign an accumulator of 64 tokens, four steps that see a quarter to all of its sum,
    loses 2.5 x 2^-23 / 3 = 1.0e-7 (one of 128 tokens 1.8e-7); everything else is rounded to nearest.  The normaliser adds a step's
    sixteen numbers only: roundings to nearest of random sign, which stay below 2^-24 of the sum."""
    g = torch.Generator(device="cuda").manual_seed(n)
    k, v = [torch.randn(4, n, 64, generator=g, device="cuda").abs().bfloat16() for _ in range(2)]
    st = fastmax_b200.FastmaxDecodeState(4, 4, 64, dtype=torch.bfloat16, device="cuda:0")
    st.append(k, v)
    got, ref = rows_of(st.state, 4, 64, 2)[1], want(k, v, 2).cpu()
    err = [float((a - b).norm() / b.norm()) for a, b in ((got[..., :64], ref[..., :64]), (got[..., 64], ref[..., 64]))]
    assert err[0] < 1.4e-7 and err[1] < 2.0 ** -24, err


@pytest.mark.parametrize("d,ratio", [(64, 1), (64, 5), (32, 6), (128, 3)])
def test_step_reads_groups_of_any_size_and_keeps_the_state_symmetric(d, ratio):
    g = torch.Generator().manual_seed(d + ratio)
    kv, n = 2, 70
    k, v = [torch.randn(kv, n, d, generator=g) for _ in range(2)]
    q = torch.randn(kv * ratio, 1, d, generator=g)
    st = fastmax_b200.FastmaxDecodeState(kv * ratio, kv, d, dtype=torch.float32, device="cuda:0", normalize=False)
    st.append(k[:, :-1].contiguous().cuda(), v[:, :-1].contiguous().cuda())
    q = q * d ** -0.5
    out = st.step(q.cuda(), k[:, -1:].contiguous().cuda(), v[:, -1:].contiguous().cuda())
    s = (q.double().view(kv, ratio, d) @ k.double().transpose(1, 2))
    f = 1 + s + 0.5 * s * s
    ref = (f @ v.double()) / f.sum(-1, keepdim=True)
    got = out.double().cpu().view(kv, ratio, d)
    assert float((got - ref).abs().max() / ref.abs().max()) < 1e-4
    head, rows = rows_of(st.state, kv, d, 2)
    s2 = rows[:, :d * d].view(kv, d, d, d + 1)
    assert torch.equal(s2, s2.transpose(1, 2)) and not head[:, 2:].any()
    assert head[:, 1].contiguous().view(torch.int32).tolist() == [n] * kv
