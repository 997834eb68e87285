"""float32 unmasked second-order forward in moment form against float64: last groups of 1, 15, 65 and 161 of 256 query rows,
last key blocks of 1, 15 and 63 of 64, grouped heads, more query groups than SMs, keys and queries whose squares alone would
leave float32's range.

Bound: operands and products are exact to 2^-24; a sum over n keys is rounded to nearest once per 64 keys, a random walk of
sqrt(n / 64) steps of 2^-25 of it, 13 steps at 10 000 keys, and the rows average 4 160 such sums.  1e-6 in the 2-norm is
six times the 1.6e-7 of a result that is rounded a few times.  On N(0,1) inputs scores are small and the second order is
half a percent of the result, so this bound sees a product of parts of order 2^-8 (4e-6 or more when dropped) and the first
order, but not the products of order 2^-16; those are what the second test is for."""
import pytest
import torch

from fastmax_b200 import _cabi

pytestmark = pytest.mark.gpu


def reference(q, k, v, norm, a):
    out, den = torch.empty_like(q, dtype=torch.float64), torch.empty(q.shape[:2], dtype=torch.float64, device=q.device)
    ratio = q.shape[0] // k.shape[0]
    for h in range(q.shape[0]):
        x, y, z = q[h].double(), k[h // ratio].double(), v[h // ratio].double()
        if norm:
            x, y = x / x.norm(dim=1).max(), y / y.norm(dim=1).max()
        for i in range(0, x.shape[0], 4096):
            s = x[i:i + 4096] @ y.T
            f = a[0] + a[1] * s + a[2] * s * s
            den[h, i:i + 4096] = f.sum(1)
            out[h, i:i + 4096] = f @ z / f.sum(1, keepdim=True)
    return out, den


def rel(a, b):
    return float((a.double() - b).norm() / b.norm())


# query heads, key heads, nq, nk, scale of the keys, of the queries
@pytest.mark.parametrize("bh,bhkv,nq,nk,kscale,qscale", [
    (8, 8, 9999, 9999, 1.0, 1.0), (8, 2, 40001, 2111, 1e17, 1e-18), (16, 4, 4097, 8191, 0.1, 1e18),
    (64, 64, 4001, 4033, 1e-17, 1e18)])
def test_moment_form_forward_against_float64(bh, bhkv, nq, nk, kscale, qscale):
    g = torch.Generator(device="cuda").manual_seed(nq)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v = rnd(bh, nq, 64) * qscale, rnd(bhkv, nk, 64) * kscale, rnd(bhkv, nk, 64)
    _cabi.profile(True)
    out, den, _ = _cabi.forward(q, k, v, mask=0, normalize=1, p=2, a0=1.0, a1=0.7, a2=0.4, lim=1.0)
    names = {n for n, _ in _cabi.profile_records()}
    _cabi.profile(False)
    assert "fm_split_readout" in names, names
    assert _cabi.device_status() == 0
    ref, ref_den = reference(q, k, v, 1, (1.0, 0.7, 0.4))
    assert rel(out, ref) < 1e-6 and rel(den, ref_den) < 1e-6, (rel(out, ref), rel(den, ref_den))


@pytest.mark.parametrize("heads,nq,nk", [(64, 4033, 4097), (72, 4999, 3333)])
def test_every_product_of_parts_counts(heads, nq, nk):
    """Queries and keys of about equal norms in a plane of two feature axes, another pair of axes in each head, and f = 1 + 4 s^2:
    two thirds of a denominator, and as much of a result, are one to three second-order sums, with no other 4 000 to average
    their errors away.  Emulated in float64, leaving out one of the five products below h h in the sums moves the result
    by 1.4e-6 or more, in the read-out the result or the denominator by 1.1e-6 or more; rounding of the kind above stays
    below 3e-7 (sqrt(64) steps of 2^-25 and a handful of roundings of the row)."""
    g = torch.Generator(device="cuda").manual_seed(heads)
    q, k = [torch.zeros(heads, n, 64, device="cuda") for n in (nq, nk)]
    for h in range(heads):
        axes = torch.randperm(64, generator=torch.Generator().manual_seed(h))[:2].cuda()
        for t in (q, k):
            x = torch.randn(t.shape[1], 2, device="cuda", generator=g)
            t[h][:, axes] = x / x.norm(dim=1, keepdim=True) * (1 - 0.1 * torch.rand(len(x), 1, device="cuda", generator=g))
    v = torch.randn(heads, nk, 64, device="cuda", generator=g)
    _cabi.profile(True)
    out, den, _ = _cabi.forward(q, k, v, mask=0, normalize=1, p=2, a0=1.0, a1=0.0, a2=4.0, lim=1.0)
    names = {n for n, _ in _cabi.profile_records()}
    _cabi.profile(False)
    assert "fm_split_readout" in names, names
    ref, ref_den = reference(q, k, v, 1, (1.0, 0.0, 4.0))
    assert rel(out, ref) < 6e-7 and rel(den, ref_den) < 6e-7, (rel(out, ref), rel(den, ref_den))


@pytest.mark.parametrize("offset", [80.0, 800.0])
def test_unnormalised_keys_with_a_common_direction_keep_the_score_form(offset):
    """Keys share a direction that the queries do not see: scores near 8 from norms of 8 and `offset`.  A score is a sum of 64
    products of up to |q| |k| / 8, rounded to 2^-24 of the largest partial sum, which f = 1 + s + s^2 / 2 doubles: a bound of
    2^-23 (8 + offset) beside the 1e-6 of the sums over the keys, of which random signs leave about a twentieth.  Sums over
    feature pairs would be rounded to 2^-24 |q|^2 |k|^2 / 2, 1.6e-5 and 1.6e-3 on these inputs."""
    heads, n = 64, 4097
    g = torch.Generator(device="cuda").manual_seed(int(offset))
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    q, k, v, u = rnd(heads, n, 64), rnd(heads, n, 64), rnd(heads, n, 64), rnd(heads, 1, 64)
    u = u / u.norm(dim=2, keepdim=True)
    q, k = q - (q * u).sum(2, keepdim=True) * u, k + offset * u
    out, _, _ = _cabi.forward(q, k, v, mask=0, normalize=0, p=2, a0=1.0, a1=1.0, a2=0.5, lim=1.0)
    err = rel(out, reference(q, k, v, 0, (1.0, 1.0, 0.5))[0])
    assert err < 1e-6 + 2.0 ** -23 * (8 + offset) / 8, err
