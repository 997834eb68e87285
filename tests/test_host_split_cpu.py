"""Workspace sizes (host arithmetic, no device).  The operand parts of the float32 score kernels take 6 bytes per element;
very large problems and the families that name the CUDA cores need none.  The fused first-order path needs room for
its states and their bf16 copies, and backward for the scaled gradient, but for no fp32 rows.  The second-order moment family
needs room for its states, result rows and one layout of their bf16 copies."""
import pytest

from fastmax_b200 import _cabi


def sizes(**kw):
    base = dict(dtype=_cabi.F32, bh=16, bhkv=16, nq=1000, nk=1000, d=32, mask=1, normalize=1, p=2, impl=0, a0=1, a1=1,
                a2=0.5, lim=1, temperature=1)
    base.update(kw)
    prob, L = _cabi.Problem(**base), _cabi.lib()
    return L.fastmax_b200_forward_workspace_bytes(prob), L.fastmax_b200_backward_workspace_bytes(prob)


def test_parts_take_six_bytes_per_element():
    fwd, bwd = sizes()
    elements = 16 * 1000 * 32
    assert 3 * 6 * elements <= fwd <= 3 * (6 * elements + 256)
    assert 4 * 6 * elements <= bwd <= 4 * (6 * elements + 256) + 4 * 16 * 1000 + 1024


@pytest.mark.parametrize("kw", [dict(impl=1), dict(d=16), dict(d=128), dict(bh=4096, bhkv=4096, nq=10000, nk=10000, d=64)],
                         ids=["cuda cores named", "d 16", "d 128", "parts above 48 GiB"])
def test_other_problems_need_no_forward_workspace(kw):
    fwd, bwd = sizes(**kw)
    rows = kw.get("bh", 16) * kw.get("nq", 1000)
    assert fwd == 0 and bwd <= 4 * rows + 8 * kw.get("bh", 16) + 1024


@pytest.mark.parametrize("kw", [dict(), dict(d=64, p=1, nq=8000, nk=8000), dict(d=32, mask=0, p=1, nq=8000, nk=8000),
                                dict(dtype=_cabi.BF16, d=64)], ids=["score", "moments", "unmasked moments", "bf16"])
def test_least_workspace_leaves_out_the_operand_parts(kw):
    base = dict(dtype=_cabi.F32, bh=16, bhkv=16, nq=1000, nk=1000, d=32, mask=1, normalize=1, p=2, impl=0, a0=1, a1=1, a2=0.5,
                lim=1, temperature=1)
    prob, L = _cabi.Problem(**{**base, **kw}), _cabi.lib()
    fwd, bwd = sizes(**kw)
    least = (L.fastmax_b200_forward_workspace_least_bytes(prob), L.fastmax_b200_backward_workspace_least_bytes(prob))
    element = prob.bh * prob.nq * prob.d
    parts = 6 * element if prob.dtype == _cabi.F32 and prob.mask else 0
    assert fwd - least[0] == 3 * parts
    moments = _cabi.selected_impl(prob) == "moments"
    # score form: the parts take the place of the CUDA-core kernels' row dots
    assert 4 * parts <= bwd - least[1] <= 4 * parts + (4 * prob.bh * prob.nq + 256) * (moments and parts > 0)


@pytest.mark.parametrize("heads,n", [(256, 2048), (256, 1233), (64, 8192)])
def test_fused_first_order_needs_no_fp32_rows(heads, n):
    fwd, bwd = sizes(dtype=_cabi.BF16, bh=heads, bhkv=heads, nq=n, nk=n, d=64, p=1)
    tensor = 2 * heads * n * 64
    # states: 65 rows of 68 floats per 512 tokens, copies: 64 x 64 bf16; a last partial chunk counts as a whole one
    states = heads * -(-n // 512) * (65 * 68 * 4 + 64 * 64 * 2)
    assert fwd <= states + 4096
    assert bwd <= tensor + states + 2 * 4 * heads * n + 8 * heads + 4096


@pytest.mark.parametrize("kw,moment", [
    (dict(), True), (dict(normalize=0), False), (dict(a1=-1.0), True), (dict(a1=1.01), False), (dict(a1=-1.01), False),
    (dict(a2=2.3), True), (dict(a2=2.6), False), (dict(a1=0.0, a2=4.0), True), (dict(a1=0.0, a2=4.01), False),
    (dict(a1=0.0, a2=-0.66), True), (dict(a1=0.0, a2=-0.67), False), (dict(a1=0.5, a2=-0.5), False),
    (dict(a0=2.0, a1=2.0, a2=1.0), True), (dict(lim=0.5), True), (dict(lim=-1.0), True), (dict(lim=1.01), False),
    (dict(lim=0.0), True), (dict(a0=0.0), False), (dict(a0=-1.0, a1=-1.0, a2=-0.5), False), (dict(a0=0.9), False),
    (dict(a1=float("nan")), False), (dict(a2=float("nan")), False), (dict(lim=float("inf")), False)])
def test_moment_form_forward_only_where_the_terms_hardly_cancel(kw, moment):
    """Its sums round relative to a2 |q|^2 |k|^2, whatever the scores are: on |s| <= lim^2 the polynomial has to stay above a
    fifth of the sizes of its terms.  The workspace tells which form is planned."""
    heads, nq, nk = 64, 4000, 4033
    fwd, _ = sizes(**{**dict(bh=heads, bhkv=heads, nq=nq, nk=nk, d=64, mask=0), **kw})
    parts = 6 * 64 * heads * (nq + 2 * nk)
    assert (fwd > parts + 1024) == moment


# heads, n, mask, chunk, family (3: moments), bytes of the forward and backward workspace and of the shards' that an earlier
# layout took: a caller that keeps buffers of those sizes is served
@pytest.mark.parametrize("heads,n,mask,chunk,impl,most", [
    (1024, 10000, 1, 0, 0, (12510199808, 19104768000, 5556469760, 12110069760)),
    (32, 262144, 1, 0, 0, (9168331264, 14570595072, 4496293888, 9865003008)),
    (64, 6000, 0, 0, 0, (498106368, 745402880, 208367616, 454127616)),
    (16, 2049, 1, 0, 3, (80937984, 102051328, 26611968, 47593728)),
    (16, 1, 1, 256, 3, (45265664, 45276416, 9048320, 9058560)),
    (4, 10000, 1, 256, 3, (286453760, 312214016, 100839680, 126439680)),
    (4, 300, 0, 256, 3, (18415872, 19188992, 4834048, 5602048)),
    (3, 2431, 1, 2048, 3, (15474176, 20171264, 5287680, 9955328)),
    (16, 12001, 1, 1536, 3, (285254144, 408912896, 122276096, 245166336))])
def test_second_order_moments_need_room_for_one_layout_of_copies(heads, n, mask, chunk, impl, most):
    prob = _cabi.Problem(dtype=_cabi.BF16, bh=heads, bhkv=heads, nq=n, nk=n, d=64, mask=mask, normalize=1, p=2, impl=impl, a0=1,
                         a1=1, a2=0.5, lim=1, temperature=1, chunk=chunk)
    L = _cabi.lib()
    got = (L.fastmax_b200_forward_workspace_bytes(prob), L.fastmax_b200_backward_workspace_bytes(prob),
           L.fastmax_b200_shard_forward_workspace_bytes(prob), L.fastmax_b200_shard_backward_workspace_bytes(prob))
    assert all(g <= m for g, m in zip(got, most)), (got, most)
    # states of 4161 rows of 68 floats a chunk, a total, rows of 65 floats and copies of 344 064 bytes a state
    states = heads * -(-n // (chunk or 2048))
    rows = heads * n * 65 * 4
    assert got[0] <= states * (4161 * 68 * 4 + 344064) + heads * 4161 * 68 * 4 + rows + 4096


@pytest.mark.parametrize("n,chunk,kept", [(10000, 0, True), (12001, 1536, False), (1649 * 7, 1792, False), (1650 * 7, 1792, True),
                                          (1500, 1536, False), (1, 256, False)])
def test_which_states_are_kept_does_not_hang_on_the_layout_of_their_copies(n, chunk, kept):
    """fp32 states and 68 x 64 rows of 64 bf16 against twice the tensors: from 1650 tokens a chunk on."""
    heads = 16
    prob = _cabi.Problem(dtype=_cabi.BF16, bh=heads, bhkv=heads, nq=n, nk=n, d=64, mask=1, normalize=1, p=2, impl=3, a0=1, a1=1,
                         a2=0.5, lim=1, temperature=1, chunk=chunk)
    assert (_cabi.lib().fastmax_b200_stats_bytes(prob) > 8 * 2 * heads + 256) == kept
