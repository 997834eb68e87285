"""CPU-side checks: the C ABI library loads and exports what the header declares,
the host wrappers validate their arguments, and the pure-PyTorch path of the
package agrees with the reference-generated vectors."""
import ctypes
import os
import re

import pytest
import torch

from conftest import ROOT, case_kwargs, load_small_cases
from oracle.fastmax_oracle import rel_err

import fastmax_b200
from fastmax_b200 import _cabi

CASES = load_small_cases()


def _declared_functions():
    names = set()
    for fn in os.listdir(os.path.join(ROOT, "include")):
        if fn.endswith(".h"):
            txt = open(os.path.join(ROOT, "include", fn)).read()
            txt = re.sub(r"/\*.*?\*/", "", txt, flags=re.S)
            names |= set(re.findall(r"\b(fastmax_b200_\w+)\s*\(", txt))
    return sorted(names)


def test_library_exports_every_declared_symbol():
    lib = ctypes.CDLL(_cabi.LIB_PATH)
    declared = _declared_functions()
    assert len(declared) >= 8
    for name in declared:
        assert hasattr(lib, name), f"{name} is declared in include/ but not exported"
    assert set(_cabi.EXPORTS) <= set(declared)


def test_version_and_size_queries_need_no_gpu():
    L = _cabi.lib()
    assert L.fastmax_b200_version() >= 100
    prob = _cabi.Problem(dtype=0, bh=6, bhkv=3, nq=10, nk=12, d=32, mask=1, normalize=1, p=2, impl=0,
                         a0=1, a1=1, a2=0.5, lim=1, temperature=1)
    assert L.fastmax_b200_stats_bytes(prob) == 8 * 9
    assert L.fastmax_b200_backward_workspace_bytes(prob) >= 4 * (9 + 60)
    assert ctypes.sizeof(_cabi.Problem) == 64


def test_family_selection_follows_the_measured_break_even_points():
    """The library's choice of kernel family (host arithmetic, no device): tensor-core score kernels for short
    rows, the moment family beyond the rule's lines -- causal bf16 p=2 d=64 from about 9 300 keys on (the
    headline shape has 10 000), unmasked from about 5 400, p=1 at almost any length -- and never for a few
    query rows against many keys; fp32 stays on the CUDA-core score kernels."""
    def pick(**kw):
        base = dict(dtype=_cabi.BF16, bh=1024, bhkv=1024, nq=10000, nk=10000, d=64, mask=1, normalize=1, p=2,
                    impl=0, a0=1, a1=1, a2=0.5, lim=1, temperature=1)
        base.update(kw)
        return _cabi.selected_impl(_cabi.Problem(**base))

    assert pick() == "moments"                                           # the headline shape
    assert pick(nq=8192, nk=8192) == "dense_tc"
    assert pick(nq=9216, nk=9216) == "dense_tc"
    assert pick(nq=12288, nk=12288) == "moments"
    assert pick(bh=32, bhkv=32, nq=262144, nk=262144) == "moments"       # the long-context configuration
    assert pick(mask=0, nq=4096, nk=4096) == "dense_tc"
    assert pick(mask=0, nq=6144, nk=6144) == "moments"
    assert pick(mask=0, nq=256, nk=6000) == "dense_tc"                   # few query rows, many keys
    assert pick(mask=0, nq=1, nk=100000) == "dense_tc"
    assert pick(mask=0, p=1, d=128, nq=16384, nk=16384, normalize=0) == "moments"
    assert pick(mask=0, d=128, nq=16384, nk=16384, normalize=0) == "dense_tc"
    assert pick(dtype=_cabi.F32, d=32, nq=1000, nk=1000) == "dense_ffma"
    assert pick(impl=_cabi.IMPL["dense_tc"]) == "dense_tc"               # a forced family is reported as such
    assert pick(impl=_cabi.IMPL["moments_ffma"]) == "moments"
    with pytest.raises(RuntimeError):
        pick(impl=_cabi.IMPL["dense_tc"], dtype=_cabi.F32, d=32)


FIRST_ORDER_LINES = [   # dtype, d, heads, longest length in score form, shortest on the moment family
    (_cabi.BF16, 64, 256, 1216, 1248), (_cabi.BF16, 64, 8, 3520, 3552), (_cabi.BF16, 128, 256, 2800, 2832),
    (_cabi.F32, 32, 256, 3120, 3152), (_cabi.F32, 64, 256, 3952, 3984),
    # both families on the CUDA cores: by what is saved, and beyond 1100 (d = 128: 880) tokens for any number of heads
    (_cabi.F32, 8, 256, 528, 544), (_cabi.F32, 16, 256, 576, 592), (_cabi.F32, 16, 64, 656, 672), (_cabi.F32, 16, 1, 1100, 1101),
    (_cabi.BF16, 8, 256, 528, 544), (_cabi.BF16, 16, 8, 1088, 1101), (_cabi.BF16, 32, 256, 560, 576), (_cabi.BF16, 32, 8, 944, 960),
    (_cabi.F32, 128, 256, 880, 881), (_cabi.F32, 128, 1, 880, 881),
    # operand parts above 48 GiB: no split kernels, so the rate model of the CUDA-core kernels, beyond one chunk of 2048
    (_cabi.F32, 64, 40000, 2128, 2144)]


@pytest.mark.parametrize("dtype,d,heads,below,above", FIRST_ORDER_LINES)
def test_causal_first_order_lines_between_the_families(dtype, d, heads, below, above):
    def pick(n):
        return _cabi.selected_impl(_cabi.Problem(dtype=dtype, bh=heads, bhkv=heads, nq=n, nk=n, d=d, mask=1, normalize=1,
                                                 p=1, impl=0, a0=1, a1=1, a2=0.5, lim=1, temperature=1))
    dense = "dense_tc" if dtype == _cabi.BF16 and d >= 64 else "dense_ffma"
    assert [pick(n) for n in (272, 500, below, above, 4 * above)] == [dense] * 3 + ["moments"] * 2


@pytest.mark.parametrize("dtype,d,n,mask,chunk", [(_cabi.BF16, 64, 1100, 1, 0), (_cabi.BF16, 64, 8000, 0, 0), (_cabi.F32, 8, 600, 1, 0)])
def test_more_heads_than_a_grid_dimension_stay_in_score_form(dtype, d, n, mask, chunk):
    def pick(heads):
        return _cabi.selected_impl(_cabi.Problem(dtype=dtype, bh=heads, bhkv=heads, nq=n, nk=n, d=d, mask=mask, normalize=1,
                                                 p=1, impl=0, a0=1, a1=1, a2=0.5, lim=1, temperature=1, chunk=chunk))
    assert pick(65535) == "moments"
    assert pick(65536) == pick(70000) == ("dense_tc" if dtype == _cabi.BF16 else "dense_ffma")


def test_bad_arguments_are_rejected_before_any_launch():
    L = _cabi.lib()
    prob = _cabi.Problem(dtype=0, bh=2, bhkv=2, nq=4, nk=4, d=32, mask=1, normalize=0, p=3, impl=0,
                         a0=1, a1=1, a2=0.5, lim=1, temperature=1)
    rc = L.fastmax_b200_forward(prob, 1, 1, 1, 1, 1, 1, None, 0, None)
    assert rc == -1 and b"p must be 1 or 2" in L.fastmax_b200_last_error()
    assert L.fastmax_b200_backward(prob, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1, None, 0, None) == -1
    assert L.fastmax_b200_forward_packed(prob, 1, 1, 1, 1, 1, None, 0, None) == -1
    prob.p, prob.d = 2, 24
    assert L.fastmax_b200_forward(prob, 1, 1, 1, 1, 1, 1, None, 0, None) == -1
    prob.d, prob.nk = 32, 3
    assert L.fastmax_b200_forward(prob, 1, 1, 1, 1, 1, 1, None, 0, None) == -1
    prob.nk, prob.bhkv = 4, 3
    assert L.fastmax_b200_forward(prob, 1, 1, 1, 1, 1, 1, None, 0, None) == -1


@pytest.mark.skipif(torch.cuda.is_available(), reason="made-up addresses, which only a machine without a device may see")
@pytest.mark.parametrize("p", [1, 2])
@pytest.mark.parametrize("mask", [0, 1])
def test_unaligned_state_buffers_are_an_argument_error(p, mask):
    """The bf16 moment kernels move states, their copies and result rows 16 bytes at a time, all of them in the caller's
    workspace: an unaligned one is refused before any launch, as are unaligned states and totals of a shard."""
    L, good, bad, big = _cabi.lib(), 1 << 20, (1 << 20) + 8, 1 << 40
    prob = _cabi.Problem(dtype=_cabi.BF16, bh=2, bhkv=2, nq=5000, nk=5000, d=64, mask=mask, normalize=1, p=p, impl=3, a0=1,
                         a1=1, a2=0.5, lim=1, temperature=1)

    def codes(ws, state):
        g = good
        yield L.fastmax_b200_forward(prob, g, g, g, g, g, g, ws, big, None)
        yield L.fastmax_b200_backward(prob, g, g, g, g, g, g, g, g, g, g, ws, big, None)
        if mask:
            yield L.fastmax_b200_forward_bt(prob, g, g, g, g, g, g, 2, ws, big, None)
            yield L.fastmax_b200_backward_bt(prob, g, g, g, g, g, g, g, 2, g, g, g, ws, big, None)
            yield L.fastmax_b200_shard_dq_far(prob, g, g, g, g, g, state, ws, big, None)
        yield L.fastmax_b200_shard_forward(prob, g, g, g, g, state, state, g, g, ws, big, None)
        yield L.fastmax_b200_shard_qg_state(prob, g, g, g, g, g, state, state, ws, big, None)
        yield L.fastmax_b200_shard_backward(prob, g, g, g, g, g, g, g, g, state, state, state, g, g, g, g, 0, ws, big, None)

    for ws, state in ((bad, good), (bad, bad)):
        for rc in codes(ws, state):
            assert rc == -1 and b"16-byte aligned" in L.fastmax_b200_last_error(), (rc, L.fastmax_b200_last_error())
    for rc in (L.fastmax_b200_shard_kv_state(prob, good, good, bad, good, None),
               L.fastmax_b200_shard_kv_state(prob, good, good, good, bad, None),
               L.fastmax_b200_shard_forward(prob, good, good, good, good, bad, bad, good, good, good, big, None)):
        assert rc == -1
    assert all(rc not in (0, -1) for rc in codes(good, good))       # nothing else is wrong with these calls: no device here


def test_custom_path_refuses_cpu_tensors():
    q = torch.randn(1, 2, 8, 8)
    with pytest.raises(RuntimeError):
        fastmax_b200.FASTMultiHeadAttention()(q, q, q, None, True)
    with pytest.raises(ValueError):
        fastmax_b200.fastmax_function(q, q, q, p=3)


@pytest.mark.parametrize("c", CASES, ids=[c["tag"] for c in CASES])
def test_pytorch_path_matches_reference_vectors(c):
    q, k, v, go = [c[x].double().requires_grad_(x != "go") for x in ("q", "k", "v", "go")]
    mod = fastmax_b200.FASTMultiHeadAttention(use_custom_gradient=False)
    out = mod(q, k, v, None, c["mask"], 0.0, c["normalize"], 1.0, c["a0"], c["a1"], c["a2"], c["lim"], c["p"])
    out.backward(go)
    tol = 1e-9 if c["a0"] == 1.0 else 1e-6   # see tests/test_oracle.py::tol64
    for got, name in ((out.detach(), "out"), (q.grad, "dq"), (k.grad, "dk"), (v.grad, "dv")):
        assert rel_err(got, c[name + "64"]) < tol, name


def test_pytorch_path_blocked_scan_and_attn_matrix():
    c = [x for x in CASES if x["tag"] == "m1p2n0_a"][0]
    q, k, v = [c[x].double() for x in ("q", "k", "v")]
    kw = dict(mask=1, normalize=0, a0=c["a0"], a1=c["a1"], a2=c["a2"], lim=c["lim"], p=2)
    a = fastmax_b200.fastmax_function(q, k, v, block=5, **kw)
    assert rel_err(a, c["out64"]) < 1e-10
    n = q.shape[2]
    tri = torch.tril(torch.ones(n, n))
    ans, attn = fastmax_b200.fastmax_function(q, k, v, mask=tri, a0=c["a0"], a1=c["a1"], a2=c["a2"],
                                              create_attn_matrix=1)
    assert rel_err(ans, c["out64"]) < 1e-10
    assert torch.allclose(attn.sum(-1), torch.ones_like(attn.sum(-1)))


def test_rpe_matrix_creator_shapes():
    r = fastmax_b200.rpe_matrix_creator(5, 8, "cpu", torch.float32)
    assert r.shape == (9, 8) and float(r.abs().sum()) == 0.0
    r = fastmax_b200.rpe_matrix_creator(5, 8, "cpu", torch.float32, structured=True)
    assert r.shape == (9, 8) and torch.allclose(r[4], torch.tensor([0., 1.] * 4))


def test_numa_preference_is_a_no_op_without_a_gpu():
    """The helper must never raise: without CUDA (or without a readable topology) it reports -1."""
    from fastmax_b200.host import prefer_gpu_numa_node
    if not torch.cuda.is_available():
        assert prefer_gpu_numa_node("cuda:0") == -1
    else:
        assert prefer_gpu_numa_node("cuda:0") >= -1
