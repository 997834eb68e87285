"""Workspace sizes of the float32 score kernels (host arithmetic, no device): the operand parts take 6 bytes per element;
very large problems and the families that name the CUDA cores need none, as before."""
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
