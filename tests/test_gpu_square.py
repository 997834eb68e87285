"""grad_v and grad_k of the bf16 score kernels that evaluate the polynomial as a square and a rest (d = 64, equal heads, second
order): chunks, mid-length rows and long rows, masked and not, with second-order coefficients down to where the square would
cancel, and at every scale of the inputs.

Bound: the polynomial, the scaled upstream gradient and the result are each rounded to bf16 once, 2^-9 at most, so the 2-norm error
against float32 on the CUDA cores is within 3 x 2^-9."""
import pytest
import torch

from fastmax_b200 import _cabi

pytestmark = pytest.mark.gpu

# heads, tokens, chunk, mask
SHAPES = {"chunks of 256": (240, 641, 256, 1), "chunks of 512": (34, 1281, 512, 1), "mid-length": (38, 1000, 0, 1),
          "mid-length unmasked": (60, 650, 0, 0), "long": (8, 4096, 0, 1), "long unmasked": (8, 4100, 0, 0)}
BOUND = 3 * 2.0 ** -9


def errors(shape, scale=1.0, **coef):
    heads, n, chunk, mask = SHAPES[shape]
    g = torch.Generator(device="cuda").manual_seed(n)
    q, k, v, go = [torch.randn(heads, n, 64, generator=g, device="cuda") for _ in range(4)]
    q, k, v, go = (q * scale).bfloat16(), (k * scale).bfloat16(), v.bfloat16(), go.bfloat16()
    kw = dict(mask=bool(mask), normalize=True, p=2, **coef)

    def run(q, k, v, go, **impl):
        out, den, st = _cabi.forward(q, k, v, **kw, **impl)
        return _cabi.backward(q, k, v, out, den, st, go, **kw, **impl)[1:]

    got = run(q, k, v, go, **(dict(impl="moments", chunk=chunk) if chunk else dict(impl="dense_tc")))
    want = run(*[t.float() for t in (q, k, v, go)], impl="dense_ffma")
    assert _cabi.device_status() == 0
    return [float((x.double() - r.double()).norm() / r.double().norm()) for x, r in zip(got, want)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("coef", [dict(a2=0.5), dict(a2=1 / 64), dict(a2=1 / 65), dict(a2=1e-3), dict(a2=1e-5), dict(a2=1e-7),
                                  dict(a2=1e-9), dict(a0=0.2, a1=0.0, a2=0.5), dict(a0=2.0, a1=-1.0, a2=0.25)],
                         ids=lambda c: ",".join("%s=%g" % x for x in c.items()))
def test_small_second_order_coefficients_do_not_cancel(shape, coef):
    dk, dv = errors(shape, **coef)
    assert dk < BOUND and dv < BOUND, (dk, dv)


@pytest.mark.parametrize("shape", ["chunks of 256", "long"])
def test_precision_does_not_hang_on_the_scale_of_the_inputs(shape):
    """Normalised inputs give the same scores at any scale.  Eight scales over an octave, whose second-order coefficients take
    every mantissa: the errors, means over a million roundings each, agree to a few in a thousand."""
    dv = [errors(shape, scale=2.0 ** (i / 8))[1] for i in range(8)]
    assert max(dv) < 1.04 * min(dv), dv
    if shape == "long":           # (the chunks' states hold products of raw keys and values, which have left float32 there)
        dk, dv = errors(shape, scale=1e9)
        assert dk < BOUND and dv < BOUND, (dk, dv)
