"""The C++ host side of the frequent calls: the same results, errors and autograd behaviour as the Python functions."""
import pytest
import torch

import fastmax_b200
from fastmax_b200 import _native
from fastmax_b200.attention import FASTMultiHeadAttention_Function

pytestmark = pytest.mark.gpu
KW = dict(mask=True, normalize=True, temperature=2.0, a0=1.0, a1=1.0, a2=0.5, lim=1.0, p=2)


def _inputs(dtype=torch.float32, heads=4, kv=4, n=70, d=32):
    g = torch.Generator(device="cuda").manual_seed(3)
    t = [torch.randn(1, h, n, d, generator=g, device="cuda").to(dtype) for h in (heads, kv, kv, heads)]
    return [x.requires_grad_(True) for x in t[:3]] + [t[3]]


def _python(q, k, v):
    return FASTMultiHeadAttention_Function.apply(q, k, v, None, KW["mask"], 0.0, KW["normalize"], KW["temperature"], 1.0,
                                                 1.0, 0.5, 1.0, 2)


def test_module_is_here():
    assert _native.host() is not None and _native.plain_mode()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kv", [4, 2])
def test_same_as_the_python_function(dtype, kv):
    q, k, v, go = _inputs(dtype, kv=kv)
    mod = fastmax_b200.FASTMultiHeadAttention()
    a, b = mod(q, k, v, **KW), _python(q, k, v)
    assert a.grad_fn is not None and torch.equal(a, b)
    # the dots of the normalisation gradient are summed by atomics: one row a head may differ by its last bits
    tol = dict(rtol=0, atol=1e-5 if dtype == torch.float32 else 2e-2)
    for x, y in zip(torch.autograd.grad(a, (q, k, v), go), torch.autograd.grad(b, (q, k, v), go)):
        assert torch.allclose(x, y, **tol)
    # a transposed input and an upstream gradient of another layout
    qt = q.detach().transpose(2, 3).contiguous().transpose(2, 3).requires_grad_(True)
    gx = torch.autograd.grad(mod(qt, k, v, **KW), qt, go.transpose(2, 3).contiguous().transpose(2, 3))[0]
    assert torch.allclose(gx, torch.autograd.grad(_python(q, k, v), q, go)[0], **tol)


def test_graph_rules():
    q, k, v, go = _inputs()
    mod = fastmax_b200.FASTMultiHeadAttention()
    out = mod(q, k, v, **KW)
    out.backward(go)
    with pytest.raises(RuntimeError):
        out.backward(go)                                     # saved tensors are freed
    out = mod(q, k, v, **KW)
    with torch.no_grad():
        k.mul_(2.0)
    with pytest.raises(RuntimeError):
        out.backward(go)                                     # a saved input was modified
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t.shape) or t.clone(), lambda t: t):
        out = mod(q, k, v, **KW)
    out.backward(go)
    assert len(seen) == 6
    with torch.no_grad():
        assert mod(q, k, v, **KW).grad_fn is None
    mod(q.detach(), k.detach(), v, **KW).backward(go)


@pytest.mark.parametrize("change,error", [
    (dict(p=3), ValueError), (dict(k=lambda t: t[:, :, :, :16]), ValueError), (dict(k=lambda t: t.double()), ValueError),
    (dict(q=lambda t: t.cpu()), RuntimeError)])
def test_errors_are_those_of_the_python_function(change, error):
    q, k, v, _ = _inputs()
    kw = dict(KW, p=change.get("p", 2))
    q, k = change.get("q", lambda t: t)(q), change.get("k", lambda t: t)(k)
    with pytest.raises(error):
        fastmax_b200.FASTMultiHeadAttention()(q, k, v, **kw)


def test_transforms_take_the_python_function():
    q, k, v, go = _inputs()
    mod = fastmax_b200.FASTMultiHeadAttention()
    for f in (lambda: torch.func.vmap(lambda a: mod(a, k[0], v[0], **KW))(q),
              lambda: torch.func.grad(lambda a: mod(a, k, v, **KW).sum())(q)):
        with pytest.raises(RuntimeError):
            f()


def test_call_site_and_decode(monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(5)
    qkv = torch.randn(2, 45, 8 * 64, generator=g, device="cuda").bfloat16().requires_grad_(True)
    cos, sin = [torch.randn(45, 32, generator=g, device="cuda") for _ in range(2)]
    go = torch.randn(2, 45, 4 * 64, generator=g, device="cuda").bfloat16()

    def site():
        y = fastmax_b200.fastmax_attention_from_qkv(qkv, cos, sin, 4, 2, 64, 32)
        return y, torch.autograd.grad(y, qkv, go)[0]

    def decode():
        st = fastmax_b200.FastmaxDecodeState(4, 2, 64, torch.bfloat16, "cuda")
        rows = [torch.randn(h, 1, 64, generator=torch.Generator(device="cuda").manual_seed(h), device="cuda").bfloat16()
                for h in (4, 2, 2)]
        with pytest.raises(ValueError):
            st.step(rows[0][:2], rows[1], rows[2])
        return st.step(*rows), st.state.clone(), st.tokens

    a, da = site(), decode()
    monkeypatch.setattr(_native, "host", lambda: None)
    b, db = site(), decode()
    assert torch.equal(a[0], b[0]) and torch.allclose(a[1], b[1], rtol=0, atol=2e-2)
    assert torch.equal(da[0], db[0]) and torch.equal(da[1], db[1]) and da[2] == db[2] == 1


def test_decode_step_lets_other_threads_run():
    """A launch waits once the device's queue is full (some 1000 kernels); other Python threads go on meanwhile."""
    import threading
    import time

    st = fastmax_b200.FastmaxDecodeState(4, 4, 64, torch.bfloat16, "cuda")
    row = torch.randn(4, 1, 64, device="cuda").bfloat16()
    st.step(row, row, row)
    torch.cuda.synchronize()
    gaps, done = [0.0], threading.Event()

    def watch():
        last = time.perf_counter()
        while not done.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    t = threading.Thread(target=watch)
    t.start()
    start = time.perf_counter()
    torch.cuda._sleep(1_500_000_000)        # clocks: 0.75 s and more
    for _ in range(3000):
        st.step(row, row, row)
    issued = time.perf_counter() - start
    done.set()
    t.join()
    torch.cuda.synchronize()
    assert issued > 0.5, issued             # the queue was full for most of the pause
    assert max(gaps) < 0.25, max(gaps)


def test_tables_that_no_rotation_reads_may_change():
    g = torch.Generator(device="cuda").manual_seed(6)
    qkv = torch.randn(2, 45, 8 * 64, generator=g, device="cuda").bfloat16().requires_grad_(True)
    cos, sin = torch.zeros(45, 64, device="cuda"), torch.zeros(45, 64, device="cuda")
    y = fastmax_b200.fastmax_attention_from_qkv(qkv, cos, sin, 4, 2, 64, 0)
    cos.add_(1.0)
    sin.add_(1.0)
    y.sum().backward()
    assert torch.isfinite(qkv.grad).all()


def test_function_modes_see_the_calls_inside(monkeypatch):
    """A torch function mode takes the Python function, as with the module absent; a default device is no such mode."""
    class Record(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            self.seen.append(getattr(func, "__name__", str(func)))
            return func(*args, **(kwargs or {}))

    q, k, v, _ = _inputs()
    mod = fastmax_b200.FASTMultiHeadAttention()
    seen = []
    for present in (True, False):
        if not present:
            monkeypatch.setattr(_native, "host", lambda: None)
        with Record() as mode:
            mode.seen = []
            mod(q, k, v, **KW)
        seen.append(mode.seen)
    assert "contiguous" in seen[0] and seen[0] == seen[1]
    with torch.device("cuda"):
        assert _native.plain_mode()


def test_without_the_queries_of_torch_the_python_function_serves(monkeypatch):
    q, k, v, _ = _inputs()
    monkeypatch.setattr(_native, "_queries", None)
    assert torch.equal(fastmax_b200.FASTMultiHeadAttention()(q, k, v, **KW), _python(q, k, v))


def test_two_threads_with_streams_of_their_own():
    import threading

    mod = fastmax_b200.FASTMultiHeadAttention()
    t = [_inputs(torch.bfloat16, n=300 + 40 * i, d=64) for i in range(2)]
    want = []
    for q, k, v, go in t:
        out = mod(q, k, v, **KW)
        want.append((out.detach(),) + torch.autograd.grad(out, (q, k, v), go))
    torch.cuda.synchronize()
    bad = []

    def work(i):
        try:
            q, k, v, go = t[i]
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(30):
                    out = mod(q, k, v, **KW)
                    got = (out.detach(),) + torch.autograd.grad(out, (q, k, v), go)
                    torch.cuda.current_stream().synchronize()
                    # outputs bit for bit; of the gradients, the atomically summed dots may move one row a head
                    assert torch.equal(got[0], want[i][0]) and torch.equal(got[3], want[i][3])
                    assert all(torch.allclose(x, y, rtol=0, atol=2e-2) for x, y in zip(got, want[i]))
        except BaseException as e:          # noqa: BLE001 -- handed to the main thread
            bad.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    [x.start() for x in threads]
    [x.join() for x in threads]
    assert not bad, bad


def test_under_graph_capture():
    """A training step and a decode step captured once and replayed on new inputs."""
    mod = fastmax_b200.FASTMultiHeadAttention()
    q, k, v, go = _inputs(torch.bfloat16, n=333, d=64)
    st = fastmax_b200.FastmaxDecodeState(4, 4, 64, torch.bfloat16, "cuda")
    row = torch.randn(4, 1, 64, device="cuda").bfloat16()

    def both():
        out = mod(q, k, v, **KW)
        return (out.detach(),) + torch.autograd.grad(out, (q, k, v), go) + (st.step(row, row, row),)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        both()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = both()
    with torch.no_grad():
        for x in (q, k, v, row):
            x.copy_(torch.randn_like(x))
    st.reset()
    graph.replay()
    torch.cuda.synchronize()
    got = [x.clone() for x in got]
    st.reset()
    for x, y in zip(got, both()):
        assert torch.allclose(x, y, rtol=0, atol=2e-2)
