"""The work whose speed this repository is judged by: its public entry points on realistic inputs.

A case is a dict of plain values.  ``kind`` says which entry point it goes through:

* ``train``   -- ``FASTMultiHeadAttention`` forward and backward through autograd
* ``forward`` -- the same module under ``no_grad`` (evaluation, scoring)
* ``site``    -- ``fastmax_attention_from_qkv`` forward and backward (the model's call site)
* ``append``  -- ``FastmaxDecodeState.append`` of a prompt into a cleared state
* ``step``    -- ``FastmaxDecodeState.step``, one token per sequence

``b`` sequences of ``h`` query heads over ``g`` key/value heads, ``n`` tokens, head size ``d``.
"""
import math

import torch

import fastmax_b200

COEF = dict(a0=1.0, a1=1.0, a2=0.5, lim=1.0)
DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}


def _case(name, kind, dtype, b, h, g, n, d, p, mask, normalize):
    return dict(name=name, kind=kind, dtype=dtype, b=b, h=h, g=g, n=n, d=d, p=p, mask=mask, normalize=normalize)


def listed():
    return [
        # one short sequence, forward and backward: what launches and latency cost a small model or a test run
        _case("train_small_bf16", "train", "bf16", 1, 8, 8, 197, 64, 2, True, True),
        # the small fp32 configuration of the benchmark (unmasked, 16 heads in all)
        _case("train_small_fp32", "train", "fp32", 2, 8, 8, 1024, 32, 2, False, True),
        # the fp32 training configuration of the benchmark, ragged length
        _case("train_fp32", "train", "fp32", 64, 8, 8, 1000, 32, 2, True, True),
        # the reference's published timings are fp32 forward passes over 10 000 tokens; an eighth of its batch
        _case("forward_fp32", "forward", "fp32", 8, 8, 8, 10000, 64, 2, False, True),
        # the benchmark's headline configuration: causal bf16 training over 10 000 tokens
        _case("train_bf16", "train", "bf16", 64, 16, 16, 10000, 64, 2, True, True),
        # grouped key/value heads, large heads, a length that divides nothing
        _case("train_grouped_bf16", "train", "bf16", 2, 32, 8, 2047, 128, 2, True, True),
        # the benchmark's long unmasked first-order configuration, a quarter of its batch
        _case("train_first_order_bf16", "train", "bf16", 8, 32, 32, 16384, 128, 1, False, False),
        # one long context of 32 heads
        _case("train_long_bf16", "train", "bf16", 1, 32, 32, 262144, 64, 2, True, True),
        # the model's call site as the benchmark runs it: projection, rotary embedding, attention and back
        _case("site_bf16", "site", "bf16", 8, 32, 32, 4096, 64, 1, True, True),
        # serving: the prompts of four sequences enter their decode state
        _case("append_bf16", "append", "bf16", 4, 16, 16, 4000, 64, 2, True, True),
        # serving one sequence: a token through a state of grouped heads
        _case("step_small_bf16", "step", "bf16", 1, 32, 8, 100, 64, 2, True, True),
        # serving a batch of 64 sequences, the benchmark's decode configuration
        _case("step_bf16", "step", "bf16", 64, 16, 16, 50, 64, 2, True, True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "forward", "site", "append", "step"])
    dtype = rng.choice(["fp32", "bf16"])
    p, mask, normalize = rng.choice([1, 2, 2]), rng.random() < 0.6, True
    group = rng.choice([1, 1, 1, 2, 4])
    if kind == "append":
        d, n = rng.choice([64, 64, 128]), _log_int(rng, 33, 4096)
        most = (4_000_000 if p == 1 else 250_000) // (8 if d == 128 else 1)
        heads, mask = max(1, min(64, most // n)), True
    elif kind == "step":
        d, n, mask = rng.choice([64, 64, 128]), _log_int(rng, 8, 128), True
        heads = _log_int(rng, 4, 1024 if d == 64 else 160)
    else:
        if dtype == "fp32":
            d, n = rng.choice([32, 32, 64]), _log_int(rng, 100, 4096 if kind == "train" else 10000)
            most = 250_000 if d == 32 else 60_000
        else:
            d, n = rng.choice([64, 64, 128]), _log_int(rng, 100, 32768)
            most = 2_000_000 if d == 64 or p == 1 else 300_000
        if kind == "site":
            mask, n = True, min(n, 8192)
        heads = max(4, min(512, most // n, _log_int(rng, 4, 512)))
        normalize = mask or p == 2 or rng.random() < 0.5
    b = max(1, heads // 16) if heads >= 32 else 1
    h = max(group, heads // b // group * group)
    return {k: v for k, v in _case("", kind, dtype, b, h, h // group, n, d, p, mask, normalize).items() if k != "name"}


def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed))


def _inputs(case, seed):
    """q, k, v, upstream gradient ~ N(0,1); q and k are divided by sqrt(d) when nothing normalises them."""
    c, gen, dt = case, _gen(seed), DTYPES[case["dtype"]]
    s = 1.0 if c["normalize"] else c["d"] ** -0.5

    def make(heads, scale):
        t = torch.empty(c["b"], heads, c["n"], c["d"], dtype=dt, device="cuda")
        for i in range(c["b"]):
            t[i] = torch.randn(heads, c["n"], c["d"], generator=gen, device="cuda") * scale
        return t

    return make(c["h"], s), make(c["g"], s), make(c["g"], 1.0), make(c["h"], 1.0)


def _site_inputs(case, seed):
    """Packed projection ~ N(0,1), rotary tables of every other position scheme's usual base, gradient."""
    c, gen, dt = case, _gen(seed), DTYPES[case["dtype"]]
    width = (c["h"] + 2 * c["g"]) * c["d"]
    qkv = torch.randn(c["b"], c["n"], width, generator=gen, device="cuda").to(dt)
    go = torch.randn(c["b"], c["n"], c["h"] * c["d"], generator=gen, device="cuda").to(dt)
    theta = 10000.0 ** (-torch.arange(0, c["d"], 2, device="cuda", dtype=torch.float64) / c["d"])
    ang = torch.arange(c["n"], device="cuda", dtype=torch.float64)[:, None] * theta
    ang = torch.cat([ang, ang], 1)
    return qkv, go, ang.cos().float(), ang.sin().float()


def _decode_inputs(case, seed):
    """Keys and values of the prompt (bhkv, n, d), and the query, key and value of one more token."""
    c, gen, dt = case, _gen(seed), DTYPES[case["dtype"]]
    kv, bh = c["b"] * c["g"], c["b"] * c["h"]
    shapes = [(kv, c["n"], c["d"]), (kv, c["n"], c["d"]), (bh, 1, c["d"]), (kv, 1, c["d"]), (kv, 1, c["d"])]
    return [torch.randn(*s, generator=gen, device="cuda").to(dt) for s in shapes]


def prepare(case, seed):
    c = case
    if c["kind"] in ("train", "forward"):
        q, k, v, go = _inputs(c, seed)
        if c["kind"] == "train":
            q, k, v = [t.requires_grad_(True) for t in (q, k, v)]
        return dict(case=c, module=fastmax_b200.FASTMultiHeadAttention(), q=q, k=k, v=v,
                    go=go if c["kind"] == "train" else None)
    if c["kind"] == "site":
        qkv, go, cos, sin = _site_inputs(c, seed)
        return dict(case=c, qkv=qkv.requires_grad_(True), go=go, cos=cos, sin=sin)
    k, v, q1, k1, v1 = _decode_inputs(c, seed)
    st = fastmax_b200.FastmaxDecodeState(c["b"] * c["h"], c["b"] * c["g"], c["d"], dtype=DTYPES[c["dtype"]],
                                         device="cuda", normalize=c["normalize"], p=c["p"], **COEF)
    if c["kind"] == "append":
        return dict(case=c, decoder=st, k=k, v=v)
    st.append(k, v)
    return dict(case=c, decoder=st, q=q1, k=k1, v=v1)


def run(state):
    c = state["case"]
    if c["kind"] == "train":
        leaves = (state["q"], state["k"], state["v"])
        out = state["module"](*leaves, mask=c["mask"], normalize=c["normalize"], p=c["p"], **COEF)
        return (out,) + torch.autograd.grad(out, leaves, state["go"])
    if c["kind"] == "forward":
        with torch.no_grad():
            return state["module"](state["q"], state["k"], state["v"], mask=c["mask"], normalize=c["normalize"],
                                   p=c["p"], **COEF)
    if c["kind"] == "site":
        y = fastmax_b200.fastmax_attention_from_qkv(state["qkv"], state["cos"], state["sin"], c["h"], c["g"], c["d"],
                                                    c["d"], mask=c["mask"], normalize=c["normalize"], p=c["p"], **COEF)
        return (y,) + torch.autograd.grad(y, (state["qkv"],), state["go"])
    st = state["decoder"]
    if c["kind"] == "append":
        st.reset()
        st.append(state["k"], state["v"])
        return st.state
    return st.step(state["q"], state["k"], state["v"]), st.state


def work(case):
    """Inputs read once and outputs written once; the cheaper of the two evaluation orders of the path -- the
    score form (every query against its keys) and the factorised form (sums of key features, each unordered
    pair of features once, read by every query)."""
    c = case
    d, n, es = c["d"], c["n"], 2 if c["dtype"] == "bf16" else 4
    q, kv = c["b"] * c["h"], c["b"] * c["g"]
    feats = d + 1 + (d * (d + 1) // 2 if c["p"] == 2 else 0)
    if c["kind"] == "step":
        return dict(bytes=kv * 8 * feats * (d + 1) + es * d * (2 * q + 2 * kv), flops=2 * (q + kv) * feats * (d + 1))
    if c["kind"] == "append":
        return dict(bytes=4 * kv * feats * (d + 1) + 2 * es * kv * n * d, flops=2 * kv * n * feats * (d + 1))
    keys = (n + 1) / 2 if c["mask"] else n
    score, moment = 4.0 * keys * d, 4.0 * feats * (d + 1)
    # products of the score form: q.k and p.v forward; q.k, g.v and three more backward.  Factorised: one set of
    # sums and one read-out forward, one more set and two and a half read-outs backward.
    passes = 1.0 if c["kind"] == "forward" else 3.5
    tokens = es * d * n
    moved = tokens * (2 * q + 2 * kv)                    # q, k, v in, out back
    if c["kind"] != "forward":
        moved += tokens * (2 * q + 2 * kv)               # upstream gradient in, three gradients out
    return dict(bytes=moved, flops=passes * q * n * min(score, moment))


def tolerance(case):
    """fp32: sums of up to 10^4 terms in another order.  bf16: operands and results carry 8 bits."""
    if case["kind"] in ("append", "step"):
        # the state is fp32 whatever the inputs are; a step's row has the inputs' type
        return {"rel": 1e-5 if case["kind"] == "append" or case["dtype"] == "fp32" else 1e-2, "max": 0.5}
    return {"rel": 2e-5, "max": 0.5} if case["dtype"] == "fp32" else {"rel": 2e-2, "max": 0.9}


# ---- the same in float64 with plain torch ------------------------------------------------------------------

def _states(y, zt, p):
    """Sums over tokens of (zt, y zt, y y zt): (H, d+1), (H, d, d+1), (H, d*d, d+1)."""
    s0, s1 = zt.sum(1), y.transpose(1, 2) @ zt
    s2 = None
    if p == 2:
        y2 = (y.unsqueeze(3) * y.unsqueeze(2)).flatten(2)
        s2 = y2.transpose(1, 2) @ zt
    return [s0, s1, s2]


def _add(a, b):
    return b if a is None else [x if x is None else x + y for x, y in zip(a, b)]


def _read_a(x, st, p, a0, a1, a2):
    """sum_j f(x_i . y_j) zt_j from the sums over j."""
    r = a0 * st[0][:, None] + a1 * (x @ st[1])
    if p == 2:
        r = r + a2 * ((x.unsqueeze(3) * x.unsqueeze(2)).flatten(2) @ st[2])
    return r


def _read_b(x, ut, st, p, a1, a2):
    """sum_j f'(x_i . y_j) (ut_i . zt_j) y_j from the sums over j."""
    r = a1 * (ut @ st[1].transpose(1, 2))
    if p == 2:
        h, n, d = x.shape
        t = (ut @ st[2].transpose(1, 2)).view(h, n, d, d)
        r = r + 2 * a2 * (t @ x.unsqueeze(3)).squeeze(3)
    return r


def _attention64(q, k, v, go, mask, p, normalize, a0, a1, a2, lim):
    """out, grad_q, grad_k, grad_v in float64 for (H, n, d) inputs (gradients None without ``go``)."""
    heads, n, d = q.shape
    cq = lim / q.norm(dim=2).amax(1) if normalize else torch.ones(heads, dtype=q.dtype, device=q.device)
    ck = lim / k.norm(dim=2).amax(1) if normalize else torch.ones(heads, dtype=q.dtype, device=q.device)
    qh, kh = q * cq[:, None, None], k * ck[:, None, None]
    vt = torch.cat([v, v.new_ones(heads, n, 1)], 2)
    step = 512 if d <= 64 else 256
    cuts = [(lo, min(lo + step, n)) for lo in range(0, n, step)]

    def sums(y, zt, lo, hi):
        return _states(y[:, lo:hi], zt[:, lo:hi], p)

    def scores(x, y):
        s = x @ y.transpose(1, 2)
        return a0 + a1 * s + (a2 * s * s if p == 2 else 0), a1 + (2 * a2 * s if p == 2 else 0 * s)

    out, gq, gk, gv = torch.empty_like(q), None, None, None
    ut = None
    if go is not None:
        gq, gk, gv, ut = torch.empty_like(q), torch.empty_like(k), torch.empty_like(v), torch.empty_like(vt)
    st = None
    if not mask:
        for lo, hi in cuts:
            st = _add(st, sums(kh, vt, lo, hi))
    for lo, hi in cuts:                       # forward and grad_q, the sums of earlier tokens in hand
        x, num, low = qh[:, lo:hi], 0.0, None
        if st is not None:
            num = _read_a(x, st, p, a0, a1, a2)
        if mask:
            f, f1 = scores(x, kh[:, lo:hi])
            low = torch.ones(hi - lo, hi - lo, dtype=torch.bool, device=q.device).tril()
            num = num + f.masked_fill(~low, 0) @ vt[:, lo:hi]
        out[:, lo:hi] = num[..., :d] / num[..., d:]
        if go is not None:
            g = go[:, lo:hi]
            ut[:, lo:hi] = torch.cat([g, -(g * out[:, lo:hi]).sum(2, keepdim=True)], 2) / num[..., d:]
            r = _read_b(x, ut[:, lo:hi], st, p, a1, a2) if st is not None else 0.0
            if mask:
                e = (f1 * (ut[:, lo:hi] @ vt[:, lo:hi].transpose(1, 2))).masked_fill(~low, 0)
                r = r + e @ kh[:, lo:hi]
            gq[:, lo:hi] = r
        if mask:
            st = _add(st, sums(kh, vt, lo, hi))
    if go is None:
        return out, None, None, None
    st = None
    if not mask:
        for lo, hi in cuts:
            st = _add(st, sums(qh, ut, lo, hi))
    for lo, hi in reversed(cuts):             # grad_k and grad_v, the sums of later tokens in hand
        y, a, b = kh[:, lo:hi], 0.0, 0.0
        if st is not None:
            a, b = _read_b(y, vt[:, lo:hi], st, p, a1, a2), _read_a(y, st, p, a0, a1, a2)
        if mask:
            f, f1 = scores(qh[:, lo:hi], y)
            low = torch.ones(hi - lo, hi - lo, dtype=torch.bool, device=q.device).tril()
            e = (f1 * (ut[:, lo:hi] @ vt[:, lo:hi].transpose(1, 2))).masked_fill(~low, 0)
            a = a + e.transpose(1, 2) @ qh[:, lo:hi]
            b = b + f.masked_fill(~low, 0).transpose(1, 2) @ ut[:, lo:hi]
            st = _add(st, sums(qh, ut, lo, hi))
        gk[:, lo:hi], gv[:, lo:hi] = a, b[..., :d]
    for grad, x, c in ((gq, q, cq), (gk, k, ck)):
        grad *= c[:, None, None]
        if normalize:                         # the scale depends on the row of largest norm
            row = x.norm(dim=2).argmax(1)
            at = torch.arange(heads, device=q.device)
            top = x[at, row]
            grad[at, row] -= (grad * x).sum((1, 2))[:, None] * top / (top * top).sum(1, keepdim=True)
    return out, gq, gk, gv


def _grouped64(q, k, v, go, c):
    """``_attention64`` over (b, h, n, d) queries and (b, g, n, d) keys and values, some heads at a time."""
    b, h, n, d = q.shape
    g, r = k.shape[1], h // k.shape[1]
    q, k, v = q.reshape(b * h, n, d), k.reshape(b * g, n, d), v.reshape(b * g, n, d)
    go = None if go is None else go.reshape(b * h, n, d)
    wide = lambda t, s: t[s].double().repeat_interleave(r, 0)  # noqa: E731
    out = torch.empty(q.shape, dtype=torch.float64, device=q.device)
    grads = [torch.empty(t.shape, dtype=torch.float64, device=q.device) if go is not None else None
             for t in (q, k, v)]
    at_once = max(1, int(3e9 / (min(n, 512) * d * (d if c["p"] == 2 else 1) + n * d * 12)) // r)
    for lo in range(0, b * g, at_once):
        s, sq = slice(lo, lo + at_once), slice(lo * r, (lo + at_once) * r)
        o, gq, gk, gv = _attention64(q[sq].double(), wide(k, s), wide(v, s), None if go is None else go[sq].double(),
                                     c["mask"], c["p"], c["normalize"], **COEF)
        out[sq] = o
        if go is not None:
            grads[0][sq] = gq                 # the copies' normalisation terms add up to the shared head's
            grads[1][s], grads[2][s] = [t.view(-1, r, n, d).sum(1) for t in (gk, gv)]
    return [out.view(b, h, n, d)] + [None if t is None else t.view(b, -1, n, d) for t in grads]


def exact(case, seed):
    c = case
    if c["kind"] in ("train", "forward"):
        q, k, v, go = _inputs(c, seed)
        got = _grouped64(q, k, v, go if c["kind"] == "train" else None, c)
        return tuple(got) if c["kind"] == "train" else got[0]
    if c["kind"] == "site":
        qkv, go, cos, sin = _site_inputs(c, seed)
        return _site64(qkv, go, cos.double(), sin.double(), c)
    return _decode64(c, seed)


def _rotate(x, cos, sin, back=False):
    """Rotary embedding of (..., n, d) by halves, or its transpose."""
    half = x.shape[-1] // 2
    if back:
        y = x * sin
        return x * cos + torch.cat([y[..., half:], -y[..., :half]], -1)
    return x * cos + torch.cat([-x[..., half:], x[..., :half]], -1) * sin


def _site64(qkv, go, cos, sin, c):
    b, n, h, g, d = c["b"], c["n"], c["h"], c["g"], c["d"]
    r = h // g
    x = qkv.view(b, n, g, r + 2, d).permute(0, 2, 3, 1, 4).double()
    q = _rotate(x[:, :, :r], cos, sin).reshape(b, h, n, d)
    k, v = _rotate(x[:, :, r], cos, sin), x[:, :, r + 1]
    dout = go.view(b, n, h, d).transpose(1, 2).double()
    out, gq, gk, gv = _grouped64(q, k, v, dout, c)
    gx = torch.empty_like(x)
    gx[:, :, :r] = _rotate(gq.view(b, g, r, n, d), cos, sin, back=True)
    gx[:, :, r], gx[:, :, r + 1] = _rotate(gk, cos, sin, back=True), gv
    return out.transpose(1, 2).reshape(b, n, h * d), gx.permute(0, 3, 1, 2, 4).reshape(b, n, -1)


def _decode64(c, seed):
    """The decode state as float64 -- per key/value head the largest squared key norm, the token count as the
    bits of an integer, two spare words, then the second-order, first-order and constant rows -- and a step's row."""
    k, v, q1, k1, v1 = _decode_inputs(c, seed)
    if c["kind"] == "step":
        k, v = torch.cat([k, k1], 1), torch.cat([v, v1], 1)
    kv, n, d = k.shape
    p = c["p"]
    rows = d + 1 + (d * d if p == 2 else 0)
    state = torch.zeros(kv, 4 + rows * (d + 1), dtype=torch.float64, device="cuda")
    out = torch.empty(c["b"] * c["h"], 1, d, dtype=torch.float64, device="cuda")
    r = c["h"] // c["g"]
    count = torch.tensor([n], dtype=torch.int32).view(torch.float32).double().item()
    for h in range(kv):
        kd, vt = k[h:h + 1].double(), torch.cat([v[h].double(), torch.ones(n, 1, dtype=torch.float64, device="cuda")], 1)[None]
        st = None
        for lo in range(0, n, 1024):
            st = _add(st, _states(kd[:, lo:lo + 1024], vt[:, lo:lo + 1024], p))
        top = (kd * kd).sum(2).max()
        state[h, 0], state[h, 1] = top, count
        state[h, 4:] = torch.cat([s.reshape(-1) for s in ([st[2]] if p == 2 else []) + [st[1], st[0]]])
        if c["kind"] == "step":
            q = q1[h * r:(h + 1) * r, 0].double()[None]
            sc = COEF["lim"] / top.sqrt() if c["normalize"] else 1.0
            if c["normalize"]:
                q = COEF["lim"] * q / q.norm(dim=2, keepdim=True)
            num = _read_a(q * sc, st, p, COEF["a0"], COEF["a1"], COEF["a2"])[0]
            out[h * r:(h + 1) * r, 0] = num[:, :d] / num[:, d:]
    return (out, state.view(-1)) if c["kind"] == "step" else state.view(-1)
