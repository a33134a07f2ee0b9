"""Performance cases: what a program built on this package has it do, through its public entry points.

The path is the 8-bit inference of a video DiT block (hidden 2048 = 32 heads x 64, FFN 8192, 6144 video
tokens per clip, 128 text tokens), its text encoder's FP8 linears (4096 / 10240), and the frozen-weight
training side (activation gradients, low-rank adapters).  Every case is a dict with a ``kind``:

* ``linear``   one quantised linear (``q8_linear`` / ``fp8_linear``) on bf16 activations, or on rows that
               the program already quantised (``ready``)
* ``attn``     ``flash_attn_func`` on bf16 q, k, v, self- or masked cross-attention
* ``block``    one ``LTXTransformerBlock`` forward
* ``grad``     forward and backward of a frozen INT8 linear; with ``rank`` the low-rank adapter module
* ``norm``     RMS norm + rotary embedding of a projection, forward and backward
"""
import math

import torch

from q8_kernels_b200.blocks import LTXTransformerBlock
from q8_kernels_b200.functional.flash_attention import flash_attn_func
from q8_kernels_b200.functional.linear import fp8_linear, q8_linear
from q8_kernels_b200.functional.rms_norm import rms_norm_8bit
from q8_kernels_b200.functional.rope import apply_rope
from q8_kernels_b200.modules import Q8LinearLora

BF16 = torch.bfloat16
E4M3 = torch.float8_e4m3fn


# ------------------------------------------------------------------------------------------ the cases

def _linear(name, dtype, batch, tokens, k, n, gelu=False, rotate=True, ready=False):
    return {"name": name, "kind": "linear", "dtype": dtype, "batch": batch, "tokens": tokens, "k": k, "n": n,
            "gelu": gelu, "rotate": rotate, "ready": ready}


def listed():
    return [
        # key (or value) projection of a cross-attention: 128 text tokens, the smallest linear of a block
        _linear("text_kv_int8", "int8", 1, 128, 2048, 2048),
        # text encoder, FFN up-projection of one odd-length prompt: FP8 without rotation, weights dominate
        _linear("encoder_up_fp8", "fp8", 1, 77, 4096, 10240, rotate=False),
        # FFN up-projection with its fused GELU over four clips: the largest activation of a block
        _linear("ffn_up_int8_gelu", "int8", 4, 6144, 2048, 8192, gelu=True),
        # FFN down-projection of one clip with rotated FP8 activations: the longest contraction
        _linear("ffn_down_fp8", "fp8", 1, 6144, 8192, 2048),
        # stacked Q/K/V projection over four clips of rows that a fused producer has quantised: the bare GEMM
        _linear("qkv_fp8_ready", "fp8", 1, 24576, 2048, 6144, ready=True),
        # self-attention of two clips with the Hadamard rotation of q and k
        {"name": "self_attn", "kind": "attn", "batch": 2, "heads": 32, "sq": 6144, "skv": 6144, "rotate": True,
         "masked": False, "out": "bf16"},
        # cross-attention on up to 128 text tokens, per-clip key lengths
        {"name": "cross_attn", "kind": "attn", "batch": 2, "heads": 32, "sq": 6144, "skv": 128, "rotate": True,
         "masked": True, "out": "e4m3"},
        # one block of the stack on one clip
        {"name": "block_int8", "kind": "block", "dtype": "int8", "batch": 1, "tokens": 6144, "text": 128, "heads": 32},
        # one block on two short low-resolution clips of odd length with FP8 linears: latency and tails
        {"name": "block_fp8_short", "kind": "block", "dtype": "fp8", "batch": 2, "tokens": 1001, "text": 77, "heads": 32},
        # fine-tuning through a frozen INT8 projection: output and activation gradient
        {"name": "frozen_grad", "kind": "grad", "batch": 1, "tokens": 6144, "k": 2048, "n": 2048, "rank": 0},
        # adapter training step on a short odd-length clip: output, activation and adapter gradients
        {"name": "lora_grad", "kind": "grad", "batch": 2, "tokens": 1001, "k": 2048, "n": 2048, "rank": 16},
        # q/k norm and rotary embedding of one clip as separate ops, forward and backward
        {"name": "norm_rope_grad", "kind": "norm", "batch": 1, "tokens": 6144, "heads": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "linear", "attn", "attn", "block", "grad", "norm"])
    if kind == "linear":
        dtype = rng.choice(["int8", "fp8"])
        ready = rng.random() < 0.25
        k = 16 * _log_int(rng, 32, 512) if rng.random() < 0.5 else rng.choice([1024, 2048, 4096, 8192])
        n = 16 * _log_int(rng, 16, 640) if rng.random() < 0.5 else rng.choice([2048, 6144, 8192, 10240])
        batch = rng.choice([1, 1, 2])
        tokens = min(_log_int(rng, 1, 6144), 2 ** 38 // (batch * k * n))    # no more work than the listed FFN up-projection
        return {"kind": "linear", "dtype": dtype, "batch": batch, "tokens": tokens, "k": k, "n": n,
                "gelu": dtype == "int8" and rng.random() < 0.5,
                "rotate": dtype == "int8" or rng.random() < 0.5, "ready": ready}
    if kind == "attn":
        cross = rng.random() < 0.5
        return {"kind": "attn", "batch": rng.choice([1, 2]), "heads": rng.choice([4, 8, 16, 20, 32]),
                "sq": _log_int(rng, 64, 6144), "skv": rng.randint(16, 256) if cross else _log_int(rng, 64, 6144),
                "rotate": rng.random() < 0.7, "masked": cross, "out": rng.choice(["bf16", "e4m3"])}
    if kind == "block":
        return {"kind": "block", "dtype": rng.choice(["int8", "fp8"]), "batch": rng.choice([1, 2]),
                "tokens": _log_int(rng, 64, 3072), "text": rng.randint(16, 160), "heads": rng.choice([8, 16, 32])}
    if kind == "grad":
        return {"kind": "grad", "batch": rng.choice([1, 2]), "tokens": _log_int(rng, 16, 3072),
                "k": rng.choice([1024, 2048]), "n": rng.choice([1024, 2048, 4096, 8192]), "rank": rng.choice([0, 8, 16, 32])}
    return {"kind": "norm", "batch": rng.choice([1, 2]), "tokens": _log_int(rng, 16, 6144), "heads": rng.choice([8, 16, 24, 32, 64])}


# ------------------------------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def _activations(g, *shape):
    """~N(0,1) with 0.1 % of the channels twenty times as large, as DiT activations have them."""
    x = _randn(g, *shape)
    n = max(1, math.ceil(0.001 * shape[-1]))
    x[..., torch.randperm(shape[-1], generator=g, device="cuda")[:n]] *= 20.0
    return x.to(BF16)


def _quantised(x, dtype):
    """Rows of x as int8 or e4m3 values with one fp32 scale each (what a checkpoint or a producer holds)."""
    x = x.float()
    amax = x.abs().amax(dim=-1)
    top = 127.0 if dtype == "int8" else 448.0
    q = x * (top / amax).unsqueeze(-1)
    return (q.round().clamp(-127, 127).to(torch.int8) if dtype == "int8" else q.to(E4M3)), amax / top


def _weight(g, n, k, dtype):
    return _quantised(_randn(g, n, k) * 0.02, dtype)


def _linear_inputs(c, seed):
    g = _gen(seed)
    x = _activations(g, c["batch"], c["tokens"], c["k"])
    w, ws = _weight(g, c["n"], c["k"], c["dtype"])
    s = {"x": x, "xs": None, "w": w, "ws": ws, "bias": _randn(g, c["n"]) * 0.02}
    if c["ready"]:
        s["x"], s["xs"] = _quantised(x, c["dtype"])
    return s


def _attn_inputs(c, seed):
    g = _gen(seed)
    b, h = c["batch"], c["heads"]

    def heads(x):
        return x.view(b, -1, h, 64).transpose(1, 2)

    s = {"q": heads(_activations(g, b, c["sq"], h * 64)), "k": heads(_activations(g, b, c["skv"], h * 64)),
         "v": heads(_randn(g, b, c["skv"], h * 64).to(BF16)), "lens": None}
    if c["masked"]:
        s["lens"] = torch.randint(min(16, c["skv"]), c["skv"] + 1, (b,), generator=g, device="cuda").int()
    return s


def _rotary(tokens, dim):
    """cos / sin rows of an interleaved-pair rotary embedding, [1, tokens, dim] fp32."""
    freq = 10000.0 ** (-torch.arange(dim // 2, device="cuda", dtype=torch.float64) / (dim // 2))
    angle = (torch.arange(tokens, device="cuda", dtype=torch.float64).unsqueeze(-1) * freq).repeat_interleave(2, dim=-1)
    return angle.cos().float().unsqueeze(0), angle.sin().float().unsqueeze(0)


def _block_linears(dim):
    out = []
    for a in ("attn1", "attn2"):
        out += [("%s.%s" % (a, p), dim, dim) for p in ("to_q", "to_k", "to_v", "to_out")]
    return out + [("ff.act.proj", 4 * dim, dim), ("ff.proj_down", dim, 4 * dim)]


def _block_inputs(c, seed):
    g = _gen(seed)
    b, dim = c["batch"], c["heads"] * 64
    p = {}
    for name, n, k in _block_linears(dim):
        p[name + ".weight"], p[name + ".scales"] = _weight(g, n, k, c["dtype"])
        p[name + ".bias"] = _randn(g, n) * 0.02
    for a in ("attn1", "attn2"):
        for m in ("q_norm", "k_norm"):
            p["%s.%s.weight" % (a, m)] = 1.0 + 0.1 * _randn(g, dim)
    p["scale_shift_table"] = (_randn(g, 6, dim) / dim ** 0.5).to(BF16)
    return {"params": p, "x": _activations(g, b, c["tokens"], dim), "text": _randn(g, b, c["text"], dim).to(BF16),
            "lens": torch.randint(min(16, c["text"]), c["text"] + 1, (b,), generator=g, device="cuda").int(),
            "time": (0.3 * _randn(g, b, 1, 6 * dim)).to(BF16), "freqs": _rotary(c["tokens"], dim)}


def _grad_inputs(c, seed):
    g = _gen(seed)
    w, ws = _weight(g, c["n"], c["k"], "int8")
    s = {"x": _activations(g, c["batch"], c["tokens"], c["k"]), "w": w, "ws": ws, "bias": _randn(g, c["n"]) * 0.02,
         "g": (_randn(g, c["batch"], c["tokens"], c["n"]) * 0.1).to(BF16)}
    if c["rank"]:
        s["a"] = (_randn(g, c["rank"], c["k"]) / c["rank"]).to(BF16)
        s["b"] = (_randn(g, c["n"], c["rank"]) * 0.02).to(BF16)
    return s


def _norm_inputs(c, seed):
    g = _gen(seed)
    dim = c["heads"] * 64
    cos, sin = _rotary(c["tokens"], dim)
    return {"x": _activations(g, c["batch"], c["tokens"], dim), "w": 1.0 + 0.1 * _randn(g, dim), "cos": cos, "sin": sin,
            "g": (_randn(g, c["batch"], c["tokens"], dim) * 0.1).to(BF16)}


# ------------------------------------------------------------------------------------------ the path

def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        s = _linear_inputs(case, seed)
    elif kind == "attn":
        s = _attn_inputs(case, seed)
    elif kind == "norm":
        s = _norm_inputs(case, seed)
        s["x"].requires_grad_(True)
    elif kind == "grad":
        s = _grad_inputs(case, seed)
        s["x"].requires_grad_(True)
        if case["rank"]:
            m = Q8LinearLora(case["k"], case["n"], case["rank"], device="cuda")
            m.weight.data, m.scales.data, m.bias.data = s["w"], s["ws"], s["bias"]
            m.lora_a.data, m.lora_b.data = s["a"], s["b"]
            s["module"] = m
    else:
        s = _block_inputs(case, seed)
        dim = case["heads"] * 64
        m = LTXTransformerBlock(dim, case["heads"], 64, dim, linear=case["dtype"]).cuda()
        own = dict(m.named_parameters())
        own.update(dict(m.named_buffers()))
        for name, value in s.pop("params").items():
            own[name].data = value
        s["module"] = m
    s["case"] = case
    return s


def run(state):
    c = state["case"]
    if c["kind"] == "linear":
        with torch.no_grad():
            if c["dtype"] == "int8":
                return q8_linear(state["x"], state["w"], state["bias"], state["xs"], state["ws"], c["gelu"], BF16)
            return fp8_linear(state["x"], state["w"], state["bias"], state["xs"], state["ws"], c["rotate"], BF16)
    if c["kind"] == "attn":
        with torch.no_grad():
            return flash_attn_func(state["q"], state["k"], state["v"], batch_mask=state["lens"],
                                   apply_qk_hadamard=c["rotate"], out_dtype=BF16 if c["out"] == "bf16" else None)
    if c["kind"] == "block":
        with torch.no_grad():
            return state["module"](state["x"], state["freqs"], None, state["text"], state["lens"], state["time"])
    if c["kind"] == "norm":
        y = apply_rope(rms_norm_8bit(state["x"], state["w"], BF16), state["cos"], state["sin"], BF16)
        return y.detach(), torch.autograd.grad(y, [state["x"]], state["g"])[0]
    if c["rank"]:
        m = state["module"]
        y = m(state["x"], out_dtype=BF16)
        return (y.detach(),) + tuple(torch.autograd.grad(y, [state["x"], m.lora_a, m.lora_b], state["g"]))
    y = q8_linear(state["x"], state["w"], state["bias"], None, state["ws"], False, BF16)
    return y.detach(), torch.autograd.grad(y, [state["x"]], state["g"])[0]


# ------------------------------------------------------------------------------------------ what it takes

def _linear_work(m, n, k, x_bytes=2, out_bytes=2):
    return {"bytes": m * k * x_bytes + n * k + m * n * out_bytes + 8 * n, "flops": 2 * m * n * k}


def work(case):
    if case["kind"] == "linear":
        return _linear_work(case["batch"] * case["tokens"], case["n"], case["k"], 1 if case["ready"] else 2)
    if case["kind"] == "attn":
        bh = case["batch"] * case["heads"]
        keys = (min(16, case["skv"]) + case["skv"]) / 2 if case["masked"] else case["skv"]   # mean of the key lengths
        return {"bytes": int(bh * 64 * (case["sq"] * (4 if case["out"] == "bf16" else 3) + 4 * keys)),
                "flops": int(4 * bh * case["sq"] * keys * 64)}
    if case["kind"] == "block":
        dim, m, t = case["heads"] * 64, case["batch"] * case["tokens"], case["batch"] * case["text"]
        keys = (min(16, case["text"]) + case["text"]) / 2
        flops = 2 * m * dim * dim * (6 + 8) + 2 * t * dim * dim * 2 + 4 * m * dim * (case["tokens"] + keys)
        return {"bytes": int(m * dim * 4 + t * dim * 2 + 16 * dim * dim + case["tokens"] * dim * 8), "flops": int(flops)}
    m = case["batch"] * case["tokens"]
    if case["kind"] == "norm":
        dim = case["heads"] * 64
        return {"bytes": m * dim * 8 + case["tokens"] * dim * 8 + 4 * dim, "flops": 30 * m * dim}
    n, k, r = case["n"], case["k"], case["rank"]
    return {"bytes": m * (4 * k + 4 * n) + n * k + 4 * r * (n + k), "flops": 4 * m * n * k + 10 * m * r * (n + k)}


def tolerance(case):
    # The difference of two correct implementations: one step of the 16-bit (or e4m3) result where sums are
    # taken in another order, and now and then one 8-bit step of an operand that sits on a rounding boundary.
    # Each is about four times the distance to exact() (linear 1.7e-3, e4m3 attention 2.8e-2 at most with e4m3 results,
    # gradients 3e-3, norm and rotation 2.3e-3); twice where that distance is the 8-bit probabilities' own
    # (attention 1.1e-2 with bf16 results) or a chain of 8-bit operands (block 1.8e-2).
    if case["kind"] == "linear":
        return {"rel": 7e-3}
    if case["kind"] == "attn":
        return {"rel": 2e-2 if case["out"] == "bf16" else 6e-2}
    if case["kind"] == "block":
        return {"rel": 4e-2}
    if case["kind"] == "grad":
        return {"rel": 1.2e-2}
    return {"rel": 1e-2}


# ------------------------------------------------------------------------------------------ in 64 bits

def _round(x, dtype=BF16):
    return x.to(dtype).double()


def _rotated(x, scale):
    """Sylvester-Hadamard transform of the last dim, zero-padded to a power of two, times scale."""
    d = x.shape[-1]
    n = 1 << (d - 1).bit_length()
    y = torch.nn.functional.pad(x, (0, n - d)).reshape(-1, n)
    s = 1
    while s < n:
        y = y.view(-1, n // (2 * s), 2, s)
        y = torch.stack((y[:, :, 0] + y[:, :, 1], y[:, :, 0] - y[:, :, 1]), dim=2)
        s *= 2
    return (y.reshape(-1, n)[:, :d] * scale).reshape(x.shape)


def _rows8(x, dtype):
    """Per-row quantisation: the 8-bit values as doubles, and the row scales."""
    top = 127.0 if dtype == "int8" else 448.0
    amax = x.abs().amax(dim=-1, keepdim=True)
    q = x * (top / amax)
    q = torch.trunc(q + torch.copysign(torch.full_like(q, 0.5), q)) if dtype == "int8" else q.float().to(E4M3).double()
    return q, amax / top


def _linear64(x, w, ws, bias, dtype, rotate=True, gelu=False):
    """x: double rows holding what the activation tensor holds."""
    if rotate:
        x = _round(_rotated(x, x.shape[-1] ** -0.5))
    q, s = _rows8(x, dtype)
    y = (q @ w.double().T) * s * ws.double() + (0.0 if bias is None else bias.double())
    return torch.nn.functional.gelu(y, approximate="tanh") if gelu else y


def _attention64(q, k, v, lens, scale):
    """q, k, v: doubles [B,H,S,64] holding e4m3 values."""
    out = torch.empty_like(q)
    for b in range(q.shape[0]):
        n = k.shape[2] if lens is None else int(lens[b])
        for h in range(q.shape[1]):
            p = torch.softmax((q[b, h] @ k[b, h, :n].T) * scale, dim=-1)
            out[b, h] = p @ v[b, h, :n]
    return out


def _heads8(x, rotate):
    x = x.double()
    return _round((_rotated(x, 0.125 * 8.0 ** -0.5) if rotate else x).float(), E4M3)


def _rms64(x, w):
    y = x * torch.rsqrt((x * x).mean(dim=-1, keepdim=True))
    return y if w is None else y * w.double()


def _swap(x):
    """(a, b) -> (-b, a) for every pair of channels."""
    p = x.unflatten(-1, (-1, 2))
    return torch.stack((-p[..., 1], p[..., 0]), dim=-1).flatten(-2)


def _attn_module64(s, name, x, kv, heads, dtype, freqs, lens):
    p = s["params"]

    def lin(part, t):
        f = "%s.%s." % (name, part)
        return _linear64(t, p[f + "weight"], p[f + "scales"], p[f + "bias"], dtype)

    q, k, v = _round(lin("to_q", x)), _round(lin("to_k", kv)), _round(lin("to_v", kv))
    q, k = _rms64(q, p[name + ".q_norm.weight"]), _rms64(k, p[name + ".k_norm.weight"])
    if freqs is not None:
        cos, sin = freqs[0].double(), freqs[1].double()
        q, k = q * cos + _swap(q) * sin, k * cos + _swap(k) * sin

    def split(t):
        return t.unflatten(-1, (heads, 64)).transpose(1, 2)

    o = _attention64(_heads8(split(q), True), _heads8(split(k), True), _heads8(split(v), False), lens, 1.0)
    o = _round(o.transpose(1, 2).flatten(2).float(), E4M3)
    # the e4m3 attention output is rotated in e4m3, the type it is held in
    d = o.shape[-1]
    y = _round(_rotated(o, d ** -0.5).float(), E4M3)
    f = name + ".to_out."
    return _linear64(y, p[f + "weight"], p[f + "scales"], p[f + "bias"], dtype, rotate=False)


def _block64(c, seed):
    s = _block_inputs(c, seed)
    p, x, dt = s["params"], s["x"].double(), c["dtype"]
    ada = _round(p["scale_shift_table"].double() + s["time"].double().view(c["batch"], 1, 6, -1))
    shift1, scale1, gate1, shift2, scale2, gate2 = ada.unbind(dim=2)
    h = _round(_rms64(x, None) * (1 + scale1) + shift1)
    x = _round(x + gate1 * _attn_module64(s, "attn1", h, h, c["heads"], dt, s["freqs"], None))
    x = _round(x + _attn_module64(s, "attn2", x, s["text"].double(), c["heads"], dt, None, s["lens"]))
    h = _round(_rms64(x, None) * (1 + scale2) + shift2)
    u = _round(_linear64(h, p["ff.act.proj.weight"], p["ff.act.proj.scales"], p["ff.act.proj.bias"], dt, gelu=True))
    return x + gate2 * _linear64(u, p["ff.proj_down.weight"], p["ff.proj_down.scales"], p["ff.proj_down.bias"], dt)


def _grad64(c, seed):
    s = _grad_inputs(c, seed)
    x, g, w, ws = s["x"].double(), s["g"].double(), s["w"].double(), s["ws"].double()
    y = _linear64(x, s["w"], s["ws"], s["bias"], "int8")
    gq, gs = _rows8(g, "fp8")
    k = c["k"]
    if not c["rank"]:
        wq, wsc = _rows8((w * ws.unsqueeze(-1)).T, "fp8")
        return y, _rotated(_round((gq @ wq.T) * gs * wsc.squeeze(-1)), k ** -0.5)
    a, b = s["a"].double(), s["b"].double()
    wr = _round(_rotated(_round(w * ws.unsqueeze(-1)), k ** -0.5))
    wq, wsc = _rows8(wr.T, "fp8")
    low = (x @ a.T)
    y = y + low @ b.T
    gb = g @ b
    gx = (gq @ wq.T) * gs * wsc.squeeze(-1) + gb @ a
    return y, gx, (gb.flatten(0, 1).T @ x.flatten(0, 1)), (g.flatten(0, 1).T @ low.flatten(0, 1))


def _norm64(c, seed):
    s = _norm_inputs(c, seed)
    x, w, cos, sin, g = (s[n].double() for n in ("x", "w", "cos", "sin", "g"))
    n = _rms64(x, w)
    gn = g * cos - _swap(g * sin)                       # transposed rotation
    r = torch.rsqrt((x * x).mean(dim=-1, keepdim=True))
    gw = gn * w
    return n * cos + _swap(n) * sin, r * (gw - x * r * r * (gw * x).mean(dim=-1, keepdim=True))


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "linear":
            s = _linear_inputs(case, seed)
            if case["ready"]:
                y = ((s["x"].double() @ s["w"].double().T) * s["xs"].double().unsqueeze(-1) * s["ws"].double()
                     + s["bias"].double())
                return torch.nn.functional.gelu(y, approximate="tanh") if case["gelu"] else y
            return _linear64(s["x"].double(), s["w"], s["ws"], s["bias"], case["dtype"], case["rotate"], case["gelu"])
        if case["kind"] == "attn":
            s = _attn_inputs(case, seed)
            q, k, v = _heads8(s["q"], case["rotate"]), _heads8(s["k"], case["rotate"]), _heads8(s["v"], False)
            return _attention64(q, k, v, s["lens"], 1.0 if case["rotate"] else 0.125)
        if case["kind"] == "block":
            return _block64(case, seed)
        if case["kind"] == "grad":
            return _grad64(case, seed)
        return _norm64(case, seed)
