"""What the library's speed is judged on: calls of its public entry points over the sizes that its users have.

Every case is one pass of a kind of work:

  matvec   a quantised matvec with host vectors, one call that returns the result (``q4_matvec`` / ``q8_matvec``)
  linear   quantised linear layers over device buffers, a recorded run over distinct matrices (decode rows) or one call
           (many rows)
  decode   one decode step of the Llama-shaped model, replayed from a graph as ``generate`` does
  prefill  one chunk of prompt tokens through the same model
  moe      one mixture-of-experts layer (router, routed and shared experts)
  mla      one decode step of the latent attention layer (projections, rotation, attention, output projection)
  tofazen  the dense bf16 family: prompts of different lengths in one ragged step, or a decode step over them

Shapes are those of bench.py and the tests: Llama-3-8B-shaped and "1b", DeepSeek-V2-Lite-shaped experts,
DeepSeek-V3-shaped latent attention.  Weights are random, quantised from normal values; caches are normal; everything
follows from the seed.  ``exact`` computes the same from the same inputs in 64 bits with torch alone.
"""
import math

import numpy as np
import torch

import tang_b200 as tb
from tang_b200.tofazen import TofazenConfig, TofazenLayer, TofazenModel, tensor_names

KINDS = {"q4_f32": tb.Q4_F32, "q4_f16": tb.Q4_F16, "q8_f32": tb.Q8_F32, "i8_row": tb.I8_ROW}
LLAMA = {  # layers, width, heads, kv heads, head size, ffn, vocabulary
    "8b": (32, 4096, 32, 8, 128, 14336, 128256),
    "1b": (16, 2048, 16, 4, 128, 8192, 32000),
}
TOFAZEN = {  # layers, width, heads, kv heads, size of a map's head, value size, ff, vocabulary
    "1b": (16, 2048, 16, 4, 64, 128, 8192, 32000),
}
MOE = (2048, 1408, 64, 6, 2)            # width, expert ffn, experts, chosen, shared
MLA = (7168, 1536, 512, 128, 64, 128)   # width, query rank, latent, nope, rope, value size
EPS, ROPE_BASE, MLA_BASE = 1e-5, 500000.0, 10000.0


def listed():
    return [
        # the smallest call there is: one matvec of the reference's benchmark size with host vectors; all latency
        {"name": "matvec_q8_576", "path": "matvec", "kind": "q8_f32", "rows": 576, "cols": 576},
        # the up projection of one decoded token, eight layers' worth (more than L2 holds); memory bound
        {"name": "linear_q4_m1", "path": "linear", "kind": "q4_f16", "rows": 14336, "cols": 4096, "m": 1, "layers": 8, "x": "bf16", "y": "bf16"},
        # the same projection over a prompt chunk; tensor bound
        {"name": "linear_q4_m2048", "path": "linear", "kind": "q4_f16", "rows": 14336, "cols": 4096, "m": 2048, "layers": 1, "x": "bf16", "y": "bf16"},
        # a single user's decode step: latency of the chain of layers
        {"name": "decode_8b_b1", "path": "decode", "size": "8b", "batch": 1, "ctx": 2048},
        # a small server's decode step, contexts of different lengths
        {"name": "decode_8b_b16", "path": "decode", "size": "8b", "batch": 16, "ctx": 2048},
        # the largest batch the model takes: caches weigh more than weights
        {"name": "decode_8b_b64", "path": "decode", "size": "8b", "batch": 64, "ctx": 2048},
        # a prompt of 2048 tokens
        {"name": "prefill_8b_2048", "path": "prefill", "size": "8b", "batch": 1, "q_len": 2048, "start": 0},
        # a decode batch through an expert layer: every expert gets a few rows
        {"name": "moe_64", "path": "moe", "tokens": 64, "renorm": False},
        # a prompt chunk through an expert layer
        {"name": "moe_4096", "path": "moe", "tokens": 4096, "renorm": False},
        # latent attention for a single user, and for a batch at a long context
        {"name": "mla_4096_b1", "path": "mla", "heads": 128, "batch": 1, "ctx": 4096},
        {"name": "mla_16384_b16", "path": "mla", "heads": 128, "batch": 16, "ctx": 16384},
        # the dense family: four prompts of different lengths in one step, window of 512 with four kept tokens
        {"name": "tofazen_1b_prompts", "path": "tofazen", "size": "1b", "seqs": 4, "longest": 1024, "decode": False, "window": 512, "keep": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: the kind of work as often as it is listed, sizes over its whole range."""
    path = rng.choice(["matvec"] + ["linear"] * 2 + ["decode"] * 3 + ["prefill"] + ["moe"] * 2 + ["mla"] * 2 + ["tofazen"])
    if path == "matvec":
        return {"path": path, "kind": rng.choice(["q4_f32", "q8_f32"]), "rows": _log(rng, 64, 4096), "cols": 32 * _log(rng, 4, 128)}
    if path == "linear":
        m = _log(rng, 1, 2048)
        odd = rng.random() < 0.25   # widths that are no multiple of the kernels' tiles
        rows = _log(rng, 512, 14336) if odd else 128 * _log(rng, 4, 112)
        return {"path": path, "kind": rng.choice(list(KINDS)), "rows": rows, "cols": 64 * _log(rng, 8, 224) if odd else 128 * _log(rng, 4, 112), "m": m,
                "layers": 8 if m <= 64 else 1, "x": "f32" if m <= 64 and rng.random() < 0.2 else "bf16", "y": rng.choice(["bf16", "f32"])}
    if path == "decode":
        return {"path": path, "size": rng.choice(["8b", "1b"]), "batch": _log(rng, 1, 64), "ctx": _log(rng, 64, 2048)}
    if path == "prefill":
        batch = rng.choice([1, 1, 2, 3])
        return {"path": path, "size": rng.choice(["8b", "1b"]), "batch": batch, "q_len": max(2, _log(rng, 16, 2048) // batch), "start": rng.choice([0, 0, rng.randrange(1, 1024)])}
    if path == "moe":
        return {"path": path, "tokens": _log(rng, 1, 4096), "renorm": rng.random() < 0.5}
    if path == "mla":
        return {"path": path, "heads": rng.choice([128, 128, 64, 32, 16]), "batch": _log(rng, 1, 64), "ctx": _log(rng, 256, 32768)}
    return {"path": path, "size": "1b", "seqs": rng.randrange(1, 9), "longest": _log(rng, 16, 1024), "decode": rng.random() < 0.5, **rng.choice(
        [{"window": 512, "keep": 4}, {"window": 4096, "keep": 0}, {"window": 128, "keep": 0}])}


# ---------------------------------------------------------------------------------------------- inputs
_device = None


def device():
    """The program's one device handle (one stream, one set of workspaces)."""
    global _device
    if _device is None:
        _device = tb.QuantComputeDevice(0)
    return _device


def _gen(seed, tag):
    return torch.Generator(device="cuda").manual_seed(seed * 1000003 + tag)


def normal(seed, tag, shape, std=1.0, mean=0.0):
    """bf16 normal values."""
    return (torch.randn(shape, device="cuda", generator=_gen(seed, tag)) * std + mean).bfloat16()


def quantised(seed, tag, kind, rows, cols, std=None):
    """(payload, scales) of normal weights (std 1 / sqrt(cols)) in the layout of ``qweight_from_device``."""
    g, std = _gen(seed, tag), cols ** -0.5 if std is None else std
    pay, sc = [], []
    step = max(1, (1 << 27) // cols)
    for r in range(0, rows, step):
        w = torch.randn((min(step, rows - r), cols), device="cuda", generator=g) * std
        if kind == "i8_row":
            s = w.abs().amax(1, keepdim=True) / 127
            pay.append((w / s).round_().to(torch.int8))
            sc.append(s[:, 0])
            continue
        w = w.view(w.shape[0], cols // 32, 32)
        s = w.abs().amax(2, keepdim=True) / (127 if kind == "q8_f32" else 7)
        s = s.half() if kind == "q4_f16" else s
        q = (w / s.float()).round_()
        if kind == "q8_f32":
            pay.append(q.clamp_(-127, 127).to(torch.int8).view(-1, cols))
        else:
            q = q.clamp_(-8, 7).add_(8).to(torch.uint8).view(-1, cols // 2, 2)
            pay.append(q[:, :, 0] | (q[:, :, 1] << 4))
        sc.append(s[:, :, 0])
    return torch.cat(pay), torch.cat(sc)


def dequantised(kind, pay, sc):
    """The weights that (payload, scales) stand for, in 64 bits."""
    if kind == "i8_row":
        return pay.double() * sc.double()[:, None]
    if kind != "q8_f32":
        pay = torch.stack((pay & 15, pay >> 4), 2).view(pay.shape[0], -1).to(torch.int8) - 8
    return (pay.view(pay.shape[0], -1, 32).double() * sc.double()[:, :, None]).view(pay.shape[0], -1)


def qweight(seed, tag, kind, rows, cols, std=None):
    dev = device()
    pay, sc = quantised(seed, tag, kind, rows, cols, std)
    torch.cuda.synchronize()
    w = dev.qweight_from_device(KINDS[kind], pay.data_ptr(), sc.data_ptr(), rows, cols)
    dev.sync()
    return w


def buf(t):
    """A torch tensor's memory as the library sees it."""
    return tb.Buffer(device(), t.data_ptr(), t.numel(), {torch.bfloat16: tb.BF16, torch.float32: tb.F32, torch.int32: tb.I32}[t.dtype], owns=False)


class Owner:
    """Destroys a model when neither a state nor a view of its memory is left."""

    def __init__(self, model):
        self.model = model

    def __del__(self):
        try:
            device().sync()
            self.model.destroy()
        except Exception:
            pass


class _Memory:
    def __init__(self, owner, ptr, shape, strides):
        self.owner = owner   # a tensor made of this object keeps it, and so the memory, alive
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": tuple(shape), "strides": tuple(2 * s for s in strides), "typestr": "<i2", "version": 3}


def view(owner, ptr, shape, strides):
    """Device memory of the owner's model, as a bf16 tensor."""
    return torch.as_tensor(_Memory(owner, ptr, shape, strides), device="cuda").view(torch.bfloat16)


class State:
    """What a program holds: `keep` (weights, inputs, the model's owner), `out` (result buffers) and `call`, the pass."""

    def __init__(self, call, out, keep, graph=None):
        self.call, self.out, self.keep, self.graph = call, out, keep, graph

    def __del__(self):
        try:
            if self.graph is not None:
                self.graph.free()
        except Exception:
            pass


def recorded(call):
    """`call` once eagerly (it sizes the workspaces), then as a graph."""
    dev = device()
    torch.cuda.synchronize()
    call()
    dev.sync()
    dev.begin_capture()
    call()
    return dev.end_capture()


# ---------------------------------------------------------------------------------------------- the kinds of work
def _host(seed, case):
    r = np.random.default_rng(seed)
    rows, cols = case["rows"], case["cols"]
    w = (r.standard_normal((rows, cols // 32, 32)) / math.sqrt(cols)).astype(np.float32)
    s = np.abs(w).max(2) / np.float32(127 if case["kind"] == "q8_f32" else 7)
    q = np.rint(w / s[:, :, None])
    return (q.clip(-127, 127) if case["kind"] == "q8_f32" else q.clip(-8, 7)).astype(np.int8), s, r.standard_normal(cols)


def prepare_matvec(case, seed):
    q, s, x = _host(seed, case)
    shape, dev = [case["rows"], case["cols"]], device()
    if case["kind"] == "q8_f32":
        w = dev.upload_q8(tb.QuantizedQ8(s.reshape(-1), q.reshape(-1), shape))
        return State(lambda: dev.q8_matvec(w, x), None, [w, x])
    c = (q.reshape(-1, 2) + 8).astype(np.uint8)
    w = dev.upload_q4(tb.QuantizedQ4(s.reshape(-1), c[:, 0] | (c[:, 1] << 4), shape))
    return State(lambda: dev.q4_matvec(w, x), None, [w, x])


def exact_matvec(case, seed):
    q, s, x = _host(seed, case)
    return (q * s[:, :, None].astype(np.float64)).reshape(case["rows"], case["cols"]) @ x


def _linear_x(case, seed, i):
    t = torch.randn((case["m"], case["cols"]), device="cuda", generator=_gen(seed, 100 + i))
    return t if case["x"] == "f32" else t.bfloat16()


def prepare_linear(case, seed):
    dev, n, m = device(), case["layers"], case["m"]
    dt = torch.float32 if case["y"] == "f32" else torch.bfloat16
    w = [qweight(seed, i, case["kind"], case["rows"], case["cols"]) for i in range(n)]
    x = [_linear_x(case, seed, i) for i in range(n)]
    out = [torch.empty((m, case["rows"]), dtype=dt, device="cuda") for _ in range(n)]
    xb, ob = [buf(t) for t in x], [buf(t) for t in out]

    def call():
        for i in range(n):
            dev.qlinear(xb[i], w[i], m, out=ob[i])

    if n == 1:
        return State(call, out, [w, x])
    g = recorded(call)
    return State(g.launch, out, [w, x], graph=g)


def exact_linear(case, seed):
    return [_linear_x(case, seed, i).double() @ dequantised(case["kind"], *quantised(seed, i, case["kind"], case["rows"], case["cols"])).T for i in range(case["layers"])]


# -- the Llama-shaped model: int4 weights in groups of 32 with f16 scales, bf16 cache
def _llama_shapes(size):
    L, d, H, G, hd, f, V = LLAMA[size]
    return [((H + 2 * G) * hd, d), (d, H * hd), (2 * f, d), (d, f)]


def _lengths(case):
    """Cached positions of each sequence: the longest `ctx`, the others down to about half of it in equal steps."""
    step = case["ctx"] // (2 * case["batch"])
    return [case["ctx"] - i * step for i in range(case["batch"])], step


def _shown(layers):
    """Layers whose new cache rows are among the outputs (all, or every other one of many)."""
    return range(0, layers, 1 if layers <= 31 else 2)


def _llama(case, seed, max_seq):
    dev, (L, d, H, G, hd, f, V), batch = device(), LLAMA[case["size"]], case["batch"]
    model = tb.LlamaModel(dev, tb.LlamaConfig(L, d, H, G, hd, f, V, max_seq, batch, EPS, ROPE_BASE))
    owner = Owner(model)
    keep = [owner]
    for i in range(L):
        w = [qweight(seed, 10 * i + j, "q4_f16", r, c) for j, (r, c) in enumerate(_llama_shapes(case["size"]))]
        gains = [normal(seed, 10 * i + j, (d,), 0.1, 1.0) for j in (4, 5)]
        keep.append(gains)
        model.set_layer(i, tb.LlamaLayerWeights(w[0], w[1], dev.interleave_gate_up(w[2]), w[3], buf(gains[0]), buf(gains[1])))
        kp, vp, stride = model.kv_cache(i)
        for j, p in ((6, kp), (7, vp)):
            view(owner, p, (batch, max_seq, G * hd), (stride, G * hd, 1)).normal_(generator=_gen(seed, 10 * i + j))
    embed, gain = normal(seed, 9001, (V, d)), normal(seed, 9002, (d,), 0.1, 1.0)
    model.set_head(buf(embed), buf(gain), qweight(seed, 9003, "q4_f16", V, d))
    keep += [embed, gain]
    return model, keep


def _tokens(seed, shape, vocab):
    return torch.randint(0, vocab, shape, dtype=torch.int32, device="cuda", generator=_gen(seed, 9100))


def prepare_decode(case, seed):
    L, d, H, G, hd, f, V = LLAMA[case["size"]]
    B, max_seq = case["batch"], case["ctx"] + 1
    model, keep = _llama(case, seed, max_seq)
    lens, step = _lengths(case)
    tok, pos = _tokens(seed, (B,), V), torch.tensor(lens, dtype=torch.int32, device="cuda")
    out = {"logits": torch.empty((B, V), device="cuda"), "k": [], "v": []}
    for i in _shown(L):
        kp, vp, stride = model.kv_cache(i)
        for n, p in (("k", kp), ("v", vp)):   # the appended row of sequence b is row lens[b] of its cache
            out[n].append(view(keep[0], p + 2 * lens[0] * G * hd, (B, G * hd), (stride - step * G * hd, 1)))
    tb_, pb, lb = buf(tok), buf(pos), buf(out["logits"])
    g = recorded(lambda: model.decode(tb_, pb, B, max_seq, lb))
    return State(g.launch, out, [keep, tok, pos], g)


def prepare_prefill(case, seed):
    L, d, H, G, hd, f, V = LLAMA[case["size"]]
    B, n, start = case["batch"], case["q_len"], case["start"]
    model, keep = _llama(case, seed, start + n)
    tok, st = _tokens(seed, (B, n), V), torch.full((B,), start, dtype=torch.int32, device="cuda")
    out = {"logits": torch.empty((B, V), device="cuda"), "k": [], "v": []}
    for i in _shown(L):
        kp, vp, stride = model.kv_cache(i)
        for name, p in (("k", kp), ("v", vp)):
            out[name].append(view(keep[0], p + 2 * start * G * hd, (B, n, G * hd), (stride, G * hd, 1)))
    tb_, sb, lb = buf(tok), buf(st), buf(out["logits"])
    torch.cuda.synchronize()
    return State(lambda: model.prefill(tb_, sb, B, n, lb), out, [keep, tok, st])


def _rms(x, gain, eps=EPS):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * gain.double()


def _rope(x, pos, base):
    """Pairs (2i, 2i + 1) of x [..., n, heads, dim] turned by the angles of positions pos [..., n]."""
    half = x.shape[-1] // 2
    a = pos.double()[..., None, None] / base ** (torch.arange(half, device="cuda").double() / half)
    c, s, e, o = a.cos(), a.sin(), x[..., 0::2], x[..., 1::2]
    return torch.stack((e * c - o * s, e * s + o * c), -1).flatten(-2)


def _exact_llama(case, seed, starts, n, max_seq):
    """Logits of the last of n new tokens per sequence, and the new cache rows."""
    L, d, H, G, hd, f, V = LLAMA[case["size"]]
    B = case["batch"]
    tok = _tokens(seed, (B, n) if case["path"] == "prefill" else (B,), V).view(B, n)
    h = normal(seed, 9001, (V, d))[tok.long()].double()
    pos = torch.tensor(starts, device="cuda")[:, None] + torch.arange(n, device="cuda")
    out = {"logits": None, "k": [], "v": []}
    for i in range(L):
        W = lambda j: dequantised("q4_f16", *quantised(seed, 10 * i + j, "q4_f16", *_llama_shapes(case["size"])[j]))
        caches = [torch.empty((B, max_seq, G * hd), dtype=torch.bfloat16, device="cuda").normal_(generator=_gen(seed, 10 * i + j)) for j in (6, 7)]
        qkv = (_rms(h, normal(seed, 10 * i + 4, (d,), 0.1, 1.0)) @ W(0).T).view(B, n, H + 2 * G, hd)
        q, k, v = _rope(qkv[:, :, :H], pos, ROPE_BASE), _rope(qkv[:, :, H:H + G], pos, ROPE_BASE), qkv[:, :, H + G:]
        att = torch.empty((B, n, H, hd), dtype=torch.float64, device="cuda")
        for b in range(B):
            s0 = starts[b]
            kk = torch.cat((caches[0][b, :s0].double().view(s0, G, hd), k[b]))
            vv = torch.cat((caches[1][b, :s0].double().view(s0, G, hd), v[b]))
            for g in range(G):
                qs = q[b, :, g * (H // G):(g + 1) * (H // G)]                      # [n, group, hd]
                s = torch.einsum("nhd,kd->hnk", qs, kk[:, g]) / math.sqrt(hd)
                s.masked_fill_(torch.arange(s0 + n, device="cuda")[None, :] > pos[b][:, None], -math.inf)
                att[b, :, g * (H // G):(g + 1) * (H // G)] = torch.einsum("hnk,kd->nhd", s.softmax(-1), vv[:, g])
        if i in _shown(L):
            out["k"].append(k.reshape(B, n, -1) if case["path"] == "prefill" else k.reshape(B, -1))
            out["v"].append(v.reshape(B, n, -1) if case["path"] == "prefill" else v.reshape(B, -1))
        h = h + att.view(B, n, H * hd) @ W(1).T
        gu = _rms(h, normal(seed, 10 * i + 5, (d,), 0.1, 1.0)) @ W(2).T
        h = h + (torch.nn.functional.silu(gu[..., :f]) * gu[..., f:]) @ W(3).T
    x = _rms(h[:, -1], normal(seed, 9002, (d,), 0.1, 1.0))
    pay, sc = quantised(seed, 9003, "q4_f16", V, d)
    out["logits"] = torch.cat([x @ dequantised("q4_f16", pay[r:r + 16384], sc[r:r + 16384]).T for r in range(0, V, 16384)], 1)
    return out


def exact_decode(case, seed):
    return _exact_llama(case, seed, _lengths(case)[0], 1, case["ctx"] + 1)


def exact_prefill(case, seed):
    return _exact_llama(case, seed, [case["start"]] * case["batch"], case["q_len"], case["start"] + case["q_len"])


# -- the expert layer
def _moe_shapes():
    d, f, E, k, sh = MOE
    return [(E * 2 * f, d), (E * d, f)] + [s for _ in range(sh) for s in ((2 * f, d), (d, f))]


def prepare_moe(case, seed):
    dev, (d, f, E, k, sh), T = device(), MOE, case["tokens"]
    w = [qweight(seed, j, "q4_f16", r, c) for j, (r, c) in enumerate(_moe_shapes())]
    wg, h = normal(seed, 50, (E, d), 0.02), normal(seed, 51, (T, d))
    layer = tb.MoeLayer(dev, tb.MoeConfig(d, f, E, k, sh, int(case["renorm"]), 0, 1), buf(wg), w[0], w[1], w[2::2], w[3::2])
    out = torch.empty((T, d), device="cuda")
    hb, ob = buf(h), buf(out)
    g = recorded(lambda: layer.forward(hb, T, out=ob))
    return State(g.launch, out, [Owner(layer), wg, h, w], g)


def exact_moe(case, seed):
    d, f, E, k, sh = MOE
    h = normal(seed, 51, (case["tokens"], d)).double()
    p = (h @ normal(seed, 50, (E, d), 0.02).double().T).softmax(1)
    top, idx = p.topk(k, 1)
    if case["renorm"]:
        top = top / top.sum(1, keepdim=True)
    w = [quantised(seed, j, "q4_f16", r, c) for j, (r, c) in enumerate(_moe_shapes())]
    out = torch.zeros_like(h)

    def expert(x, gu, dn):
        y = x @ dequantised("q4_f16", *gu).T
        return (torch.nn.functional.silu(y[:, :f]) * y[:, f:]) @ dequantised("q4_f16", *dn).T

    for e in range(E):
        t, c = (idx == e).nonzero(as_tuple=True)
        if len(t):
            part = lambda a, n: tuple(x[e * n:(e + 1) * n] for x in a)
            out[t] += top[t, c][:, None] * expert(h[t], part(w[0], 2 * f), part(w[1], d))
    for s in range(sh):
        out += expert(h, w[2 + 2 * s], w[3 + 2 * s])
    return out


# -- latent attention: int8 weights with a scale per row, bf16 latents
def _mla_shapes(H):
    d, r, c, nope, rope, v = MLA
    return [(r, d), (H * (nope + rope), r), (H * c, nope), (H * v, c), (d, H * v)]


def _mla_cache(case, seed):
    return torch.empty((case["batch"], case["ctx"], MLA[2] + MLA[4]), dtype=torch.bfloat16, device="cuda").normal_(generator=_gen(seed, 60))


def prepare_mla(case, seed):
    dev, (d, r, c, nope, rope, v), H, B, ctx = device(), MLA, case["heads"], case["batch"], case["ctx"]
    w = [qweight(seed, j, "i8_row", a, b) for j, (a, b) in enumerate(_mla_shapes(H))]
    gain, h, cache = normal(seed, 61, (r,), 0.1, 1.0), normal(seed, 62, (B, d)), _mla_cache(case, seed)
    layer = tb.MlaLayer(dev, tb.MlaConfig(d, H, r, c, nope, rope, v, B, ctx, EPS), w[0], buf(gain), w[1], w[2], w[3], w[4], MLA_BASE)
    lens = torch.tensor(_lengths(case)[0], dtype=torch.int32, device="cuda")
    out = torch.empty((B, d), device="cuda")
    hb, cb, lb, ob = buf(h), buf(cache), buf(lens), buf(out)
    g = recorded(lambda: layer.decode(hb, cb, lb, B, ctx * (c + rope), ctx, out=ob))
    return State(g.launch, out, [Owner(layer), w, gain, h, cache, lens], g)


def exact_mla(case, seed):
    (d, r, c, nope, rope, v), H, B = MLA, case["heads"], case["batch"]
    W = [dequantised("i8_row", *quantised(seed, j, "i8_row", a, b)) for j, (a, b) in enumerate(_mla_shapes(H))]
    cache, lens = _mla_cache(case, seed), _lengths(case)[0]
    q = (_rms(normal(seed, 62, (B, d)).double() @ W[0].T, normal(seed, 61, (r,), 0.1, 1.0)) @ W[1].T).view(B, H, nope + rope)
    q_rope = _rope(q[:, :, nope:], torch.tensor(lens, device="cuda") - 1, MLA_BASE)
    q = torch.cat((torch.einsum("bhn,hcn->bhc", q[:, :, :nope], W[2].view(H, c, nope)), q_rope), -1)
    o = torch.empty((B, H, v), dtype=torch.float64, device="cuda")
    for b in range(B):
        rows = cache[b, :lens[b]].double()
        p = (q[b] @ rows.T / math.sqrt(nope + rope)).softmax(-1)
        o[b] = torch.einsum("hc,hvc->hv", p @ rows[:, :c], W[3].view(H, v, c))
    return o.view(B, H * v) @ W[4].T


# -- the dense family
TZ_EPS, TZ_LAMBDA, TZ_DIFF, TZ_LIMIT = 1e-6, 0.5, 0.3, 7.0


def _tz_shapes(size, positions):
    L, d, H, G, D, V, f, vocab = TOFAZEN[size]
    return {"embed": (vocab, d), "pos": (positions, d), "final.norm": (1, d), "head": (vocab, d), "norm1": (1, d), "q": (2 * H * D, d), "k": (2 * G * D, d),
            "v": (G * V, d), "o": (d, H * V), "gate": (f, d), "up": (f, d), "down": (d, f)}


def _tz_tensor(case, seed, i, name):
    r, c = _tz_shapes(case["size"], case["longest"] + 1)[name]
    return normal(seed, i, (r, c), 0.1, 1.0) if r == 1 else normal(seed, i, (r, c), 1.0 if name in ("embed", "pos") else c ** -0.5)


def _tz_config(case):
    L, d, H, G, D, V, f, vocab = TOFAZEN[case["size"]]
    layers = [TofazenLayer(H, G, D, V, D ** -0.5, TZ_DIFF, case["window"], case["keep"], None, f, TZ_LIMIT) for _ in range(L)]
    return TofazenConfig(vocab, d, case["longest"] + 1, TZ_EPS, 1.0, layers)


def _tz_lengths(case):
    n = case["seqs"]
    return [max(1, case["longest"] - i * case["longest"] // (n + 1)) for i in range(n)]


def _tz_tokens(case, seed):
    """Each sequence's prompt, and the token that a decode step appends."""
    vocab = TOFAZEN[case["size"]][7]
    return [torch.randint(0, vocab, (n + 1,), dtype=torch.int32, device="cuda", generator=_gen(seed, 9200 + i)) for i, n in enumerate(_tz_lengths(case))]


def prepare_tofazen(case, seed):
    dev, cfg, lens, n = device(), _tz_config(case), _tz_lengths(case), case["seqs"]
    model = TofazenModel(dev, cfg, [TZ_LAMBDA] * len(cfg.layers), tb.BF16, n, case["longest"] + 1)
    for i, (name, tensor, layer) in enumerate(tensor_names(cfg)):
        t = _tz_tensor(case, seed, i, name if name in ("embed", "pos", "final.norm", "head") else name.split(".")[-1])
        torch.cuda.synchronize()
        model.put_pointer(tensor, layer, t.data_ptr(), tb.BF16, *t.shape)
        dev.sync()
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    toks = _tz_tokens(case, seed)
    prompt, cu = torch.cat([t[:-1] for t in toks]), ints([0] + list(np.cumsum(lens)))
    starts, last = ints([0] * n), ints([int(v) - 1 for v in np.cumsum(lens)])
    out = torch.empty((n, cfg.vocab), device="cuda")
    pb, cb, sb, eb, ob = buf(prompt), buf(cu), buf(starts), buf(last), buf(out)
    step = lambda: model.step(pb, prompt.numel(), cb, sb, None, n, max(lens), max(lens), eb, n, ob)
    keep = [Owner(model), prompt, cu, starts, last, toks]
    torch.cuda.synchronize()
    if not case["decode"]:
        return State(step, out, keep)
    step()
    dev.sync()
    new, at = torch.stack([t[-1] for t in toks]), ints(lens)
    nb, ab = buf(new), buf(at)
    g = recorded(lambda: model.decode(nb, ab, n, case["longest"] + 1, ob))
    return State(g.launch, out, keep + [new, at], g)


def exact_tofazen(case, seed):
    L, d, H, G, D, V, f, vocab = TOFAZEN[case["size"]]
    names = [n for n, _, _ in tensor_names(_tz_config(case))]
    T = lambda name: _tz_tensor(case, seed, names.index(name), name if name in ("embed", "pos", "final.norm", "head") else name.split(".")[-1]).double()
    toks = [t if case["decode"] else t[:-1] for t in _tz_tokens(case, seed)]
    norm = lambda x, g=1.0: x * torch.rsqrt(x.square().mean(-1, keepdim=True) + TZ_EPS) * g
    embed, pos = T("embed"), T("pos")
    xs = [embed[t.long()] + pos[:len(t)] for t in toks]
    for i in range(L):
        w = {n: T(f"l{i}.{n}") for n in ("norm1", "mix.q", "mix.k", "mix.v", "mix.o", "mlp.gate", "mlp.up", "mlp.down")}
        for b, x in enumerate(xs):
            n = len(x)
            h = norm(x, w["norm1"])
            q, k, v = (h @ w["mix.q"].T).view(n, G, H // G, 2, D), (h @ w["mix.k"].T).view(n, G, 2, D), (h @ w["mix.v"].T).view(n, G, V)
            s = torch.einsum("ighmd,jgmd->mghij", q, k) * D ** -0.5
            at = torch.arange(n, device="cuda")
            gap = at[:, None] - at[None, :]
            s.masked_fill_((gap < 0) | ((gap >= case["window"]) & (at[None, :] >= case["keep"])), -math.inf)
            a = torch.einsum("mghij,jgv->mighv", s.softmax(-1), v)
            o = norm(a[0] - TZ_LAMBDA * a[1]).reshape(n, H * V) * (1 - TZ_DIFF)
            g, u = (h @ w["mlp.gate"].T).clamp(max=TZ_LIMIT), (h @ w["mlp.up"].T).clamp(-TZ_LIMIT, TZ_LIMIT)
            xs[b] = x + o @ w["mix.o"].T + (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w["mlp.down"].T
    return norm(torch.stack([x[-1] for x in xs]), T("final.norm")) @ T("head").T


# ---------------------------------------------------------------------------------------------- the file's interface
def prepare(case, seed):
    state = globals()["prepare_" + case["path"]](case, seed)
    torch.cuda.synchronize()
    return state


def run(state):
    got = state.call()
    return got if state.out is None else state.out


def exact(case, seed):
    return globals()["exact_" + case["path"]](case, seed)


def _bytes_q(kind, rows, cols):
    """Stored bytes of a quantised matrix: codes and scales."""
    n = rows * cols
    return {"q4_f16": n // 2 + n // 16, "q4_f32": n // 2 + n // 8, "q8_f32": n + n // 8, "i8_row": n + 4 * rows}[kind]


def work(case):
    """What one pass cannot do without: every input read and every output written once, and the products' operations."""
    p = case["path"]
    if p == "matvec":
        return {"bytes": _bytes_q(case["kind"], case["rows"], case["cols"]) + 8 * (case["rows"] + case["cols"]), "flops": 2 * case["rows"] * case["cols"]}
    if p == "linear":
        r, c, m = case["rows"], case["cols"], case["m"]
        b = _bytes_q(case["kind"], r, c) + m * c * (4 if case["x"] == "f32" else 2) + m * r * (4 if case["y"] == "f32" else 2)
        return {"bytes": case["layers"] * b, "flops": 2 * case["layers"] * m * r * c}
    if p in ("decode", "prefill"):
        L, d, H, G, hd, f, V = LLAMA[case["size"]]
        B = case["batch"]
        n, lens = (1, _lengths(case)[0]) if p == "decode" else (case["q_len"], [case["start"]] * B)
        params = sum(r * c for r, c in _llama_shapes(case["size"]))
        pairs = sum(n * s + n * (n + 1) // 2 for s in lens)
        b = _bytes_q("q4_f16", L * params + V * d, 1) + 4 * L * G * hd * sum(s + n for s in lens) + B * (n * d * 2 + V * 4)
        return {"bytes": b, "flops": 2 * (L * params * B * n + V * d * B) + 4 * L * H * hd * pairs}
    if p == "moe":
        (d, f, E, k, sh), T = MOE, case["tokens"]
        experts = E * (1 - (1 - k / E) ** T) + sh     # experts that T tokens are expected to reach
        return {"bytes": int(experts * (_bytes_q("q4_f16", 3 * f, d)) + 6 * T * d + 2 * E * d), "flops": 2 * T * ((k + sh) * 3 * f * d + E * d)}
    if p == "mla":
        (d, r, c, nope, rope, v), H, lens = MLA, case["heads"], _lengths(case)[0]
        w = sum(a * b for a, b in _mla_shapes(H))
        rows = sum(lens)
        return {"bytes": w + 2 * rows * (c + rope) + 6 * case["batch"] * d, "flops": 2 * case["batch"] * w + 2 * rows * H * (2 * c + rope)}
    L, d, H, G, D, V, f, vocab = TOFAZEN[case["size"]]
    lens, params = _tz_lengths(case), d * (2 * H * D + 2 * G * D + G * V + H * V + 3 * f)
    near = case["window"] + case["keep"]
    rows = [1] * len(lens) if case["decode"] else lens
    pairs = sum(min(n + 1, near) if case["decode"] else sum(min(i + 1, near) for i in range(n)) for n in lens)
    kv = G * (2 * D + V) * 2
    b = 2 * (L * params + vocab * d) + L * kv * sum(min(n + 1, near) if case["decode"] else n for n in lens) + sum(rows) * 4 * d + 4 * len(lens) * vocab
    return {"bytes": b, "flops": 2 * L * params * sum(rows) + 2 * len(lens) * vocab * d + 2 * L * H * (2 * D + 2 * V) * pairs}


def tolerance(case):
    """Relative errors of another correct implementation at the same precision, about four times the error against
    ``exact``: single results rounded to bf16 0.0024, 32-bit sums of exact products 1e-7 (host vectors) to 3e-5 (scales
    of 24 bits in two bf16 terms), a layer of experts 0.0017, of latent attention 0.0045, 16 to 32 layers 0.005 to 0.012."""
    p = case["path"]
    if p == "linear":
        return {"rel": 1e-2 if case["y"] == "bf16" else 2e-4}
    return {"rel": {"matvec": 1e-6, "decode": 3e-2, "prefill": 3e-2, "moe": 7e-3, "mla": 2e-2, "tofazen": 2e-2}[p]}
