"""The work that the framework's speed is measured on: decode steps, verify steps and prompt passes through ``Engine``.

A case is one call that a server or a command-line run makes over and over: ``Engine.forward_rows`` for a step of several
requests' next tokens (or one request's drafts), ``Engine.prefill`` for a prompt.  Shapes are the presets'; ``layers`` cuts a
model to its first layers, so that weights, caches and the prompt before the call are quick to make and rounding does not grow
over the depth.  Weights are random, so the logits are what is compared: the token that a call returns is their arg-max, which
rounding decides where two are close.
"""
import dataclasses
import math

import torch

from b200serve.models.config import preset
from b200serve.models.listed import assemble, tensor_shapes
from b200serve.models.weights import random_weights
from b200serve.runtime.engine import Engine, Row


def _decode(family, layers, requests, depth, kv="bf16", rows=1, backend="auto"):
    """A step of ``rows`` consecutive tokens of each of ``requests`` requests, whose contexts are up to ``depth`` tokens long."""
    return {"op": "decode", "family": family, "layers": layers, "requests": requests, "rows": rows, "depth": depth, "kv": kv, "backend": backend}


def _prompt(family, layers, tokens, past=0, backend="auto"):
    """A prompt of ``tokens`` tokens behind ``past`` earlier ones of the same conversation."""
    return {"op": "prompt", "family": family, "layers": layers, "tokens": tokens, "past": past, "kv": "bf16", "backend": backend}


#: Layers that a family's drawn cases have.
LAYERS = {"small-dense": 2, "dense-27b": 16, "hybrid-27b": 16, "moe-35b-a3b": 16, "napadra-7b": 8}


def listed():
    return [
        # the smallest call: a two-layer model's next token, launches and host work only
        {"name": "small-decode-1", **_decode("small-dense", 2, 1, 200)},
        # one user's chat with the 27B shape: the next token behind 4096
        {"name": "dense-decode-1", **_decode("dense-27b", 32, 1, 4096, backend="w4")},
        # speculative decoding: the pending token and four drafts of one request verified together
        {"name": "dense-verify-5", **_decode("dense-27b", 16, 1, 1500, rows=5)},
        # a few users with long contexts in an int8 cache
        {"name": "dense-decode-8-int8kv", **_decode("dense-27b", 16, 8, 4000, kv="int8")},
        # a busy server: many short conversations in one step
        {"name": "dense-decode-40", **_decode("dense-27b", 16, 40, 600)},
        # gated delta-net layers, several users
        {"name": "hybrid-decode-12", **_decode("hybrid-27b", 16, 12, 900)},
        # mixture of experts, a busy server
        {"name": "moe-decode-48", **_decode("moe-35b-a3b", 16, 48, 300)},
        # unquantised model with recurrent and chunked attention layers, several users
        {"name": "napadra-decode-16", **_decode("napadra-7b", 8, 16, 500)},
        # a long document ingested
        {"name": "dense-prompt-4096", **_prompt("dense-27b", 16, 4096)},
        # the second turn of a conversation, int4 weights only in memory
        {"name": "dense-prompt-900-w4", **_prompt("dense-27b", 16, 900, past=2300, backend="w4")},
        # prompts of the other two large families
        {"name": "hybrid-prompt-3000", **_prompt("hybrid-27b", 16, 3000)},
        {"name": "moe-prompt-2048", **_prompt("moe-35b-a3b", 16, 2048)},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    family = rng.choice(("dense-27b", "dense-27b", "hybrid-27b", "moe-35b-a3b", "napadra-7b"))
    layers = LAYERS[family]
    if rng.random() < 0.6:
        if family == "dense-27b" and rng.random() < 0.3:
            return _decode(family, layers, 1, _log(rng, 100, 8000), kv=rng.choice(("bf16", "int8")), rows=rng.randint(2, 16))
        requests = _log(rng, 1, 64)
        depth = _log(rng, 40, max(80, min(8000, (8000 if family == "napadra-7b" else 24000) // requests)))
        return _decode(family, layers, requests, depth, kv=rng.choice(("bf16", "int8")) if family == "dense-27b" else "bf16")
    past = 0 if family in ("hybrid-27b", "napadra-7b") or rng.random() < 0.5 else _log(rng, 64, 2000)
    tokens = _log(rng, 80, min(4000, 4096 - past))
    backend = "auto" if family == "napadra-7b" else rng.choice(("auto", "w4"))
    return _prompt(family, layers, tokens, past, backend)


# ------------------------------------------------------------------ what a program has in hand
def _config(case):
    cfg = preset(case["family"])
    if cfg.layer_specs:
        return dataclasses.replace(cfg, layer_specs=cfg.layer_specs[: case["layers"]], n_layers=case["layers"])
    return dataclasses.replace(cfg, n_layers=case["layers"])


def _rand(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _listed_tensor(cfg, name, shape, seed):
    """A checkpoint tensor of a model that lists its layers."""
    g = _rand(seed * 100003 + sum((i + 1) * ord(c) for i, c in enumerate(name)))
    r = torch.randn(shape, device="cuda", generator=g) if len(shape) < 2 else torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0, 1, generator=g)
    last, s = name.rsplit(".", 1)[-1], cfg.block.streams
    if last == "mix":          # streams that mostly keep themselves
        return 0.9 * torch.eye(s, device="cuda") + 0.1 / s + 0.02 * r.float()
    if last in ("in", "out") and len(shape) == 1:
        return (1.0 / s if last == "in" else 1.0) + 0.1 * r
    if last == "shift":
        return torch.sigmoid(r)
    if last in ("i.b", "f.b", "b"):
        return r + (2.0 if ".f." in name else -1.0)
    if len(shape) < 2:         # norms, scales, sinks
        return 1.0 + 0.1 * r
    return r.mul_(0.02 if name == "head" else shape[1] ** -0.5)


def _centred(w4b, scale):
    """Nibbles 0 (weight -8) become 8 (weight 0): weights of mean zero, as trained ones are.  With a mean of -1/2 every product
    has a common part as large as all the rest, and rows of a prompt differ by how well it happens to cancel."""
    if w4b is None:
        return
    b = w4b.view(-1, 4352)[:, :4096]
    low, high = (b & 15) == 0, b < 16
    b |= low * 8 + high * 128
    if scale != 1.0:
        w4b.view(-1, 4352).view(torch.float16)[:, 2048:].mul_(scale)


def _weights(case, seed):
    cfg = _config(case)
    torch.manual_seed(seed)
    if cfg.layer_specs:
        shapes = tensor_shapes(cfg)
        return assemble(cfg, lambda name: _listed_tensor(cfg, name, shapes[name], seed), "cuda")
    w = random_weights(cfg, device="cuda", seed=seed, exact=False)
    g = _rand(seed + 1)
    w.embed.mul_(100.0)        # rows of about two, and half as much again from all the layers: none drowns what came before it
    for lw in w.layers:
        of = lambda p, name: getattr(getattr(p, name, None), "w4b", None)              # noqa: E731
        for t in (of(lw, "qkv"), of(lw, "gate_up"), of(lw.gdn, "in_proj"), of(lw.shared, "gate_up"), lw.experts_gate_up_w4b):
            _centred(t, 1.0)
        for t in (of(lw, "o"), of(lw, "down"), of(lw.gdn, "out_proj"), of(lw.shared, "down"), lw.experts_down_w4b):
            _centred(t, (2 * cfg.n_layers) ** -0.5)
        for name in ("input_norm", "post_norm"):
            setattr(lw, name, 1.0 + 0.1 * torch.randn(cfg.hidden, device="cuda", generator=g))
    return w


def _contexts(case):
    """Context lengths of the requests of a decode step: ``depth`` and shorter."""
    return [case["depth"] - i * 37 % (case["depth"] // 2 + 1) for i in range(case["requests"])]


def _ids(case, vocab, seed):
    """Token ids of every request: its context, then what the measured call is given."""
    g = torch.Generator().manual_seed(seed + 2)
    if case["op"] == "prompt":
        return [torch.randint(0, vocab, (case["past"] + case["tokens"],), generator=g).tolist()]
    return [torch.randint(0, vocab, (n + case["rows"],), generator=g).tolist() for n in _contexts(case)]


def prepare(case, seed):
    w = _weights(case, seed)
    ids = _ids(case, w.cfg.vocab, seed)
    longest = max(map(len, ids))
    eng = Engine(w, max_seqs=len(ids), max_len=(longest + 1087) // 1024 * 1024, kv_dtype=case["kv"], prefill_backend=case["backend"])
    new = case["tokens"] if case["op"] == "prompt" else case["rows"]
    for slot, t in enumerate(ids):
        if len(t) > new:
            eng.prefill(slot, t[:-new])
    rows = [Row(slot, len(t) - new + i, t[len(t) - new + i]) for slot, t in enumerate(ids) for i in range(new)] if case["op"] == "decode" else None
    return {"case": case, "engine": eng, "rows": rows, "past": len(ids[0]) - new, "prompt": ids[0][-new:]}


def run(state):
    eng, case = state["engine"], state["case"]
    if case["op"] == "decode":
        # the same positions each time: a pass writes their keys and values again (recurrent states go on)
        eng.forward_rows(state["rows"])
        out = {"logits": eng.logits(len(state["rows"]))}
    else:
        if state["past"]:
            eng.truncate(0, state["past"])
        else:
            eng.reset(0)
        eng.prefill(0, state["prompt"])
        row = eng.last_prefill_row
        out = {"logits": eng.model.buf.logits[row: row + 1]}
    # the cache and the recurrent states; of an int8 cache the scales (its whole numbers round either way near halves)
    out.update({name: t for name, t in eng.kv.page_tensors().items() if t.dtype != torch.int8})
    out.update(eng.kv.states)
    return out


# ------------------------------------------------------------------ what a pass cannot do without
W4 = 4352 / 8192      # bytes of an int4 weight with its share of the scales


def work(case):
    cfg, c = _config(case), case
    if c["op"] == "decode":
        ctx = [n + c["rows"] for n in _contexts(c)]
        rows, head_rows = c["requests"] * c["rows"], c["requests"] * c["rows"]
        keys, pairs = sum(ctx), sum(ctx) * c["rows"]
    else:
        rows, head_rows = c["tokens"], 1
        keys, pairs = c["past"] + rows, rows * c["past"] + rows * (rows + 1) // 2
    h = cfg.hidden
    head = cfg.vocab * h
    nbytes, flops = 2.0 * head + 4 * head_rows * cfg.vocab + 2 * rows * h, 2.0 * head * head_rows
    if cfg.layer_specs:
        for s in cfg.layer_specs:
            m = s.mixer
            n = m.linear_elems(h) + 3 * s.ffn.ff * h
            nbytes += 2 * n
            flops += 2 * n * rows
            if hasattr(m, "kv_heads"):
                nbytes += 2 * keys * m.kv_heads * (m.dim + m.vdim)
                flops += 2 * pairs * m.heads * (m.dim + m.vdim)
            else:
                state = m.heads * m.dim * m.vdim
                nbytes += 2 * 4 * state * (c["requests"] if c["op"] == "decode" else 1)
                flops += 4 * state * rows
        return {"bytes": nbytes, "flops": flops}
    kv = 2 * cfg.kv_dim * (1 + 4 / 128 if c["kv"] == "int8" else 2)
    for i in range(cfg.n_layers):
        if cfg.is_gdn_layer(i):
            n = h * (cfg.gdn_proj_dim + cfg.gdn_value_dim)
            state = cfg.gdn_v_heads * 128 * 128
            nbytes += 2 * 4 * state * (c["requests"] if c["op"] == "decode" else 1)
            flops += 6 * state * rows
        else:
            n = h * (cfg.qkv_dim + cfg.q_dim)
            nbytes += keys * kv
            flops += 4 * pairs * cfg.q_dim
        nbytes += W4 * n
        flops += 2 * n * rows
        if cfg.is_moe:
            e, one = cfg.n_experts, 3 * h * cfg.expert_ffn
            nbytes += W4 * one * (1 + e * (1 - (1 - cfg.top_k / e) ** rows)) + 2 * e * h
            flops += 2 * rows * (one * (cfg.top_k + 1) + e * h)
        else:
            nbytes += W4 * 3 * h * cfg.ffn
            flops += 2 * rows * 3 * h * cfg.ffn
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Activations rounded to bf16 in every layer: logits are 0.4 % off the 64-bit ones behind 2 layers, 0.5 - 0.6 % behind the 8
    with a residual in fp32, 0.8 - 1.3 % behind 16 and 2.2 % behind 64."""
    return {"rel": 0.016 if case["layers"] <= 2 else 0.025 if case["layers"] <= 8 else 0.03, "max": 0.5}


# ------------------------------------------------------------------ the same in 64 bits
def _matrix(w4b, n):
    """fp64 ``[n][k]`` of int4 blocks of 128 rows x 64 columns: nibbles of tile j, row g, column group t, words (32-k step, row
    half) and bytes b (low nibble k, high nibble k + 16), then the rows' fp16 scales in the same row order."""
    nb, kg, _ = w4b.shape
    q = w4b[..., :4096].reshape(nb, kg, 8, 8, 4, 2, 2, 4)                     # [j][g][t][step][half][b]
    q = torch.stack((q & 15, q >> 4), dim=-1).permute(0, 2, 6, 3, 1, 5, 8, 4, 7)   # [nb][j][half][g][kg][step][high][t][b]
    q = q.reshape(nb * 128, kg, 64).double() - 8.0
    s = w4b[..., 4096:].contiguous().view(torch.float16).reshape(nb, kg, 8, 8, 2).permute(0, 2, 4, 3, 1).reshape(nb * 128, kg, 1)
    return (q * s.double()).reshape(nb * 128, kg * 64)[:n]


def _norm(x, w, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _gated(x, gate_up, down):
    y = x @ gate_up.T
    v = y.reshape(len(x), -1, 2, 16)
    return (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(len(x), -1) @ down.T


def _blocks(x, fn, size=8192):
    return torch.cat([fn(x[i: i + size]) for i in range(0, len(x), size)])


def _softmax_rows(q, k, v, scale, slope=None, sink=None, block=512):
    """Causal attention of one sequence, ``[T][heads][d]``."""
    rep = q.shape[1] // k.shape[1]
    kt, vt = k.transpose(0, 1).repeat_interleave(rep, 0), v.transpose(0, 1).repeat_interleave(rep, 0)
    out, at = [], torch.arange(len(k), device=k.device)
    for i in range(0, len(q), block):
        pos = at[i: i + block]
        hi = int(pos[-1]) + 1
        s = torch.matmul(q[i: i + block].transpose(0, 1), kt[:, :hi].transpose(1, 2)) * scale
        back = pos[:, None] - at[None, :hi]
        if slope is not None:
            s -= slope[:, None, None] * back
        s.masked_fill_(back < 0, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[:, None, None].expand(-1, len(pos), 1)], dim=-1)
        p = torch.softmax(s, dim=-1)[..., :hi]
        out.append(torch.matmul(p, vt[:, :hi]).transpose(0, 1))
    return torch.cat(out)


def _padded(parts):
    return torch.nn.utils.rnn.pad_sequence(list(parts))


def _delta_rule(q, k, v, beta, decay):
    """``[T][sequences][heads]...`` token by token."""
    state = torch.zeros(q.shape[1], q.shape[2], q.shape[3], v.shape[3], dtype=q.dtype, device=q.device)
    out = torch.empty_like(v)
    for t in range(len(q)):
        state *= decay[t][..., None, None]
        delta = (v[t] - torch.matmul(k[t][..., None, :], state)[..., 0, :]) * beta[t][..., None]
        state += k[t][..., :, None] * delta[..., None, :]
        out[t] = torch.matmul(q[t][..., None, :], state)[..., 0, :]
    return out


def _delta_net(cfg, g, x, lens):
    nk, nv, d = cfg.gdn_k_heads, cfg.gdn_v_heads, cfg.gdn_head_dim
    kd, vd, cc = cfg.gdn_key_dim, cfg.gdn_value_dim, cfg.gdn_conv_channels
    w = _matrix(g.in_proj.w4b, g.in_proj.n)
    proj = _padded(torch.split(_blocks(x, lambda r: r @ w.T), lens))          # [T][sequences][columns]
    past = torch.cat([torch.zeros_like(proj[:3, :, :cc]), proj[..., :cc]])
    y = torch.nn.functional.silu(sum(past[i: i + len(proj)] * g.conv_w[:, i].double() for i in range(4)))
    q, k, v = (t.unflatten(-1, (-1, d)) for t in (y[..., :kd], y[..., kd: 2 * kd], y[..., 2 * kd:]))
    q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    z, b, a = proj[..., cc: cc + vd].unflatten(-1, (-1, d)), proj[..., cc + vd: cc + vd + nv], proj[..., cc + vd + nv: cc + vd + 2 * nv]
    decay = torch.exp(-torch.exp(g.a_log.double()) * torch.nn.functional.softplus(a + g.dt_bias.double()))
    o = _delta_rule(q.repeat_interleave(nv // nk, 2) * d ** -0.5, k.repeat_interleave(nv // nk, 2), v, torch.sigmoid(b), decay)
    o = (_norm(o, g.norm_w.double(), cfg.rms_eps) * torch.nn.functional.silu(z)).flatten(2)
    return torch.cat([o[:n, i] for i, n in enumerate(lens)]) @ _matrix(g.out_proj.w4b, g.out_proj.n).T


def _rotated(x, pos, theta):
    half = x.shape[-1] // 2
    ang = (pos.double()[:, None] * theta ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half))[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()], -1)


def _experts(cfg, lw, x):
    p = torch.softmax(x @ lw.router.double().T, -1)
    top, idx = torch.sort(p, dim=-1, descending=True, stable=True)
    top, idx = top[:, : cfg.top_k], idx[:, : cfg.top_k]
    top = top / top.sum(-1, keepdim=True)
    out = torch.zeros_like(x)
    if lw.shared is not None:
        out = torch.sigmoid(x @ lw.shared_gate.double().T) * _gated(x, _matrix(lw.shared.gate_up.w4b, lw.shared.gate_up.n), _matrix(lw.shared.down.w4b, lw.shared.down.n))
    order = torch.argsort(idx.flatten(), stable=True)
    count = torch.bincount(idx.flatten(), minlength=cfg.n_experts).tolist()
    at = 0
    for e, n in enumerate(count):
        if n:
            pick = order[at: at + n]
            rows = pick // cfg.top_k
            y = _gated(x[rows], _matrix(lw.experts_gate_up_w4b[e], 2 * cfg.expert_ffn), _matrix(lw.experts_down_w4b[e], cfg.hidden))
            out.index_add_(0, rows, y * top.flatten()[pick, None])
            at += n
    return out


def _trunk(w, ids):
    """Hidden rows of whole sequences, one behind the other."""
    cfg, lens = w.cfg, [len(t) for t in ids]
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    x = w.embed[torch.tensor(sum(ids, []), device="cuda")].double()
    for lw in w.layers:
        h = _norm(x, lw.input_norm.double(), cfg.rms_eps)
        if lw.gdn is not None:
            x = x + _delta_net(cfg, lw.gdn, h, lens)
        else:
            m = _matrix(lw.qkv.w4b, lw.qkv.n)
            y = _blocks(h, lambda r: r @ m.T)
            q, k, v = (t.unflatten(-1, (-1, cfg.head_dim)) for t in (y[:, : cfg.q_dim], y[:, cfg.q_dim: cfg.q_dim + cfg.kv_dim], y[:, cfg.q_dim + cfg.kv_dim:]))
            q, k = _rotated(q, pos, cfg.rope_theta), _rotated(k, pos, cfg.rope_theta)
            o = torch.cat([_softmax_rows(*part, cfg.head_dim ** -0.5) for part in zip(*(torch.split(t, lens) for t in (q, k, v)))])
            x = x + o.flatten(1) @ _matrix(lw.o.w4b, lw.o.n).T
        h = _norm(x, lw.post_norm.double(), cfg.rms_eps)
        if cfg.is_moe:
            x = x + _experts(cfg, lw, h)
        else:
            gu, dn = _matrix(lw.gate_up.w4b, lw.gate_up.n), _matrix(lw.down.w4b, lw.down.n)
            x = x + _blocks(h, lambda r: _gated(r, gu, dn))
    return _norm(x, w.final_norm.double(), cfg.rms_eps)


def _matrix_memory(q, k, v, i, f):
    """mLSTM, ``[T][sequences][heads]...`` token by token; ``i``, ``f``: log gates."""
    shape = q.shape[1:3]
    s = torch.zeros(*shape, q.shape[3], v.shape[3], dtype=q.dtype, device=q.device)
    n, m = torch.zeros(*shape, q.shape[3], dtype=q.dtype, device=q.device), torch.zeros(*shape, dtype=q.dtype, device=q.device)
    out = torch.empty_like(v)
    for t in range(len(q)):
        new = torch.maximum(f[t] + m, i[t])
        keep, add = torch.exp(f[t] + m - new)[..., None], torch.exp(i[t] - new)[..., None]
        m = new
        s = s * keep[..., None] + (add * k[t])[..., :, None] * v[t][..., None, :]
        n = n * keep + add * k[t]
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        out[t] = torch.matmul(q[t][..., None, :], s)[..., 0, :] / den[..., None]
    return out


def _napadra_trunk(cfg, seed, ids):
    shapes, lens, eps, mult = tensor_shapes(cfg), [len(t) for t in ids], cfg.rms_eps, cfg.block.mult

    def w(name):          # as it is served: matrices in bf16, the rest in fp32
        t = _listed_tensor(cfg, name, shapes[name], seed)
        return (t.bfloat16() if len(shapes[name]) == 2 and "hc" not in name else t.float()).double()
    pos = torch.cat([torch.arange(n, device="cuda") for n in lens])
    first = pos == 0
    c = torch.arange(cfg.hidden, device="cuda")
    ang = pos.double()[:, None] * cfg.block.sinusoid ** (-2.0 * (c // 2).double() / cfg.hidden)
    x = w("embed")[torch.tensor(sum(ids, []), device="cuda")] + torch.where(c % 2 == 0, ang.sin(), ang.cos())
    x = x[None].repeat(cfg.block.streams, 1, 1)
    held = {}
    for li, spec in enumerate(cfg.layer_specs):
        p, m = f"l{li}.", spec.mixer
        h = _norm(torch.einsum("s,stw->tw", w(p + "hc1.in"), x), w(p + "norm1"), eps)
        back = torch.where(first[:, None], 0.0, torch.roll(h, 1, 0))
        h = h + (back - h) * w(p + "shift")
        lin = lambda name, d: (h @ w(p + "mix." + name).T).unflatten(-1, (-1, d))       # noqa: E731
        if hasattr(m, "kv_heads"):
            src = m.kv_from if m.kv_from >= 0 else li
            if src == li:
                held[li] = lin("k", m.dim), lin("v", m.vdim)
            slope = 2.0 ** (-m.bias * torch.arange(1, m.heads + 1, dtype=torch.float64, device="cuda") / m.heads)
            q, (k, v) = lin("q", m.dim), held[src]
            y = torch.cat([_softmax_rows(*part, m.scale, slope, w(p + "mix.sink")) for part in zip(*(torch.split(t, lens) for t in (q, k, v)))])
        else:
            cap = lambda z: m.gate_cap * torch.tanh(z / m.gate_cap)                              # noqa: E731
            i = cap(h @ w(p + "mix.i").T + w(p + "mix.i.b"))
            f = torch.nn.functional.logsigmoid(cap(h @ w(p + "mix.f").T + w(p + "mix.f.b")))
            o = _matrix_memory(*(_padded(torch.split(t, lens)) for t in (lin("q", m.dim) * m.dim ** -0.5, lin("k", m.dim), lin("v", m.vdim), i, f)))
            o = torch.cat([o[:n, j] for j, n in enumerate(lens)])
            y = _norm(o, w(p + "mix.norm").unflatten(0, (m.heads, m.vdim)), eps) * torch.sigmoid(lin("g", m.vdim))
        y = y.flatten(1) @ w(p + "mix.o").T
        x = torch.einsum("sr,stw->rtw", w(p + "hc1.mix"), x) + mult * w(p + "hc1.out")[:, None, None] * (y * w(p + "ls1"))
        d = spec.ffn
        h = _norm(torch.einsum("s,stw->tw", w(p + "hc2.in"), x), w(p + "norm2"), eps)
        g, u = (h @ w(p + "mlp.gate").T).clamp(max=d.limit), (h @ w(p + "mlp.up").T).clamp(-d.limit, d.limit)
        y = (g * torch.sigmoid(d.alpha * g) * (u + d.shift)) @ w(p + "mlp.down").T
        x = torch.einsum("sr,stw->rtw", w(p + "hc2.mix"), x) + mult * w(p + "hc2.out")[:, None, None] * (y * w(p + "ls2"))
    return _norm(x.sum(0), w("final.norm"), eps), w("head")


@torch.no_grad()
def exact(case, seed):
    cfg = _config(case)
    ids = _ids(case, cfg.vocab, seed)
    rows = case["rows"] if case["op"] == "decode" else 1
    ends = torch.cumsum(torch.tensor([len(t) for t in ids]), 0).tolist()
    last = [e - rows + i for e in ends for i in range(rows)]
    if cfg.layer_specs:
        x, head = _napadra_trunk(cfg, seed, ids)
    else:
        w = _weights(case, seed)
        x, head = _trunk(w, ids), w.lm_head
    x = x[last]
    return {"logits": torch.cat([x @ part.double().T for part in torch.split(head, 16384)], dim=1)}
