"""The work a user of this package has it do, as cases that can be timed: operators at the boundary (one-row chains, row
operators, batched linears, attention), weight formats made at load time, and whole decoders - prompts, token by token decoding,
lockstep batches - over the quantized and the layered families.

listed() names the cases that are watched, draw() more of the same ranges.  prepare() makes what a program holds before the call
(weights, caches, a sequence), run() is one pass through the public entry points, work() what that pass cannot do without,
exact() its results in 64 bits from torch alone.

The synthetic models are made so that their logits are as peaked as a trained model's: the output rows are the embedding rows in
another order, so the next token is that of the current token's successor by a wide margin, whatever the rounding."""
from __future__ import annotations

import math

import numpy as np
import torch

EPS = 1e-5
ROPE_THETA = 1.0e6
# geometries of this repository's configurations and suites: width, heads, kv heads, head size, feed-forward, vocabulary
MISTRAL = dict(dim=4096, heads=32, kv_heads=8, head_dim=128, ff=14336, vocab=32000)
QWEN = dict(dim=896, heads=14, kv_heads=2, head_dim=64, ff=4864, vocab=151936)
MIDDLE = dict(dim=2048, heads=16, kv_heads=4, head_dim=128, ff=8192, vocab=32000)


def listed():
    return [
        # one projection with its residual and the norm behind it, as an operator host calls them for one token
        dict(name="chain_w4p_4096", kind="chain", fmt="w4p", rows=4096, cols=4096),
        # the row operators around the projections for a batch of sequences, bf16
        dict(name="rows_bf16_48", kind="rows", batch=48, dim=4096, ff=11008, heads=32, head_dim=128, context=4000),
        # one batched linear of a prompt portion, ragged number of rows
        dict(name="gemm_w4_300", kind="gemm", fmt="w4g128", m=300, n=18944, k=3584),
        # attention operators in f32: a prompt, then the token behind it
        dict(name="attend_777", kind="attend", tokens=777, heads=32, kv_heads=8, head_dim=128),
        # a checkpoint's matrix brought into both weight formats
        dict(name="load_14336x4096", kind="load", rows=14336, cols=4096),
        # single-stream decoding at a long context, 4-bit weights
        dict(name="decode_w4_2048", kind="decode", layers=8, fmt="w4g128", kv_bf16=False, window=0, prompt=2048, steps=32, **MISTRAL),
        # single-stream decoding of a small model: latency of the launches
        dict(name="decode_i8_small", kind="decode", layers=24, fmt="i8", kv_bf16=True, window=0, prompt=517, steps=32, **QWEN),
        # the prompt of the headline workload
        dict(name="prompt_w4_2048", kind="prompt", layers=8, fmt="w4g128", kv_bf16=False, window=0, prompt=2048, **MISTRAL),
        # a short ragged prompt, 8-bit weights, bf16 cache, sliding window
        dict(name="prompt_i8_333", kind="prompt", layers=8, fmt="i8", kv_bf16=True, window=256, prompt=333, **MISTRAL),
        # sixteen requests served in lockstep: their prompts, then their tokens
        dict(name="batch_w4_16", kind="batch", layers=8, fmt="w4g128", kv_bf16=False, window=0, prompt=200, steps=96, batch=16, **MISTRAL),
        # a layered decoder's prompt in two portions: latent attention, retention, lightning attention
        dict(name="layered_prompt_2048", kind="layered_prompt", family="pefisun", width=4096, layers=3, prompt=2048, portions=2),
        # token by token decoding of a layered decoder: grouped attention beside gated linear attention, gated delta rule
        dict(name="layered_decode_700", kind="layered_decode", family="somopel", width=4096, layers=4, prompt=700, steps=32),
    ]


def _spread(rng, lo, hi):
    """A whole number, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chain", "rows", "gemm", "attend", "load", "decode", "decode", "prompt", "prompt", "batch", "layered_prompt", "layered_decode"])
    if kind == "chain":
        fmt = rng.choice(["i8", "w4g128", "w4p"])
        return dict(kind=kind, fmt=fmt, rows=_spread(rng, 128, 32000), cols=128 * _spread(rng, 7, 112))
    if kind == "rows":
        heads = rng.choice([8, 14, 32])
        return dict(kind=kind, batch=_spread(rng, 1, 64), dim=8 * _spread(rng, 112, 512), ff=8 * _spread(rng, 608, 1792), heads=heads,
                    head_dim=rng.choice([64, 128]), context=_spread(rng, 64, 4096))
    if kind == "gemm":
        fmt = rng.choice(["i8", "w4g128"])
        return dict(kind=kind, fmt=fmt, m=_spread(rng, 1, 2048), n=_spread(rng, 896, 18944), k=128 * _spread(rng, 7, 112))
    if kind == "attend":
        kv = rng.choice([2, 4, 8])
        return dict(kind=kind, tokens=_spread(rng, 1, 1200), heads=kv * rng.choice([1, 4, 7]), kv_heads=kv, head_dim=rng.choice([64, 128]))
    if kind == "load":
        return dict(kind=kind, rows=_spread(rng, 128, 14336), cols=128 * _spread(rng, 7, 32))
    if kind in ("layered_prompt", "layered_decode"):
        c = dict(kind=kind, family=rng.choice(["pefisun", "somopel"]), width=rng.choice([2048, 4096]), layers=rng.randint(2, 4))
        if kind == "layered_prompt":
            return dict(c, prompt=_spread(rng, 5, 2048), portions=rng.choice([1, 1, 2, 3]))
        return dict(c, prompt=_spread(rng, 5, 1500), steps=rng.randint(8, 40))
    geometry = rng.choice([MISTRAL, QWEN, MIDDLE])
    layers = rng.randint(2, 6) if geometry is MISTRAL else rng.randint(4, 16)
    c = dict(kind=kind, layers=layers, fmt=rng.choice(["i8", "w4g128"]), kv_bf16=rng.random() < 0.4, window=rng.choice([0, 0, 0, 256, 1000]), **geometry)
    if kind == "prompt":
        return dict(c, prompt=_spread(rng, 1, 2048))
    if kind == "decode":
        return dict(c, prompt=_spread(rng, 1, 3000), steps=rng.randint(8, 40))
    return dict(c, prompt=_spread(rng, 8, 250), steps=rng.randint(16, 96), batch=rng.randint(2, 16))


# ---- values --------------------------------------------------------------------------------------------------------------
def _generator(seed, *place):
    key = int(seed) * 1000003 + 17
    for p in place:
        key = (key * 8191 + int(p) + 1) % (1 << 61)
    return torch.Generator(device="cuda").manual_seed(key)


def _normal(seed, place, *shape, std=1.0, mean=0.0):
    return torch.randn(shape, generator=_generator(seed, *place), device="cuda") * std + mean


def _bf16(t):
    return t.to(torch.bfloat16)


def _host16(t):
    """bf16 bit patterns as the host holds them."""
    return t.contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


def _row_i8(w):
    """Row-symmetric int8: values and f32 scales."""
    s = w.abs().amax(1) / 127.0
    return torch.round(w / s[:, None]).clamp(-127, 127).to(torch.int8), s


def _group_w4(w):
    """4-bit groups of 128: packed nibbles and f16 scales."""
    g = w.view(w.shape[0], -1, 128)
    s = (g.abs().amax(2) / 7.0).half()
    q = (torch.round(g / s.float()[:, :, None]).clamp(-7, 7) + 8).to(torch.uint8).view(w.shape)
    return q[:, 0::2] | (q[:, 1::2] << 4), s


def _quantize(fmt, w):
    return _row_i8(w) if fmt == "i8" else _group_w4(w)


def _value64(fmt, parts):
    """The weights that the stored parts mean."""
    v, s = parts
    if fmt == "i8":
        return v.double() * s.double()[:, None]
    q = torch.stack(((v & 15).double() - 8.0, (v >> 4).double() - 8.0), dim=2).view(v.shape[0], -1, 128)
    return (q * s.double()[:, :, None]).view(v.shape[0], -1)


def _matrix(fmt, parts):
    from kmll_b200 import ops
    v, s = parts
    if fmt == "i8":
        return ops.DeviceRowwiseScaledI8Matrix.from_parts(v, s)
    m = ops.DeviceW4G128Matrix(v.contiguous(), s.contiguous(), v.shape[0], v.shape[1] * 2)
    return ops.DeviceW4PMatrix.from_canonical(m) if fmt == "w4p" else m


def _frequencies(dims):
    f = np.float32
    return np.array([f(1.0) / f(float(f(ROPE_THETA)) ** float(f(2 * i) / f(dims))) for i in range(dims // 2)], dtype=np.float32)


def _prompt(seed, n, vocab, at=0):
    return np.random.default_rng([seed, n, at]).integers(0, vocab, n)


def _successor(c, seed):
    """The token that follows each token, and its inverse."""
    nxt = np.random.default_rng([seed, 77]).permutation(c["vocab"])
    back = np.empty_like(nxt)
    back[nxt] = np.arange(nxt.size)
    return nxt, back


# ---- operators -------------------------------------------------------------------------------------------------------------
def _chain_values(c, seed):
    rows, cols = c["rows"], c["cols"]
    return (_normal(seed, (1,), cols), _quantize(c["fmt"], _normal(seed, (2,), rows, cols, std=cols ** -0.5)), _normal(seed, (3,), rows),
            _bf16(_normal(seed, (4,), rows, std=0.1, mean=1.0)))


def _rows_values(c, seed):
    b, d, ff, h, hd, t = c["batch"], c["dim"], c["ff"], c["heads"], c["head_dim"], c["context"]
    positions = torch.randint(0, 4096, (b,), generator=_generator(seed, 9), device="cuda", dtype=torch.int32)
    return dict(x=_bf16(_normal(seed, (1,), b, d)), gamma=_bf16(_normal(seed, (2,), d, std=0.1, mean=1.0)), q=_bf16(_normal(seed, (3,), b, h, hd)),
                gate=_bf16(_normal(seed, (4,), b, ff)), up=_bf16(_normal(seed, (5,), b, ff)), scores=_bf16(_normal(seed, (6,), b * h, t, std=2.0)),
                freqs=torch.from_numpy(_frequencies(hd)).cuda(), positions=positions)


def _gemm_values(c, seed):
    return _normal(seed, (1,), c["m"], c["k"]), _quantize(c["fmt"], _normal(seed, (2,), c["n"], c["k"], std=c["k"] ** -0.5))


def _attend_values(c, seed):
    n, h, g, d = c["tokens"], c["heads"], c["kv_heads"], c["head_dim"]
    return [_normal(seed, (i,), n + 1, w * d) for i, w in enumerate((h, g, g))]


# ---- uniform decoders ------------------------------------------------------------------------------------------------------
_NORMS = (0, 5)  # tensor ids of the two norms of a layer; the linear ones are 1 .. 4 and 6 .. 8


def _shapes(c):
    q, kv, d, ff = c["heads"] * c["head_dim"], c["kv_heads"] * c["head_dim"], c["dim"], c["ff"]
    return {1: (q, d), 2: (kv, d), 3: (kv, d), 4: (d, q), 6: (ff, d), 7: (ff, d), 8: (d, ff)}


def _linear(c, seed, layer, tensor):
    rows, cols = _shapes(c)[tensor]
    return _quantize(c["fmt"], _normal(seed, (layer, tensor), rows, cols, std=cols ** -0.5))


def _embedding(c, seed):
    return _bf16(_normal(seed, (900,), c["vocab"], c["dim"]))


def _output(c, seed, embedding):
    _, back = _successor(c, seed)
    return _quantize(c["fmt"], embedding.float()[torch.from_numpy(back).cuda()] * (0.5 * c["dim"] ** -0.5))


def _norm_weight(c, seed, layer, tensor):
    return _bf16(_normal(seed, (layer, tensor), c["dim"], std=0.1, mean=1.0))


def _decoder(c, seed, room):
    from kmll_b200 import runtime as rt
    cfg = rt.DecoderConfig(n_layers=c["layers"], dim=c["dim"], n_heads=c["heads"], n_kv_heads=c["kv_heads"], head_dim=c["head_dim"], hidden_dim=c["ff"],
                           vocab_size=c["vocab"], rope_theta=ROPE_THETA, norm_eps=EPS, max_seq_len=room, kv_bf16=c["kv_bf16"], sliding_window=c["window"],
                           format=rt.FORMAT_RS_I8 if c["fmt"] == "i8" else rt.FORMAT_W4G128)
    dec = rt.Decoder(cfg)

    def put(layer, tensor, parts):
        v, s = (p.cpu() for p in parts)
        dec.set_tensor(layer, tensor, v.numpy(), s.view(torch.int16).numpy() if s.dtype == torch.float16 else s.numpy())

    for layer in range(c["layers"]):
        for t in _NORMS:
            dec.set_tensor(layer, t, _host16(_norm_weight(c, seed, layer, t)))
        for t in _shapes(c):
            put(layer, t, _linear(c, seed, layer, t))
    e = _embedding(c, seed)
    dec.set_tensor(-1, rt.T_FINAL_NORM, _host16(_norm_weight(c, seed, 999, 0)))
    dec.set_tensor(-1, rt.T_EMBEDDING, _host16(e))
    put(-1, rt.T_OUTPUT, _output(c, seed, e))
    return dec


def _rms64(x, eps=EPS):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps)


def _silu64(x):
    return x / (1.0 + torch.exp(-x))


def _rope64(x, freqs, positions):
    """x [..., tokens, d]: entry i with entry i + d / 2; the angle is the f32 product of position and frequency."""
    a = (positions.float()[:, None] * freqs.float()[None, :]).double()
    u, v = x.chunk(2, -1)
    return torch.cat((u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()), -1)


def _causal64(q, k, v, scale, first=None):
    """q [heads, tokens, d], k / v [kv heads, tokens, d]; `first`: the first position that each position sees."""
    n, per = q.shape[1], q.shape[0] // k.shape[0]
    at = torch.arange(n, device="cuda")
    hidden = at[None, :] > at[:, None]
    if first is not None:
        hidden |= at[None, :] < first[:, None]
    out = []
    for h in range(q.shape[0]):
        s = (q[h] @ k[h // per].T * scale).masked_fill_(hidden, -math.inf)
        out.append(torch.softmax(s, -1) @ v[h // per])
    return torch.stack(out)


def _decoder64(c, seed, sequences, wanted):
    """Logits [sequences, wanted, vocab] of whole sequences of equal length."""
    fmt, hd, H, G = c["fmt"], c["head_dim"], c["heads"], c["kv_heads"]
    tokens = torch.from_numpy(np.stack(sequences)).cuda()
    B, n = tokens.shape
    at = torch.arange(n, device="cuda")
    freqs = torch.from_numpy(_frequencies(hd)).cuda()
    first = (at - c["window"] + 1).clamp(min=0) if c["window"] else None
    e = _embedding(c, seed)
    x = e.double()[tokens]
    for layer in range(c["layers"]):
        W = {t: _value64(fmt, _linear(c, seed, layer, t)) for t in _shapes(c)}
        h = _rms64(x) * _norm_weight(c, seed, layer, 0).double()
        q, k, v = ((h @ W[t].T).view(B, n, -1, hd).transpose(1, 2) for t in (1, 2, 3))
        q, k = _rope64(q, freqs, at), _rope64(k, freqs, at)
        if c["kv_bf16"]:
            k, v = (z.float().bfloat16().double() for z in (k, v))
        o = torch.stack([_causal64(q[b], k[b], v[b], hd ** -0.5, first) for b in range(B)])
        x = x + o.transpose(1, 2).reshape(B, n, H * hd) @ W[4].T
        h = _rms64(x) * _norm_weight(c, seed, layer, 5).double()
        x = x + (_silu64(h @ W[6].T) * (h @ W[7].T)) @ W[8].T
    h = _rms64(x[:, wanted]) * _norm_weight(c, seed, 999, 0).double()
    return h @ _value64(fmt, _output(c, seed, e)).T


# ---- layered decoders ------------------------------------------------------------------------------------------------------
def _layered_config(c, room):
    """config.json of the family at one of the two widths of the operator suites."""
    w, wide = c["width"], c["width"] == 4096
    ff, H, layers = (14336 if wide else 8192), (32 if wide else 16), []
    for i in range(c["layers"]):
        if c["family"] == "pefisun":
            kind = ("latent_attention", "retention", "lightning")[i % 3]
            if kind == "latent_attention":
                m = {"heads": H, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "mask": {"size": 1024},
                     "rot": {"base": 1e4, "dims": 64, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
            else:
                h, d = (H, 128) if kind == "lightning" else (H // 2, 256)
                m = {"heads": h, "dim": d, "vdim": d, "decay": [1.0 - 2.0 ** (-4 - 6 * j / h) for j in range(h)]}
                if kind == "retention":
                    m["rot"] = {"base": 1e4, "dims": d}
        elif i % 2 == 0:
            kind = "parallel"
            m = {"left": {"heads": H, "kv_heads": H // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 512}}, "left_scale": 0.9,
                 "right": {"heads": H, "dim": 128, "vdim": 128, "tau": 12.0}, "right_scale": 1.1}
        else:
            kind, m = "channel_delta", {"heads": H, "kv_heads": H, "dim": 128, "vdim": 128, "conv": 4}
        layers.append({"type": kind, "mixer": m, "mlp": {"kind": "dense", "ff": ff}})
    return {"width": w, "vocab": 32000, "max_positions": room, "norm": {"eps": EPS}, "embedding": {"scale": 1.0}, "logit_scale": 0.5 * w ** -0.5, "layers": layers}


def _layered_parts(c, config):
    """(description of the decoder, [(tensor name, layer or -1, tensor id)])"""
    from kmll_b200 import pefisun, somopel
    if c["family"] == "pefisun":
        return pefisun.layered_config(config), pefisun.tensor_names(config)
    rank = 128 if c["width"] == 4096 else 64
    return somopel.layered_config(config, lambda name: (16 if ".right." in name else rank,)), somopel.tensor_names(config)


def _layered_tensor(c, seed, name, place, shape):
    tail = name.rsplit(".", 1)[-1]
    if name == "head":
        nxt, back = _successor(dict(vocab=shape[0]), seed)
        e = _layered_tensor(c, seed, "embed", (0,), shape)
        return _bf16(e.float()[torch.from_numpy(back).cuda()] * (0.5 * shape[1] ** -0.5))
    if name == "embed":
        place, std, mean = (0,), 1.0, 0.0
    elif name == "pos":
        std, mean = 0.3, 0.0
    elif tail == "act":
        return _bf16(torch.tensor([0.4, 0.2, 0.1, 0.05], device="cuda"))
    elif name.endswith("mix.norm") or name.endswith("dkv.norm") or name.endswith("right.norm") or (tail.startswith("norm") and c["family"] == "somopel"):
        std, mean = 0.1, 1.0
    elif name.endswith("a2.b"):
        std, mean = 1.0, 2.0
    elif tail == "dt_bias":
        std, mean = 1.0, -1.0
    elif tail == "A_log":
        std, mean = 0.7, -0.5
    elif tail == "conv":
        std, mean = 0.5, 0.0
    elif len(shape) == 1:
        std, mean = 0.1, 0.0
    else:
        std, mean = shape[1] ** -0.5 * (0.5 if tail in ("o", "down") else 1.0), 0.0
    return _bf16(_normal(seed, (500,) + place, *shape, std=std, mean=mean))


def _layered(c, seed, room):
    from kmll_b200 import runtime as rt
    cfg, names = _layered_parts(c, _layered_config(c, room))
    dec = rt.LayeredDecoder(cfg)
    for name, layer, tensor in names:
        dec.set_tensor(layer, tensor, _host16(_layered_tensor(c, seed, name, (layer + 1, tensor), cfg.tensor_shape(layer, tensor))))
    return dec


def _sigmoid64(x):
    return torch.sigmoid(x)


def _heads(x, h):
    return x.view(x.shape[0], h, -1).transpose(0, 1)


def _flat(x):
    return x.transpose(0, 1).reshape(x.shape[1], -1)


def _inverse_frequencies(rot):
    dims, base, s = rot["dims"], rot["base"], rot.get("scaling")
    f = np.array([base ** (-2.0 * i / dims) for i in range(dims // 2)])
    if not s:
        return torch.from_numpy(f).cuda(), 1.0

    def where(turns):
        return dims * math.log(s["original"] / (2 * math.pi * turns)) / (2 * math.log(base))

    lo, hi = max(math.floor(where(s["fast"])), 0), min(math.ceil(where(s["slow"])), dims - 1)
    ramp = np.clip((np.arange(dims // 2) - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    return torch.from_numpy(f / s["factor"] * ramp + f * (1.0 - ramp)).cuda(), 0.1 * math.log(s["factor"]) + 1.0


def _rotate64(x, rot):
    f, m = _inverse_frequencies(rot)
    a = torch.arange(x.shape[-2], device="cuda").double()[:, None] * f[None, :]
    u, v = x.chunk(2, -1)
    return torch.cat((u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()), -1) * m


def _recurrence64(q, k, v, alpha, beta=None):
    """[heads, tokens, d]: S <- diag(alpha) S + k u^T, o = S^T q; u = v, or beta (v - S^T k) behind the decay.  alpha [heads,
    tokens, d], or [heads, 1, 1] for a fixed decay."""
    H, n, d = q.shape
    S = torch.zeros(H, d, v.shape[2], dtype=torch.float64, device="cuda")
    out = torch.empty_like(v)
    fixed = alpha.shape[1] == 1
    for i in range(n):
        S *= alpha if fixed else alpha[:, i, :, None]
        ki = k[:, i, :, None]
        u = v[:, i, None, :] if beta is None else beta[:, i, None, None] * (v[:, i, None, :] - ki.transpose(1, 2) @ S)
        S += ki * u
        out[:, i] = (q[:, i, None, :] @ S)[:, 0]
    return out


def _mixer64(kind, h, w, m):
    if kind == "latent_attention":
        H, d, R = m["heads"], m["dim"], m["kv_rank"]
        q, both = _heads(h @ w["q"].T, H), h @ w["dkv"].T
        lat = _rms64(both[:, :R]) * w["dkv.norm"]
        kr = _rotate64(both[None, :, R:], m["rot"])
        k = torch.cat((_heads(lat @ w["uk"].T, H), kr.expand(H, -1, -1)), -1)
        q = torch.cat((q[..., :d], _rotate64(q[..., d:], m["rot"])), -1)
        first = (torch.arange(h.shape[0], device="cuda") - m["mask"]["size"] + 1).clamp(min=0)
        return _flat(_causal64(q, k, _heads(lat @ w["uv"].T, H), m["scale"], first)) @ w["o"].T
    if kind == "retention" or kind == "lightning":
        H = m["heads"]
        decay = torch.tensor(m["decay"], dtype=torch.float64, device="cuda")[:, None, None]
        q, k, v = (_heads(h @ w[n].T, H) for n in "qkv")
        if kind == "retention":
            o = _flat(_rms64(_recurrence64(_rotate64(q, m["rot"]), _rotate64(k, m["rot"]) * m["dim"] ** -0.5, v, decay)))
            return (o * _silu64(h @ w["g"].T)) @ w["o"].T
        o = _flat(_recurrence64(_silu64(q), _silu64(k), _silu64(v), decay))
        return (_rms64(o) * w["norm"] * _sigmoid64(h @ w["g"].T)) @ w["o"].T
    softplus = torch.nn.functional.softplus
    if kind == "parallel":
        a, b = m["left"], m["right"]
        x = {n[5:]: t for n, t in w.items() if n.startswith("left.")}
        H, G, size = a["heads"], a["kv_heads"], a["mask"]["size"]
        first = torch.arange(h.shape[0], device="cuda") // size * size
        o = _causal64(_heads(h @ x["q"].T, H), _heads(h @ x["k"].T, G), _heads(h @ x["v"].T, G), a["scale"], first)
        left = _flat(o * _sigmoid64(h @ x["g"].T).T[:, :, None]) @ x["o"].T
        x = {n[6:]: t for n, t in w.items() if n.startswith("right.")}
        H = b["heads"]
        z = h @ x["a1"].T @ x["a2"].T + x["a2.b"]
        alpha = _heads(torch.exp(-softplus(-z) / b["tau"]), H)
        o = _rms64(_recurrence64(_heads(h @ x["q"].T, H) * b["dim"] ** -0.5, _heads(h @ x["k"].T, H), _heads(h @ x["v"].T, H), alpha)) * x["norm"]
        return m["left_scale"] * left + m["right_scale"] * ((_flat(o) * _silu64(h @ x["g"].T)) @ x["o"].T)
    H, G = m["heads"], m["kv_heads"]

    def convolved(name):
        x, taps = h @ w[name].T, w[name + ".conv"]
        p = torch.cat((x.new_zeros(taps.shape[1] - 1, x.shape[1]), x))
        return _silu64(sum(p[j:j + x.shape[0]] * taps[:, j] for j in range(taps.shape[1])))

    def unit(x):
        return x / torch.sqrt(x.square().sum(-1, keepdim=True) + 1e-6)

    q, k = (unit(_heads(convolved(n), G)).repeat_interleave(H // G, 0) for n in "qk")
    alpha = torch.exp(-torch.exp(w["A_log"])[:, None, None] * _heads(softplus(h @ w["a1"].T @ w["a2"].T + w["dt_bias"]), H))
    o = _recurrence64(q * m["dim"] ** -0.5, k, _heads(convolved("v"), H), alpha, _sigmoid64(h @ w["b"].T).T)
    return (_flat(_rms64(o) * w["norm"]) * _sigmoid64(h @ w["g1"].T @ w["g2"].T)) @ w["o"].T


def _layered64(c, seed, room, tokens, wanted):
    """Logits [wanted, vocab] of one sequence."""
    config = _layered_config(c, room)
    cfg, names = _layered_parts(c, config)
    T = {}

    def tensor(i):
        return {n: _layered_tensor(c, seed, n, (l + 1, t), cfg.tensor_shape(l, t)).double() for n, l, t in names if l == i}

    T = tensor(-1)
    somopel = c["family"] == "somopel"

    def norm(x, part, name):
        if not somopel:
            return _rms64(x) * (1.0 + part[name])
        x = x - x.mean(-1, keepdim=True)
        return _rms64(x) * part[name] + part[name + ".b"]

    x = T["embed"][torch.from_numpy(np.asarray(tokens)).cuda()] + T["pos"][:len(tokens)]
    if somopel:
        x = norm(x, T, "embed.norm")
    for i, layer in enumerate(config["layers"]):
        part = {n.split(".", 1)[1]: t for n, t in tensor(i).items()}
        x = x + _mixer64(layer["type"], norm(x, part, "norm1"), {n[4:]: t for n, t in part.items() if n.startswith("mix.")}, layer["mixer"])
        h = norm(x, part, "norm2")
        if somopel:
            z = h @ part["mlp.gate"].T
            z = 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3))) * (h @ part["mlp.up"].T)
        else:
            u = h @ part["mlp.up"].T
            a, b, d, e = part["mlp.act"].tolist()
            z = a * _rms64(u) + b * _rms64(u ** 2) + d * _rms64(u ** 3) + e
        x = x + z @ part["mlp.down"].T
    h = norm(x[wanted], T, "final.norm")
    return h @ T["embed"].T * config["logit_scale"] if somopel else h @ T["head"].T


# ---- the interface -----------------------------------------------------------------------------------------------------------
def _room(c):
    return -(-(c["prompt"] + c.get("steps", 0) + 8) // 64) * 64


def _cuts(c):
    n, p = c["prompt"], min(c["portions"], c["prompt"])
    return [n * i // p for i in range(p + 1)]


def prepare(case, seed):
    from kmll_b200 import ops
    from kmll_b200.session import Session
    c, kind = case, case["kind"]
    if kind == "chain":
        x, parts, r, gamma = _chain_values(c, seed)
        return dict(kind=kind, x=x, w=_matrix(c["fmt"], parts), r=r, gamma=gamma)
    if kind == "rows":
        return dict(kind=kind, case=c, **_rows_values(c, seed))
    if kind == "gemm":
        x, parts = _gemm_values(c, seed)
        return dict(kind=kind, case=c, x=x, w=_matrix(c["fmt"], parts), ws=ops.linear_batched_workspace(c["m"], c["k"]))
    if kind == "attend":
        n, h, g, d = c["tokens"], c["heads"], c["kv_heads"], c["head_dim"]
        room = n + 64
        cache = [torch.zeros(room * g * d, device="cuda") for _ in range(2)]
        return dict(kind=kind, case=c, room=room, rows=_attend_values(c, seed), freqs=torch.from_numpy(_frequencies(d)).cuda(), k=cache[0], v=cache[1],
                    q_rot=torch.empty(n * h * d, device="cuda"), one=torch.empty(h * d, device="cuda"), ws=ops.single_query_attention_workspace(h, d, room))
    if kind == "load":
        w = _bf16(_normal(seed, (1,), c["rows"], c["cols"], std=0.02))
        return dict(kind=kind, w=w, w32=w.float())
    if kind in ("layered_prompt", "layered_decode"):
        dec = _layered(c, seed, _room(c))
        prompt = _prompt(seed, c["prompt"], 32000)
    else:
        dec = _decoder(c, seed, _room(c))
        prompt = _prompt(seed, c["prompt"], c["vocab"])
    session = Session(dec)
    if kind == "prompt":
        return dict(kind=kind, session=session, prompt=[int(t) for t in prompt])
    if kind == "layered_prompt":
        cuts = _cuts(c)
        return dict(kind=kind, session=session, pieces=[[int(t) for t in prompt[a:b]] for a, b in zip(cuts, cuts[1:])])
    if kind == "batch":
        return dict(kind=kind, case=c, dec=dec, prompts=[_prompt(seed, c["prompt"], c["vocab"], i) for i in range(c["batch"])])
    session.prefill(prompt)
    return dict(kind=kind, case=c, session=session, dec=dec, pending=dec.next_top())


def run(state):
    from kmll_b200 import ops
    from kmll_b200 import runtime as rt
    s, kind = state, state["kind"]
    if kind == "chain":
        h = ops.linear_residual(s["x"], s["w"], s["r"])
        return h, ops.rmsnorm(h, s["gamma"], EPS)
    if kind == "rows":
        c = s["case"]
        return (ops.rmsnorm_batched_bf16(s["x"], s["gamma"], c["batch"], c["dim"], EPS), ops.apply_rope_batched_bf16(s["q"], s["freqs"], s["positions"]),
                ops.silu_mul(s["gate"], s["up"]), ops.softmax_rows(s["scores"]))
    if kind == "gemm":
        c = s["case"]
        return ops.linear_batched(s["x"], s["w"], c["m"], c["k"], c["n"], workspace=s["ws"])
    if kind == "attend":
        c = s["case"]
        n, h, g, d = c["tokens"], c["heads"], c["kv_heads"], c["head_dim"]
        q, k, v = s["rows"]
        ops.prepare_prefill_attention_batch(q[:n], k[:n], v[:n], s["freqs"], n, h * d, g * d, d, s["q_rot"], s["k"], s["v"])
        prompt = ops.prefill_causal_attention(s["q_rot"], s["k"], s["v"], n, s["room"], h, g, d)
        ops.prepare_incremental_attention(q[n], k[n], v[n], s["freqs"], n, s["room"], h, g, d, s["one"], s["k"], s["v"])
        return prompt, ops.single_query_attention(s["one"], s["k"], s["v"], n + 1, s["room"], h, g, d, workspace=s["ws"]), s["k"], s["v"]
    if kind == "load":
        i8 = ops.DeviceRowwiseScaledI8Matrix.from_bf16_rows_symmetric(s["w"])
        w4 = ops.DeviceW4G128Matrix.from_f32_rows(s["w32"])
        return i8.values, i8.scales, w4.packed, w4.gscales, ops.DeviceW4PMatrix.from_canonical(w4).prepared, i8.dequantize(), w4.dequantize()
    if kind == "prompt":
        s["session"].prefill(s["prompt"])
        return s["session"].next_logits_to_host()
    if kind == "layered_prompt":
        s["session"].reset_sequence()
        return [s["session"].extend(p, [len(p) - 1]) for p in s["pieces"]]
    if kind == "batch":
        dec, c = s["dec"], s["case"]
        batch = rt.BatchDecoder(dec, c["batch"])
        for slot, prompt in enumerate(s["prompts"]):
            dec.prefill(prompt)
            batch.adopt(slot)
        out = batch.generate_greedy(c["steps"])
        batch.close()
        return out
    dec = s["dec"]
    dec.rewind(s["case"]["prompt"])
    dec.set_pending(s["pending"])
    tokens, logits = dec.generate_greedy(s["case"]["steps"])
    return tokens, logits, s["session"].next_logits_to_host()


def _weight_bytes(c):
    per = 1.0 if c["fmt"] == "i8" else 0.5 + 2 / 128
    n = c["layers"] * sum(r * k for r, k in _shapes(c).values())
    return n, c["vocab"] * c["dim"], per


def _layered_weights(c):
    cfg, _ = _layered_parts(c, _layered_config(c, _room(c)))
    return cfg.weight_elements() - cfg.vocab_size * cfg.dim, cfg.vocab_size * cfg.dim


def work(case):
    c, kind = case, case["kind"]
    if kind == "chain":
        n = c["rows"] * c["cols"]
        per = {"i8": 1.0, "w4g128": 0.515625, "w4p": 0.515625}[c["fmt"]]
        return dict(bytes=n * per + 4 * c["cols"] + 14 * c["rows"], flops=2 * n)
    if kind == "rows":
        b = c["batch"]
        n = 2 * b * c["dim"] + 2 * b * c["heads"] * c["head_dim"] + 3 * b * c["ff"] + 2 * b * c["heads"] * c["context"]
        return dict(bytes=2 * n, flops=4 * n)
    if kind == "gemm":
        per = 1.0 if c["fmt"] == "i8" else 0.515625
        return dict(bytes=c["n"] * c["k"] * per + 4 * c["m"] * (c["n"] + c["k"]), flops=2 * c["m"] * c["n"] * c["k"])
    if kind == "attend":
        n, h, g, d = c["tokens"] + 1, c["heads"], c["kv_heads"], c["head_dim"]
        return dict(bytes=4 * n * d * (2 * h + 4 * g), flops=2 * n * n * h * d)
    if kind == "load":
        n = c["rows"] * c["cols"]
        return dict(bytes=n * (2 + 1 + 4 + 0.515625 * 2 + 4 + 4), flops=4 * n)
    if kind in ("layered_prompt", "layered_decode"):
        n, head = _layered_weights(c)
        if kind == "layered_prompt":
            return dict(bytes=2 * (n + head), flops=2 * c["prompt"] * n + 2 * c["portions"] * head)
        return dict(bytes=2 * (c["steps"] + 1) * (n + head), flops=2 * (c["steps"] + 1) * (n + head))
    n, head, per = _weight_bytes(c)
    kv = c["layers"] * 2 * c["kv_heads"] * c["head_dim"] * (2 if c["kv_bf16"] else 4)
    q = c["layers"] * c["heads"] * c["head_dim"]
    seen = min(c["window"] or c["prompt"], c["prompt"])
    prompt_flops = 2 * c["prompt"] * n + 2 * head + 4 * q * (c["prompt"] * seen - seen * seen / 2)
    if kind == "prompt":
        return dict(bytes=(n + head) * per + c["prompt"] * kv + 4 * c["vocab"], flops=prompt_flops + 2 * head)
    steps, b = c["steps"], c.get("batch", 1)
    step_bytes = (n + head) * per + b * kv * seen
    step_flops = b * (2 * (n + head) + 4 * q * seen)
    if kind == "decode":
        return dict(bytes=steps * step_bytes + head * per, flops=steps * step_flops + 2 * head)
    return dict(bytes=steps * step_bytes + b * ((n + head) * per + c["prompt"] * kv), flops=steps * step_flops + b * prompt_flops)


def tolerance(case):
    """About four times the distance from exact() that was measured (in brackets)."""
    kind = case["kind"]
    if kind == "load":
        return "exact"
    if kind == "rows":
        return {"rel": 6e-3, "max": 0.01}   # bf16 results, one rounding each (1.7e-3)
    if kind in ("layered_prompt", "layered_decode"):
        return {"rel": 1e-2, "differ": 0.02}  # bf16 activations in prompts, bf16 latent cache (2.5e-3)
    if kind in ("decode", "prompt", "batch"):
        # a bf16 cache rounds values a few ulps apart to either side of a tie (5e-4); f32 throughout, with f16 / bf16 planes (5e-5)
        return {"rel": 2e-3 if case["kv_bf16"] else 2e-4, "differ": 0.02}
    if kind == "gemm":
        return {"rel": 4e-5}  # f32 sums of two f16 planes (8e-6)
    return {"rel": 2e-6}  # f32 sums (4e-7)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "load":
        return None  # bytes and bit patterns
    if kind == "chain":
        x, parts, r, gamma = _chain_values(c, seed)
        h = r.double() + _value64("i8" if c["fmt"] == "i8" else "w4", parts) @ x.double()
        return h, _rms64(h) * gamma.double()
    if kind == "rows":
        v = _rows_values(c, seed)
        a = (v["positions"].float()[:, None] * v["freqs"][None, :]).double()[:, None, :]
        p, q = v["q"].double().chunk(2, -1)
        rope = torch.cat((p * a.cos() - q * a.sin(), q * a.cos() + p * a.sin()), -1)
        return (_rms64(v["x"].double()) * v["gamma"].double(), rope, _silu64(v["gate"].double()) * v["up"].double(), torch.softmax(v["scores"].double(), -1))
    if kind == "gemm":
        x, parts = _gemm_values(c, seed)
        return x.double() @ _value64(c["fmt"], parts).T
    if kind == "attend":
        n, h, g, d = c["tokens"], c["heads"], c["kv_heads"], c["head_dim"]
        at, freqs = torch.arange(n + 1, device="cuda"), torch.from_numpy(_frequencies(d)).cuda()
        q, k, v = (_heads(t.double(), w) for t, w in zip(_attend_values(c, seed), (h, g, g)))
        q, k = _rope64(q, freqs, at), _rope64(k, freqs, at)
        o = _flat(_causal64(q, k, v, d ** -0.5))
        rest = torch.zeros(63 * g * d, dtype=torch.float64, device="cuda")
        return o[:n], o[n], torch.cat((_flat(k).reshape(-1), rest)), torch.cat((_flat(v).reshape(-1), rest))
    if kind == "layered_prompt":
        return [r[None] for r in _layered64(c, seed, _room(c), _prompt(seed, c["prompt"], 32000), [b - 1 for b in _cuts(c)[1:]])]
    # the tokens that follow are known: the models are peaked (the arg-max of these logits says so again)
    vocab = c.get("vocab", 32000)
    steps, n = c.get("steps", 0), c["prompt"]
    same = c.get("family") == "somopel"  # logits read the embedding table: the next token is the current one
    nxt = _successor(dict(vocab=vocab), seed)[0]
    sequences = []
    for b in range(c.get("batch", 1)):
        t = list(_prompt(seed, n, vocab, b))
        for _ in range(steps):
            t.append(t[-1] if same else nxt[t[-1]])
        sequences.append(np.asarray(t))
    wanted = list(range(n - 1, n + steps))
    if kind == "layered_decode":
        logits = _layered64(c, seed, _room(c), sequences[0], wanted)[None]
    else:
        logits = _decoder64(c, seed, sequences, wanted)
    if kind == "prompt":
        return logits[0, 0]
    top, at = logits[:, :steps].max(-1)
    if kind == "batch":
        return at, top
    return at[0], top[0], logits[0, steps]
