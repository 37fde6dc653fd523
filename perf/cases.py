"""The work that is timed: what a program built on this package does with it, over the sizes that it meets.

Products of quantized weights (single ones, and the seven of a decoder layer from a handful of tokens to a long
prompt), per-group weights, the mixture-of-experts block, a Qwen3-shaped decoder (prompt pass and decode step) and a
decoder of mixed blocks. Weights and activations are drawn on the GPU from the seed alone; weights have zero mean and a
spread of about 0.02, as trained ones do, whatever their format. `exact` restates each path in 64 bits with torch alone.
"""
import math

import numpy as np
import torch

from nn_b200 import api, moe
from nn_b200 import weight_quant as wq
from nn_b200.decoder import BlockConfig, BlockDecoder, BlockTensors, Decoder, DecoderConfig, MIXER_ATTENTION, MIXER_RECURRENT
from nn_b200.formats import QuantFormat

DEV = "cuda:0"
F64 = torch.float64

# rows of the seven projections of a layer, by model shape
SHAPES = {
    "8b": dict(hidden=4096, heads=32, kv=8, ffn=12288, vocab=151936),
    "32b": dict(hidden=5120, heads=64, kv=8, ffn=25600, vocab=151936),
}


def listed():
    return [
        # one token through one projection, f32 in and out: the smallest product a caller makes
        dict(name="linear q8_0 1 row", kind="linear", fmt="Q8_0", n=4096, k=4096, m=1, x="f32", bias=False),
        # sixteen sequences decoded together: four layers' projections, weights larger than the L2 cache
        dict(name="layers q4_k 16 rows", kind="layers", shape="8b", fmt="Q4_K", m=16, layers=4),
        # a short prompt, and a long one or a batch of short ones
        dict(name="layers q4_k 128 rows", kind="layers", shape="8b", fmt="Q4_K", m=128, layers=2),
        dict(name="layers q4_k 512 rows", kind="layers", shape="8b", fmt="Q4_K", m=512, layers=2),
        # a large prompt on the larger model shape
        dict(name="layers q6_k 4096 rows", kind="layers", shape="32b", fmt="Q6_K", m=4096, layers=1),
        # widths that are no power of two, an odd number of f32 rows, a bias: a gpt-oss projection of a few draft tokens
        dict(name="linear mxfp4 37 rows", kind="linear", fmt="MXFP4_SPLIT", n=2880, k=2880, m=37, x="f32", bias=True),
        # packed INT4 weights, one token
        dict(name="group int4 1 row", kind="group", bits=4, group=128, n=12288, k=4096, m=1, x="bf16", count=6),
        # the gpt-oss expert block: 64 sequences of one token each, and a prompt
        dict(name="moe 64 tokens", kind="moe", layout="nk", experts=32, top=4, hidden=2880, inter=2880, tokens=64),
        dict(name="moe 4096 tokens", kind="moe", layout="kn", experts=32, top=4, hidden=2880, inter=2880, tokens=4096),
        # the Qwen3-8B-shaped decoder: one token behind 2048 others, and the pass over a prompt (eight layers of it)
        dict(name="decode token", kind="token", shape="8b", layers=36, context=2048),
        dict(name="decoder prompt", kind="prompt", shape="8b", layers=8, tokens=2048),
        # a decoder of mixed blocks: a prompt and a few given tokens behind it, logits to the host
        dict(name="blocks prompt", kind="blocks", width=2048, ffn=6144, heads=16, kv=4, rec=8, window=512, tokens=1024, steps=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["linear", "linear", "layers", "layers", "group", "moe", "token", "prompt", "blocks"])
    if kind == "linear":
        fmt = rng.choice(["Q8_0", "Q4_0", "Q4_K", "Q6_K", "MXFP4_SPLIT"])
        unit = 256 if fmt in ("Q4_K", "Q6_K") else 64
        return dict(kind=kind, fmt=fmt, n=_log_int(rng, 256, 16384), k=unit * _log_int(rng, 1024 // unit, 16384 // unit), m=_log_int(rng, 1, 700),
                    x=rng.choice(["f32", "bf16"]), bias=rng.random() < 0.5)
    if kind == "layers":
        return dict(kind=kind, shape="8b", fmt=rng.choice(["Q4_K", "Q4_K", "Q6_K", "Q8_0"]), m=_log_int(rng, 1, 3000), layers=2)
    if kind == "group":
        return dict(kind=kind, bits=rng.choice([4, 8]), group=rng.choice([32, 64, 128]), n=_log_int(rng, 1000, 20000), k=128 * _log_int(rng, 8, 100),
                    m=_log_int(rng, 1, 24), x=rng.choice(["f32", "bf16"]), count=rng.choice([1, 2, 3]))
    if kind == "moe":
        return dict(kind=kind, layout=rng.choice(["nk", "kn"]), experts=rng.choice([8, 16, 32]), top=4, hidden=2880, inter=2880, tokens=_log_int(rng, 1, 4096))
    if kind == "token":
        return dict(kind=kind, shape="8b", layers=rng.choice([2, 4, 8]), context=_log_int(rng, 16, 8000))
    if kind == "prompt":
        return dict(kind=kind, shape="8b", layers=rng.choice([1, 2, 4]), tokens=_log_int(rng, 20, 4000))
    return dict(kind=kind, width=1024 * rng.choice([1, 2]), ffn=_log_int(rng, 2000, 6144) // 8 * 8, heads=16, kv=rng.choice([2, 4]), rec=8,
                window=_log_int(rng, 64, 1024), tokens=_log_int(rng, 20, 2000), steps=rng.choice([1, 4, 8]))


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _normal(g, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, device=DEV, generator=g) * scale).to(dtype)


def _bytes(g, *shape):
    return torch.randint(0, 256, shape, dtype=torch.uint8, device=DEV, generator=g)


def _f16(g, count, scale):
    """|scale| between half and one and a half times `scale`, as the bytes of f16."""
    return ((torch.rand(count, device=DEV, generator=g) + 0.5) * scale).to(torch.float16).view(torch.uint8).reshape(count, 2)


def _blocks(g, fmt, n, k):
    """Raw blocks of an [n, k] weight of zero mean and a spread of about 0.02: (bytes, scale bytes or None)."""
    if fmt == "Q8_0":
        out = _bytes(g, n * (k // 32), 34)
        out[:, 0:2] = _f16(g, out.shape[0], 0.02 / 74)
    elif fmt == "Q4_0":
        out = _bytes(g, n * (k // 32), 18)
        out[:, 0:2] = _f16(g, out.shape[0], 0.02 / 4.6)
    elif fmt == "Q4_K":
        out = _bytes(g, n * (k // 256), 144)
        out[:, 8:12] = out[:, 4:8]      # the minimum of a sub-block: its scale times 7.5
        out[:, 14:16] = out[:, 12:14]
        d = _f16(g, out.shape[0], 0.02 / (4.6 * 36)).view(torch.float16)
        out[:, 0:4] = torch.cat([d, (d.float() * 7.5).to(torch.float16)], 1).view(torch.uint8)
    elif fmt == "Q6_K":
        out = _bytes(g, n * (k // 256), 210)
        out[:, 208:210] = _f16(g, out.shape[0], 0.02 / (18 * 74))
    else:                               # MXFP4 codes and E8M0 exponents in buffers of their own
        return _bytes(g, n * (k // 2)), torch.randint(119, 122, (n * (k // 32),), dtype=torch.uint8, device=DEV, generator=g)
    return out.reshape(-1), None


def _weight(g, fmt, n, k):
    raw, scales = _blocks(g, fmt, n, k)
    return api.DeviceWeight.from_device(api.gpu_backend(), QuantFormat[fmt], raw, n, k, scales)


def _dense(raw, scales, fmt, n, k, high_first=False):
    """The [n, k] weight of raw blocks, in 64 bits."""
    def f16(b):
        return b.contiguous().view(torch.float16).to(F64)

    def nibbles(b):
        return torch.stack([b & 15, b >> 4], -1).reshape(b.shape[0], -1)

    if fmt == "Q8_0":
        b = raw.view(-1, 34)
        w = f16(b[:, 0:2]) * b[:, 2:].contiguous().view(torch.int8).to(F64)
    elif fmt == "Q4_0":
        b = raw.view(-1, 18)
        w = f16(b[:, 0:2]) * (nibbles(b[:, 2:]).to(F64) - 8)
    elif fmt == "Q4_K":
        b = raw.view(-1, 144)
        hi = b[:, 12:16].to(torch.int32)
        two = torch.stack([(hi >> s) & 3 for s in (0, 2, 4, 6)], -1)          # [blocks, 4 bytes, 4 fields]
        sc = nibbles(b[:, 4:8]).to(torch.int32) + 16 * two[:, 0:2].reshape(-1, 8)
        mn = nibbles(b[:, 8:12]).to(torch.int32) + 16 * two[:, 2:4].reshape(-1, 8)
        q = nibbles(b[:, 16:]).view(-1, 8, 32).to(F64)
        w = (f16(b[:, 0:2]) * sc).unsqueeze(-1) * q - (f16(b[:, 2:4]) * mn).unsqueeze(-1)
    elif fmt == "Q6_K":
        b = raw.view(-1, 210)
        h = torch.stack([(b[:, 128:192] >> s) & 3 for s in (0, 2, 4, 6)], -1).reshape(b.shape[0], -1)
        q = (nibbles(b[:, :128]).to(torch.int32) + 16 * h.to(torch.int32) - 32).to(F64).view(-1, 16, 16)
        w = (f16(b[:, 208:210]) * b[:, 192:208].contiguous().view(torch.int8).to(F64)).unsqueeze(-1) * q
    else:
        value = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6], dtype=F64, device=DEV)
        value = torch.cat([value, -value])
        c = raw.view(-1, 16)
        c = torch.stack([c >> 4, c & 15] if high_first else [c & 15, c >> 4], -1).reshape(-1, 32)
        w = value[c.long()] * torch.exp2(scales.to(F64) - 127).unsqueeze(-1)
    return w.reshape(n, k)


def _projections(shape):
    s = SHAPES[shape]
    d, q, kv, f = s["hidden"], s["heads"] * 128, s["kv"] * 128, s["ffn"]
    return [("q", q, d), ("k", kv, d), ("v", kv, d), ("o", d, q), ("gate", f, d), ("up", f, d), ("down", d, f)]


def _dtype(name):
    return torch.float32 if name == "f32" else torch.bfloat16


class _Model:
    """A decoder that gives its device memory back when it and the views of its buffers are dropped."""

    def __init__(self, dec):
        self.dec, self.graph, self.buffers = dec, None, None

    def views(self, at):
        """Logits, and the keys and values at the positions `at`."""
        out = [self.buffers[2][:], self.buffers[0][:, :, at], self.buffers[1][:, :, at]]
        for t in out:
            t.owner = self
        return out

    def __del__(self):
        self.graph = self.buffers = None
        self.dec.release()


_STREAMS = []


def _stream():
    """The stream of the decode loop: one for the program, as for any sequence of tokens."""
    if not _STREAMS:
        _STREAMS.append(torch.cuda.Stream())
    return _STREAMS[0]


# ------------------------------------------------------------------------------------------
# single products, layers, per-group weights
# ------------------------------------------------------------------------------------------


def _linear_inputs(c, seed):
    g = _gen(seed)
    return g, _normal(g, c["m"], c["k"], dtype=_dtype(c["x"])), _normal(g, c["n"]) if c["bias"] else None


def _layers_inputs(c, seed):
    g, s, m = _gen(seed), SHAPES[c["shape"]], c["m"]
    return g, {n: _normal(g, m, w, dtype=torch.bfloat16) for n, w in (("x", s["hidden"]), ("a", s["heads"] * 128), ("h", s["hidden"]), ("f", s["ffn"]))}


_LAYER_INPUT = {"q": "x", "k": "x", "v": "x", "o": "a", "gate": "h", "up": "h", "down": "f"}


def _group_inputs(c, seed):
    g = _gen(seed)
    x = _normal(g, c["m"], c["k"], dtype=_dtype(c["x"]))
    ws = []
    for _ in range(c["count"]):
        codes = _bytes(g, c["n"] * c["k"] * c["bits"] // 8)
        groups = c["n"] * (c["k"] // c["group"])
        scale = (torch.rand(groups, device=DEV, generator=g) + 0.5) * (0.02 / (4.6 if c["bits"] == 4 else 74))
        ws.append((codes, scale, torch.randint(-2, 3, (groups,), dtype=torch.int32, device=DEV, generator=g)))
    return x, ws


# ------------------------------------------------------------------------------------------
# the expert block
# ------------------------------------------------------------------------------------------


def _moe_inputs(c, seed):
    g, E, H, I = _gen(seed), c["experts"], c["hidden"], c["inter"]
    t = dict(router_w=_normal(g, E, H, scale=0.05), router_b=_normal(g, E, scale=0.1), gate_up_bias=_normal(g, E, 2 * I, scale=0.1),
             down_bias=_normal(g, E, H, scale=0.1))
    t["gate_up"], t["gate_up_scales"] = _blocks(g, "MXFP4", E * 2 * I, H)    # (the same bytes serve both layouts)
    t["down"], t["down_scales"] = _blocks(g, "MXFP4", E * H, I)
    return t, _normal(g, c["tokens"], H, dtype=torch.bfloat16)


def _moe_exact(c, seed):
    t, x = _moe_inputs(c, seed)
    E, H, I, kn = c["experts"], c["hidden"], c["inter"], c["layout"] == "kn"
    x = x.to(F64)
    p = torch.softmax(x @ t["router_w"].to(F64).T + t["router_b"].to(F64), -1)
    w, idx = torch.topk(p, c["top"], -1)
    w = w / w.sum(-1, keepdim=True)
    y = torch.zeros_like(x)

    def part(name, e, rows, cols):
        size, at = rows * cols // 2, rows * cols // 32
        d = (cols, rows) if kn else (rows, cols)
        m = _dense(t[name][e * size:(e + 1) * size], t[name + "_scales"][e * at:(e + 1) * at], "MXFP4", *d, high_first=kn)
        return m.T if kn else m

    for e in range(E):
        at, slot = torch.nonzero(idx == e, as_tuple=True)
        if at.numel():
            u = x[at] @ part("gate_up", e, 2 * I, H).T + t["gate_up_bias"][e].to(F64)
            gate = torch.nn.functional.silu(u[:, :I]).clamp(-7.0, 7.0)
            y.index_add_(0, at, w[at, slot].unsqueeze(-1) * ((gate * u[:, I:]) @ part("down", e, H, I).T + t["down_bias"][e].to(F64)))
    return y


# ------------------------------------------------------------------------------------------
# the Qwen3-shaped decoder
# ------------------------------------------------------------------------------------------


def _decoder_parts(c, seed):
    """Generator and, layer by layer, (raw blocks of the seven projections, four norms); then the head."""
    g, s = _gen(seed), SHAPES[c["shape"]]
    norm = lambda n: 1.0 + 0.1 * _normal(g, n)  # noqa: E731
    for _ in range(c["layers"]):
        raws = [(_blocks(g, "Q4_K", n, k)[0], n, k) for _, n, k in _projections(c["shape"])]
        yield raws, (norm(s["hidden"]), norm(s["hidden"]), norm(128), norm(128))
    # (rows of the embedding are a stretch of one long draw: no two tokens share theirs)
    yield _normal(g, s["vocab"], s["hidden"], dtype=torch.bfloat16, scale=0.5), norm(s["hidden"]), _blocks(g, "Q6_K", s["vocab"], s["hidden"])[0]


def _decoder(c, seed, max_seq):
    s, b = SHAPES[c["shape"]], api.gpu_backend()
    dec = Decoder(b, DecoderConfig(hidden=s["hidden"], n_heads=s["heads"], n_kv_heads=s["kv"], ffn=s["ffn"], n_layers=c["layers"], vocab=s["vocab"],
                                   max_seq=max_seq, act_dtype=api.BF16))
    for i, part in enumerate(_decoder_parts(c, seed)):
        if i < c["layers"]:
            raws, norms = part
            dec.set_layer(i, *[api.DeviceWeight.from_device(b, QuantFormat.Q4_K, r, n, k) for r, n, k in raws], *norms)
        else:
            embed, final, head = part
            dec.set_head(embed, final, api.DeviceWeight.from_device(b, QuantFormat.Q6_K, head, s["vocab"], s["hidden"]))
    torch.cuda.synchronize()
    return _Model(dec)


def _cache_inputs(c, seed):
    """Keys and values of the tokens in front: one stretch per layer, [layers, kv heads, context, 128]."""
    g, s = _gen(seed + 1000003), SHAPES[c["shape"]]
    return [_normal(g, c["layers"], s["kv"], c["context"], 128) for _ in range(2)], int(torch.randint(0, s["vocab"], (1,), device=DEV, generator=g))


def _prompt_ids(c, seed, vocab):
    return np.random.default_rng(seed).integers(0, vocab, c["tokens"] + c.get("steps", 0)).astype(np.int32)


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotate(x, cos, sin):
    """Half-split rotation of the last axis' first 2 * len(cos) dimensions; x [T, heads, d], cos and sin [T, pairs]."""
    h = cos.shape[-1]
    a, b, cos, sin = x[..., :h], x[..., h:2 * h], cos[:, None], sin[:, None]
    return torch.cat([a * cos - b * sin, b * cos + a * sin, x[..., 2 * h:]], -1)


def _attend(q, k, v, scale, pos0, window=None):
    """q [T, H, d] at positions pos0 .., k, v [S, G, ...] at positions 0 .., causal."""
    T, H, S, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    i, j = pos0 + torch.arange(T, device=DEV)[:, None], torch.arange(S, device=DEV)[None]
    hide = (j > i) if window is None else (j > i) | (i - j >= window)
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device=DEV)
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].T) * scale
        out[:, h] = torch.softmax(s.masked_fill_(hide, -math.inf), -1) @ v[:, h * G // H]
    return out


def _qwen3_exact(c, seed, ids, past, pos0):
    """(logits of the last token, new keys, new values) as the decoder gives them, in 64 bits."""
    s = SHAPES[c["shape"]]
    H, G, T = s["heads"], s["kv"], len(ids)
    parts = list(_decoder_parts(c, seed))
    embed, final, head = parts[-1]
    x = embed[torch.from_numpy(np.asarray(ids, np.int64)).to(DEV)].to(F64)
    # the model's angles are f32 numbers
    inv = (1.0 / 1e6 ** (np.arange(0, 128, 2) / 128.0)).astype(np.float32).astype(np.float64)
    ang = torch.from_numpy((np.arange(pos0, pos0 + T)[:, None] * inv[None]).astype(np.float32).astype(np.float64)).to(DEV)
    cos, sin = torch.cos(ang), torch.sin(ang)
    keys, values = [], []
    for i, (raws, norms) in enumerate(parts[:-1]):
        wq_, wk, wv, wo, wg, wu, wd = (lambda r=r: _dense(r[0], None, "Q4_K", r[1], r[2]).T for r in raws)
        n1, n2, nq, nk = (t.to(F64) for t in norms)
        h = _rms(x, 1e-6) * n1
        q = _rotate(_rms((h @ wq_()).view(T, H, 128), 1e-6) * nq, cos, sin)
        k = _rotate(_rms((h @ wk()).view(T, G, 128), 1e-6) * nk, cos, sin)
        v = (h @ wv()).view(T, G, 128)
        keys.append(k.transpose(0, 1))
        values.append(v.transpose(0, 1))
        if past is not None:
            k = torch.cat([past[0][i].to(F64).transpose(0, 1), k])
            v = torch.cat([past[1][i].to(F64).transpose(0, 1), v])
        x = x + _attend(q, k, v, 128 ** -0.5, pos0).reshape(T, -1) @ wo()
        h = _rms(x, 1e-6) * n2
        x = x + (torch.nn.functional.silu(h @ wg()) * (h @ wu())) @ wd()
    h = (_rms(x[-1:], 1e-6) * final.to(F64)).T
    step = 16384
    logits = [_dense(head.view(s["vocab"], -1)[r:r + step].reshape(-1), None, "Q6_K", min(step, s["vocab"] - r), s["hidden"]) @ h
              for r in range(0, s["vocab"], step)]
    return torch.cat(logits)[:, 0], torch.stack(keys), torch.stack(values)


# ------------------------------------------------------------------------------------------
# the decoder of mixed blocks: windowed attention, gated linear attention (two), retention
# ------------------------------------------------------------------------------------------

_RANK, _TAU, _VOCAB = 16, 16.0, 32768


def _block_configs(c):
    rec = dict(mixer=MIXER_RECURRENT, heads=c["rec"], dim=128, vdim=256, ffn=c["ffn"])
    attention = BlockConfig(MIXER_ATTENTION, c["heads"], c["kv"], 128, 128, c["ffn"], 128, 1e6, 128 ** -0.5, c["window"], 4, False, True)
    gla = BlockConfig(q_scale=128 ** -0.5, decay_rank=_RANK, decay_tau=_TAU, **rec)
    return [attention, gla, gla, BlockConfig(rot_dims=128, rot_base=1e6, k_scale=128 ** -0.5, **rec)]


def _block_parts(c, seed):
    """Per block its tensors (matrices bf16, the rest f32), then (embedding and head in one, final norm)."""
    g, D = _gen(seed), c["width"]
    mat = lambda n, k: _normal(g, n, k, dtype=torch.bfloat16, scale=k ** -0.5)  # noqa: E731
    vec = lambda n: 1.0 + 0.1 * _normal(g, n)  # noqa: E731
    for b in _block_configs(c):
        at = b.mixer == MIXER_ATTENTION
        kv = b.kv_heads if at else b.heads
        q, k, v, m = b.heads * b.dim, kv * b.dim, kv * b.vdim, b.heads * b.vdim
        t = dict(norm=vec(D), q=mat(q, D), k=mat(k, D), v=mat(v, D), g=mat(m, D), o=mat(D, m), gate=mat(b.ffn, D), up=mat(b.ffn, D), down=mat(D, b.ffn))
        if at:
            t.update(q_bias=_normal(g, q, scale=0.1), k_bias=_normal(g, k, scale=0.1), v_bias=_normal(g, v, scale=0.1), o_bias=_normal(g, D, scale=0.1),
                     conv=_normal(g, q + k + v, 4, scale=0.5))
        elif b.decay_rank:
            t.update(a1=mat(_RANK, D), decay_w=_normal(g, q, _RANK, scale=_RANK ** -0.5), decay_b=vec(q), head_norm=vec(b.vdim))
        else:
            t.update(decay=(1.0 - torch.exp2(-torch.linspace(5, 12, b.heads, device=DEV))))
        yield t
    yield _normal(g, _VOCAB, D, dtype=torch.bfloat16), vec(D)


def _block_decoder(c, seed):
    bits = lambda t: t.view(torch.int16).cpu().numpy().view(np.uint16) if t.dtype == torch.bfloat16 else t.cpu().numpy()  # noqa: E731
    blocks = _block_configs(c)
    dec = BlockDecoder(api.gpu_backend(), hidden=c["width"], vocab=_VOCAB, blocks=blocks, max_seq=c["tokens"] + c["steps"] + 8)
    for i, t in enumerate(_block_parts(c, seed)):
        if i < len(blocks):
            dec.set_block(i, BlockTensors(**{n: bits(v) for n, v in t.items()}))
        else:
            e = bits(t[0])
            dec.set_head(e, bits(t[1]), e)
    return _Model(dec)


def _blocks_exact(c, seed, ids):
    """Logits [T, vocab] in 64 bits."""
    parts, D, T = list(_block_parts(c, seed)), c["width"], len(ids)
    embed, final = (t.to(F64) for t in parts[-1])
    x = embed[torch.from_numpy(ids.astype(np.int64)).to(DEV)]
    ang = torch.arange(T, device=DEV, dtype=F64)[:, None] * 1e6 ** (-torch.arange(0, 128, 2, device=DEV, dtype=F64) / 128)[None]
    cos, sin = torch.cos(ang), torch.sin(ang)
    for b, t in zip(_block_configs(c), parts):
        t = {n: v.to(F64) for n, v in t.items()}
        h = _rms(x, 1e-6) * t["norm"]
        q, k, v, gate = h @ t["q"].T, h @ t["k"].T, h @ t["v"].T, h @ t["g"].T
        if b.mixer == MIXER_ATTENTION:
            u = torch.nn.functional.pad(torch.cat([q + t["q_bias"], k + t["k_bias"], v + t["v_bias"]], 1), (0, 0, 3, 0))
            u = sum(u[j:j + T] * t["conv"][:, j] for j in range(4))
            q, k, v = u.split([q.shape[1], k.shape[1], v.shape[1]], 1)
            o = _attend(_rotate(q.view(T, -1, 128), cos, sin), _rotate(k.reshape(T, -1, 128), cos, sin), v.reshape(T, -1, 128), b.scale, 0, b.window)
            mixed = (o.reshape(T, -1) * torch.sigmoid(gate)) @ t["o"].T + t["o_bias"]
        else:
            q, k, v = q.view(T, b.heads, 128), k.view(T, b.heads, 128), v.view(T, b.heads, 256)
            if b.decay_rank:
                z = (h @ t["a1"].T) @ t["decay_w"].T + t["decay_b"]
                a, q = torch.exp(torch.nn.functional.logsigmoid(z) / _TAU).view(T, b.heads, 128, 1), q * b.q_scale
            else:
                a, q, k = t["decay"].view(1, -1, 1, 1).expand(T, -1, 128, 1), _rotate(q, cos, sin), _rotate(k, cos, sin) * b.k_scale
            S = torch.zeros(b.heads, 128, 256, dtype=F64, device=DEV)
            o = torch.empty(T, b.heads, 256, dtype=F64, device=DEV)
            for i in range(T):
                S.mul_(a[i]).addcmul_(k[i].unsqueeze(-1), v[i].unsqueeze(1))
                o[i] = torch.einsum("hd,hde->he", q[i], S)
            o = _rms(o, 1e-6) * (t["head_norm"] if b.decay_rank else 1.0)
            mixed = (o.reshape(T, -1) * torch.nn.functional.silu(gate)) @ t["o"].T
        x = x + mixed + (torch.nn.functional.silu(h @ t["gate"].T) * (h @ t["up"].T)) @ t["down"].T
    return (_rms(x, 1e-6) * final) @ embed.T


# ------------------------------------------------------------------------------------------
# what is measured
# ------------------------------------------------------------------------------------------


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "linear":
        g, x, bias = _linear_inputs(c, seed)
        return kind, _weight(g, c["fmt"], c["n"], c["k"]), x, bias
    if kind == "layers":
        g, xs = _layers_inputs(c, seed)
        return kind, [{p: _weight(g, c["fmt"], n, k) for p, n, k in _projections(c["shape"])} for _ in range(c["layers"])], xs
    if kind == "group":
        x, ws = _group_inputs(c, seed)
        cfg = wq.QuantizationConfig(wq.QuantDtype(c["bits"]), c["group"], False)
        qs = [wq.QuantizedTensor(*w, cfg, [c["n"], c["k"]]) for w in ws]
        for q in qs:
            q.device_weight()
        return kind, qs, x
    if kind == "moe":
        t, x = _moe_inputs(c, seed)
        t = {n: v.cpu().numpy() for n, v in t.items()}
        layout, fmt = (moe.LAYOUT_KN_GPTOSS, QuantFormat.MXFP4_GPTOSS) if c["layout"] == "kn" else (moe.LAYOUT_NK, QuantFormat.MXFP4_SPLIT)
        return kind, moe.MoeBlock(c["experts"], c["hidden"], c["inter"], c["top"], 7.0, t["router_w"], t["router_b"], layout, fmt, t["gate_up"],
                                  t["gate_up_scales"], t["gate_up_bias"], t["down"], t["down_scales"], t["down_bias"]), x
    if kind == "token":
        m = _decoder(c, seed, c["context"] + 8)
        past, token = _cache_inputs(c, seed)
        m.buffers = m.dec.buffers()
        for cache, old in zip(m.buffers, past):
            cache[:, :, :c["context"]] = old
        at, st = c["context"], _stream()
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            m.dec.reset(token, at, st)
            m.dec.step(st)
            st.synchronize()
            m.dec.reset(token, at, st)
            m.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(m.graph, stream=st):
                m.dec.step(torch.cuda.current_stream())
        return kind, m, token, at
    if kind == "prompt":
        m = _decoder(c, seed, c["tokens"] + 8)
        m.buffers = m.dec.buffers()
        return kind, m, _prompt_ids(c, seed, SHAPES[c["shape"]]["vocab"])
    return kind, _block_decoder(c, seed), _prompt_ids(c, seed, _VOCAB), c["tokens"]


def run(state):
    kind = state[0]
    if kind == "linear":
        _, w, x, bias = state
        return api.quantized_linear(x, w, bias)
    if kind == "layers":
        out = []
        for w in state[1]:
            x = state[2]
            out += api.linear_batch([x["x"]] * 3, [w["q"], w["k"], w["v"]])
            out.append(api.quantized_linear(x["a"], w["o"]))
            out += api.linear_batch([x["h"]] * 2, [w["gate"], w["up"]])
            out.append(api.quantized_linear(x["f"], w["down"]))
        return out
    if kind == "group":
        return [wq.quantized_matmul(state[2], w) for w in state[1]]
    if kind == "moe":
        return state[1](state[2])
    if kind == "token":      # the loop of a caller that chooses the tokens itself: token and position in, one replay
        _, m, token, at = state
        m.dec.reset(token, at, _stream())
        with torch.cuda.stream(_stream()):
            m.graph.replay()
        return m.views(at)
    if kind == "prompt":
        _, m, ids = state
        m.dec.prefill(ids, 0)
        return m.views(slice(0, len(ids)))
    _, m, ids, n = state
    out = [m.dec.extend(ids[:n], 0, [n - 1])]
    for i in range(n, len(ids)):
        out.append(m.dec.extend(ids[i:i + 1], i, [0]))
    return np.concatenate(out)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "linear":
        g, x, bias = _linear_inputs(c, seed)
        raw, scales = _blocks(g, c["fmt"], c["n"], c["k"])
        y = x.to(F64) @ _dense(raw, scales, c["fmt"], c["n"], c["k"]).T
        return y if bias is None else y + bias.to(F64)
    if kind == "layers":
        g, xs = _layers_inputs(c, seed)
        out = []
        for _ in range(c["layers"]):
            for p, n, k in _projections(c["shape"]):
                raw, scales = _blocks(g, c["fmt"], n, k)
                out.append(xs[_LAYER_INPUT[p]].to(F64) @ _dense(raw, scales, c["fmt"], n, k).T)
        return out
    if kind == "group":
        x, ws = _group_inputs(c, seed)
        out = []
        for codes, scale, zp in ws:
            if c["bits"] == 4:
                q = torch.stack([codes & 15, codes >> 4], -1).to(torch.int32)
                q = torch.where(q > 7, q - 16, q)
            else:
                q = codes.view(torch.int8).to(torch.int32)
            q = q.reshape(-1, c["group"]).to(F64)
            out.append(x.to(F64) @ ((q - zp.to(F64)[:, None]) * scale.to(F64)[:, None]).reshape(c["n"], c["k"]).T)
        return out
    if kind == "moe":
        return _moe_exact(c, seed)
    if kind == "token":
        past, token = _cache_inputs(c, seed)
        logits, k, v = _qwen3_exact(c, seed, [token], past, c["context"])
        return logits, k[:, :, 0], v[:, :, 0]
    if kind == "prompt":
        return _qwen3_exact(c, seed, _prompt_ids(c, seed, SHAPES[c["shape"]]["vocab"]), None, 0)
    ids = _prompt_ids(c, seed, _VOCAB)
    return _blocks_exact(c, seed, ids)[c["tokens"] - 1:]


_BITS = {"Q8_0": 8.5, "Q4_0": 4.5, "Q4_K": 4.5, "Q6_K": 6.5625, "MXFP4_SPLIT": 4.25}


def work(case):
    c, kind = case, case["kind"]
    if kind == "linear":
        e, n, k, m = (4 if c["x"] == "f32" else 2), c["n"], c["k"], c["m"]
        return {"bytes": n * k * _BITS[c["fmt"]] / 8 + m * (n + k) * e, "flops": 2 * m * n * k}
    if kind == "layers":
        s, m, p = SHAPES[c["shape"]], c["m"], _projections(c["shape"])
        size = sum(n * k for _, n, k in p)
        x = 2 * s["hidden"] + s["heads"] * 128 + s["ffn"]
        return {"bytes": c["layers"] * (size * _BITS[c["fmt"]] / 8 + m * 2 * sum(n for _, n, _ in p)) + 2 * m * x, "flops": c["layers"] * 2 * m * size}
    if kind == "group":
        n, k, m = c["n"], c["k"], c["m"]
        return {"bytes": c["count"] * (n * k * c["bits"] / 8 + n * k / c["group"] * 8 + 4 * m * n) + m * k * (4 if c["x"] == "f32" else 2),
                "flops": c["count"] * 2 * m * n * k}
    if kind == "moe":
        E, H, I, T = c["experts"], c["hidden"], c["inter"], c["tokens"]
        used = E * (1 - (1 - c["top"] / E) ** T)                # experts that some token takes, on average
        return {"bytes": used * 3 * H * I * 4.25 / 8 + T * H * 6 + E * H * 4, "flops": T * c["top"] * 6 * H * I + 2 * T * E * H}
    if kind == "blocks":
        D, attention, rec = c["width"], (3 * c["heads"] + 2 * c["kv"]) * 128, c["rec"] * (2 * 128 + 3 * 256)
        size = D * (attention + 3 * rec + 4 * 3 * c["ffn"])
        total, T, n = 2 * size + 2 * D * _VOCAB, c["tokens"], 1 + c["steps"]
        seen = sum(min(i + 1, c["window"]) for i in range(T + c["steps"]))
        return {"bytes": n * total + n * 4 * _VOCAB, "flops": 2 * size * (T + c["steps"]) + 4 * seen * c["heads"] * 128
                + 3 * (T + c["steps"]) * c["rec"] * 128 * 256 * 4 + 2 * n * D * _VOCAB}
    s = SHAPES[c["shape"]]
    size = sum(n * k for _, n, k in _projections(c["shape"]))
    head, kv = s["vocab"] * s["hidden"], c["layers"] * s["kv"] * 128 * 4 * 2
    T, seen = (1, c["context"] + 1) if kind == "token" else (c["tokens"], c["tokens"] * (c["tokens"] + 1) / 2)
    return {"bytes": c["layers"] * size * 4.5 / 8 + head * 6.5625 / 8 + kv * ((c["context"] if kind == "token" else 0) + T) + 4 * s["vocab"],
            "flops": 2 * c["layers"] * size * T + 2 * head + 4 * c["layers"] * s["heads"] * 128 * seen}


def tolerance(case):
    """About four times what the paths are off `exact` by: sums of products of f32 (or of 16-bit numbers, not rounded
    again) in 32 bits where so few rows take them, bf16 operands and results elsewhere. The decoders round to bf16 four
    times a layer: 36 layers leave 1.9e-2 of the logits, eight 1.2e-2, the four mixed blocks 5e-3."""
    c, kind = case, case["kind"]
    few = (kind == "linear" and c["x"] == "f32" and c["m"] <= 8 or kind == "group" and c["m"] <= 16
           or kind == "moe" and c["tokens"] * c["top"] < 32 * c["experts"])
    return {"rel": 2e-5 if few else 3e-2 if kind in ("token", "prompt") else 2e-2 if kind == "blocks" else 1e-2}
