"""Prompt pass of a Qwen3-shaped decoder with bf16 product inputs at the sizes where its attention changes form: below and
from 32 query vectors per key / value head, around the edges of 128-vector and 64-key tiles, every size of head group, in
one portion and in two."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from nn_b200 import api, decoder
from nn_b200 import formats as F
from nn_b200.formats import QuantFormat as Q
from oracle import qwen3_ref as ref

pytestmark = pytest.mark.gpu
FFN, VOCAB, EPS = 192, 160, 1e-6


def _model(group, count, hidden=128, shift=0):
    HIDDEN = hidden
    rng = np.random.default_rng(100 + group)
    kv = 2 if group < 8 else 1
    cfg = decoder.DecoderConfig(hidden=HIDDEN, n_heads=kv * group, n_kv_heads=kv, ffn=FFN, n_layers=2, vocab=VOCAB, max_seq=count + 3, act_dtype=api.BF16)
    dec, b = decoder.Decoder(api.gpu_backend(), cfg), api.gpu_backend()

    def weight(n, k):
        w = torch.from_numpy(rng.standard_normal((n, k)).astype(np.float32) / np.sqrt(k).astype(np.float32)).to(torch.bfloat16).cuda()
        return api.DeviceWeight.from_device(b, Q.BF16_DENSE, w.view(torch.uint8).reshape(-1), n, k), w.float().cpu().numpy()

    norm = lambda n: (1.0 + 0.1 * rng.standard_normal(n)).astype(np.float32)  # noqa: E731
    model = {"layers": [], "cfg": cfg}
    q, k = cfg.n_heads * 128, kv * 128
    for i in range(cfg.n_layers):
        ws = [weight(n, m) for n, m in ((q, HIDDEN), (k, HIDDEN), (k, HIDDEN), (HIDDEN, q), (FFN, HIDDEN), (FFN, HIDDEN), (HIDDEN, FFN))]
        ns = [norm(HIDDEN), norm(HIDDEN), norm(128), norm(128)]
        dec.set_layer(i, *[w for w, _ in ws], *ns)
        model["layers"].append(([f for _, f in ws], ns))
    embed = torch.empty(VOCAB * HIDDEN + shift, dtype=torch.bfloat16, device="cuda")[shift:].view(VOCAB, HIDDEN)   # (rows off their 8-byte boundaries)
    embed.copy_(torch.from_numpy(rng.standard_normal((VOCAB, HIDDEN)).astype(np.float32)))
    head, model["head"] = weight(VOCAB, HIDDEN)
    model["head_weight"] = head
    model["embed"], model["final"] = embed.float().cpu().numpy(), norm(HIDDEN)
    dec.set_head(embed, model["final"], head)
    return dec, model


def _forward(model, ids):
    """All rows at once in f32, the products' inputs rounded to bf16 as the decoder rounds them."""
    c, T, r = model["cfg"], len(ids), ref.bf16_round
    cos, sin = ref.rope_tables(128, T, c.rope_theta)
    h = model["embed"][ids]
    for (q, k, v, o, g, u, d), (n1, n2, nq, nk) in model["layers"]:
        x = r(ref.rms_norm(h, n1, EPS))
        Q_ = ref.rotate(ref.rms_norm((x @ q.T).reshape(T, -1, 128), nq, EPS), cos[:, None], sin[:, None])
        K = ref.rotate(ref.rms_norm((x @ k.T).reshape(T, -1, 128), nk, EPS), cos[:, None], sin[:, None])
        V = (x @ v.T).reshape(T, -1, 128)
        out = np.empty_like(Q_)
        for j in range(c.n_heads):
            m = j // (c.n_heads // c.n_kv_heads)
            s = (Q_[:, j] @ K[:, m].T) / np.sqrt(np.float32(128))
            s[np.triu_indices(T, 1)] = -np.inf
            p = np.exp(s - s.max(1, keepdims=True))
            out[:, j] = (p / p.sum(1, keepdims=True)) @ V[:, m]
        h = h + r(out.reshape(T, -1)) @ o.T
        x = r(ref.rms_norm(h, n2, EPS))
        gate = x @ g.T
        h = h + r(gate / (1 + np.exp(-gate)) * (x @ u.T)) @ d.T
    return r(ref.rms_norm(h, model["final"], EPS)) @ model["head"].T


@pytest.mark.parametrize("group", [1, 2, 4, 8])
@pytest.mark.parametrize("count", [3, 7, 8, 31, 33, 64, 65, 130])
def test_prompt_rows_of_every_group_size(group, count):
    dec, model = _model(group, count)
    ids = np.random.default_rng(count).integers(0, VOCAB, count)
    want = _forward(model, ids)
    for cut in (0, count // 3):
        got = np.concatenate([dec.extend(ids[a:e], a, list(range(e - a))) for a, e in ((0, cut), (cut, count)) if e > a])
        # both sides round the same five inputs of a layer's products to bf16: the bar of the decoder's bf16 tests
        assert np.max(np.abs(got - want)) <= 1e-2 * np.max(np.abs(want)), (cut, np.max(np.abs(got - want)) / np.max(np.abs(want)))
    dec.backend.device_status()
    dec.release()


@pytest.mark.parametrize("hidden,shift", [(128, 1), (4096, 0), (4352, 0), (8192, 0), (8448, 0)])
def test_norm_of_prompt_rows_of_every_width(hidden, shift):
    """Row norms with the row in registers (up to 4096 and up to 8192 wide) and in two passes (wider, or an odd table)."""
    dec, model = _model(2, 9, hidden, shift)
    ids = np.random.default_rng(hidden).integers(0, VOCAB, 9)
    want, got = _forward(model, ids), dec.extend(ids, 0, list(range(9)))
    assert np.max(np.abs(got - want)) <= 1e-2 * np.max(np.abs(want)), np.max(np.abs(got - want)) / np.max(np.abs(want))
    dec.backend.device_status()
    dec.release()


def test_a_value_that_is_no_number_reaches_no_earlier_block_of_rows():
    """The f32 kernel multiplies masked values of its own block of 16 / group rows with zero and no others: rows in front of the
    block that holds a NaN are those of a prompt without it, also where the tensor cores take 32 and more of them at once."""
    group, count, at = 4, 100, 70
    dec, model = _model(group, count)
    ids = np.random.default_rng(5).integers(0, VOCAB - 1, count)
    ids[at] = VOCAB - 1
    want = _forward(model, ids)
    first = at // (16 // group) * (16 // group)
    bad = model["embed"].copy()
    bad[VOCAB - 1] = np.nan
    dec.set_head(torch.from_numpy(bad).to(torch.bfloat16).cuda(), model["final"], model["head_weight"])
    got = dec.extend(ids, 0, list(range(count)))
    assert np.all(np.isnan(got[at:]))
    assert np.max(np.abs(got[:first] - want[:first])) <= 1e-2 * np.max(np.abs(want[:first]))
    dec.backend.device_status()
    dec.release()


def test_many_blocks_of_rows_of_a_head_with_a_value_that_is_no_number():
    """More blocks of 16 / group rows than the f32 kernel has warps for a kv head at a time."""
    group, count, at = 8, 2500, 2100
    dec, model = _model(group, count)
    ids = np.random.default_rng(5).integers(0, VOCAB - 1, count)
    ids[at] = VOCAB - 1
    want = _forward(model, ids)
    bad = model["embed"].copy()
    bad[VOCAB - 1] = np.nan
    dec.set_head(torch.from_numpy(bad).to(torch.bfloat16).cuda(), model["final"], model["head_weight"])
    got = dec.extend(ids, 0, list(range(count)))
    assert np.all(np.isnan(got[at:]))
    assert np.max(np.abs(got[:at] - want[:at])) <= 1e-2 * np.max(np.abs(want[:at]))
    dec.backend.device_status()
    dec.release()


def test_operand_tiles_of_some_heads_at_a_time():
    """A longer context behind a short one (the room for the operand tiles grows), and the same with memory for one of the two kv heads
    at a time: the same bits."""
    rows, pos, got = 64, 16000, []
    ids = np.random.default_rng(7).integers(0, VOCAB, rows)
    for short in (False, True):
        dec, _ = _model(4, pos + rows)
        keys, values = dec.buffers()[:2]
        dec.prefill(ids, 0)
        g = torch.Generator(device="cuda").manual_seed(3)
        for c in (keys, values):
            c[:, :, :pos] = torch.randn((*c.shape[:2], pos, 128), device="cuda", generator=g)
        torch.cuda.synchronize()
        hog = None
        if short:   # (64 KB of tiles per head and 64 positions: 16.1 MB for one, 32.1 for both)
            torch.cuda.empty_cache()
            hog = torch.empty(torch.cuda.mem_get_info()[0] - (26 << 20), dtype=torch.uint8, device="cuda")
        dec.prefill(ids, pos)
        torch.cuda.synchronize()
        dec.backend.device_status()
        del hog
        torch.cuda.empty_cache()
        got.append([c[1, :, pos:pos + rows].clone() for c in (keys, values)])
        dec.release()
    for one, other in zip(*got):
        assert torch.isfinite(one).all() and torch.equal(one, other)


def test_values_that_cancel_keep_their_f32_digits():
    """Keys of zero give every visible value the same weight; two tokens whose values are opposite but for 2^-15 of them alternate,
    so that every second row's mean consists of the values' last bits. Two f16 terms hold a value to 2^-23, and each of the up to
    12 sums of a tile is rounded at 2^-23 of the values at most: 2^-19 of the mean magnitude in all (two bf16 terms would be up to
    2^-17 off). The output is rounded to bf16 twice on its way to the logits."""
    rng = np.random.default_rng(3)
    count, hidden, half = 100, 128, 64
    cfg = decoder.DecoderConfig(hidden=hidden, n_heads=4, n_kv_heads=1, ffn=64, n_layers=1, vocab=VOCAB, max_seq=count, act_dtype=api.BF16)
    b = api.gpu_backend()
    dec = decoder.Decoder(b, cfg)

    def weight(w):
        return api.DeviceWeight.from_device(b, Q.BF16_DENSE, torch.from_numpy(w.astype(np.float32)).to(torch.bfloat16).cuda().view(torch.uint8).reshape(-1), *w.shape)

    pick = np.zeros((hidden, 512))        # rows 64 .. 127 of the model take the first 64 dimensions of head 0
    pick[half + np.arange(half), np.arange(half)] = 1
    ws = [rng.standard_normal((512, hidden)), rng.standard_normal((128, hidden)), rng.standard_normal((128, hidden)), pick,
          np.zeros((64, hidden)), np.zeros((64, hidden)), np.zeros((hidden, 64))]
    dec.set_layer(0, *[weight(w) for w in ws], np.ones(hidden, np.float32), np.ones(hidden, np.float32), np.ones(128, np.float32), np.zeros(128, np.float32))
    embed = np.zeros((VOCAB, hidden), np.float32)
    embed[0, :half] = F.bf16_bits_to_f32(F.to_bf16_bits(rng.standard_normal(half).astype(np.float32)))
    embed[0, 0] = 2.0 ** -5
    embed[1] = -embed[0]
    embed[1, 0] *= 1 + 2.0 ** -6
    head = np.zeros((VOCAB, hidden))
    head[np.arange(half), half + np.arange(half)] = 1
    dec.set_head(torch.from_numpy(embed).to(torch.bfloat16).cuda(), np.ones(hidden, np.float32), weight(head))
    ids = np.arange(count) % 2
    got = dec.extend(ids, 0, list(range(count)))[:, :half].astype(np.float64)
    v = dec.buffers()[1][0, 0, :count, :half].cpu().numpy().astype(np.float64)
    mean = np.cumsum(v, 0) / np.arange(1, count + 1)[:, None]
    h = embed[ids].astype(np.float64)
    rms = np.sqrt((np.sum(h * h, 1) + np.sum(mean * mean, 1)) / hidden + cfg.rms_eps)
    even = np.arange(1, count, 2)
    assert np.max(np.abs(mean[even])) < 2.0 ** -12 * np.max(np.abs(v))
    bound = 2.0 ** -19 * np.mean(np.abs(v), 0) + 2.0 ** -7 * np.abs(mean)
    assert np.all((np.abs(got * rms[:, None] - mean) <= bound)[even]), np.max((np.abs(got * rms[:, None] - mean) / bound)[even])
    dec.backend.device_status()
    dec.release()
