"""Decode step of a Qwen3-shaped decoder whose norms, rotation, activation and residual sums are parts of the kernels around them,
against the same step with kernels of their own (a forced product path): every head group, contexts around the batches of 16 keys
and where a warp takes a second batch (148 warps per key / value head). The two differ in the rounding of the normed rows, bf16
(2^-9) on one side and f16 on the other: a product of such rows differs by less than 2^-9 of its magnitudes, three products follow
one another, so 1e-2 in the 2-norm."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from nn_b200 import api, decoder
from nn_b200 import formats as F
from nn_b200.formats import QuantFormat as Q

pytestmark = pytest.mark.gpu
HIDDEN, FFN, VOCAB = 2048, 2304, 320


def _model(heads, kv, layers, max_seq, HIDDEN=HIDDEN):
    b, rng = api.gpu_backend(), np.random.default_rng(heads + kv)
    dec = decoder.Decoder(b, decoder.DecoderConfig(hidden=HIDDEN, n_heads=heads, n_kv_heads=kv, ffn=FFN, n_layers=layers, vocab=VOCAB, max_seq=max_seq,
                                                   act_dtype=api.BF16))

    def weight(n, k):
        w = rng.standard_normal((n, k)).astype(np.float32) / np.sqrt(np.float32(k))
        blocks, _ = api.quantize(torch.from_numpy(w).cuda(), Q.Q4_K_GGML, b)
        return api.DeviceWeight.from_device(b, Q.Q4_K_GGML, blocks, n, k)

    norm = lambda n: (1.0 + 0.1 * rng.standard_normal(n)).astype(np.float32)  # noqa: E731
    q, k = heads * 128, kv * 128
    for i in range(layers):
        ws = [weight(*s) for s in ((q, HIDDEN), (k, HIDDEN), (k, HIDDEN), (HIDDEN, q), (FFN, HIDDEN), (FFN, HIDDEN), (HIDDEN, FFN))]
        dec.set_layer(i, *ws, norm(HIDDEN), norm(HIDDEN), norm(128), norm(128))
    embed = torch.from_numpy(rng.standard_normal((VOCAB, HIDDEN)).astype(np.float32)).to(torch.bfloat16).cuda()
    dec.set_head(embed, norm(HIDDEN), weight(VOCAB, HIDDEN))
    return dec


@pytest.mark.parametrize("heads,kv", [(2, 2), (16, 8), (16, 4), (16, 2)])
def test_against_separate_kernels(heads, kv):
    contexts = [0, 1, 15, 16, 17, 100, 2366, 2367, 2368, 2384, 5000]
    dec, b = _model(heads, kv, 2, 5002), api.gpu_backend()
    keys, values, logits = dec.buffers()[:3]
    g = torch.Generator(device="cuda").manual_seed(3)
    past = [torch.randn(keys.shape, device="cuda", generator=g) for _ in range(2)]
    for at in contexts:
        got = []
        for path in (api.PATH_AUTO, api.PATH_SKINNY):
            keys[:], values[:] = past
            b.set_path(path)
            try:
                dec.reset(7, at)
                before = b.launch_count()
                dec.step()
                launches = b.launch_count() - before
            finally:
                b.set_path(api.PATH_AUTO)
            torch.cuda.synchronize()
            b.device_status()
            got.append((launches, logits[:].clone(), keys[:, :, at].clone(), values[:, :, at].clone()))
            assert torch.equal(keys[:, :, :at], past[0][:, :, :at]) and torch.equal(values[:, :, at + 1:], past[1][:, :, at + 1:])
        assert got[0][0] < got[1][0]   # (the fused step is what ran)
        for one, other in zip(got[0][1:], got[1][1:]):
            assert float((one - other).norm() / other.norm()) < 1e-2, at
    dec.release()


@pytest.mark.parametrize("heads,kv", [(16, 8), (8, 2)])
def test_wide_rows(heads, kv):
    """More row tiles than the token-column kernel takes for o and down: the one-row kernel adds them to the residual row, from
    eight super-blocks of K on (o of 16 heads), below that the token-column kernel (o of 8 heads)."""
    dec, b, at, got = _model(heads, kv, 2, 64, 4864), api.gpu_backend(), 40, []
    keys, values, logits = dec.buffers()[:3]
    g = torch.Generator(device="cuda").manual_seed(3)
    past = [torch.randn(keys.shape, device="cuda", generator=g) for _ in range(2)]
    for path in (api.PATH_AUTO, api.PATH_SKINNY):
        keys[:], values[:] = past
        b.set_path(path)
        try:
            dec.reset(7, at)
            before = b.launch_count()
            dec.step()
            launches = b.launch_count() - before
        finally:
            b.set_path(api.PATH_AUTO)
        torch.cuda.synchronize()
        b.device_status()
        got.append((launches, logits[:].clone(), keys[:, :, at].clone(), values[:, :, at].clone()))
    assert got[0][0] < got[1][0]
    for one, other in zip(got[0][1:], got[1][1:]):
        assert float((one - other).norm() / other.norm()) < 1e-2
    dec.release()
