"""Prompt rows whose gate and up products and activation are one GEMM, against a product each (a forced path): formats, reductions of a
power of two of 32-weight chunks and others, ragged rows and tiles. Both sides round the weights to bf16 (2^-9) and the activation to
bf16; the products differ in the order of their f32 sums alone, the roundings that this moves follow one another through two layers:
1e-2 in the 2-norm."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from nn_b200 import api, decoder
from nn_b200 import formats as F
from nn_b200.formats import QuantFormat as Q

pytestmark = pytest.mark.gpu


def _model(fmt, hidden, ffn, max_seq=720, backend=None):
    """The decoder, and the device memory that setting its layers took."""
    b, rng = backend or api.gpu_backend(), np.random.default_rng(hidden)
    dec = decoder.Decoder(b, decoder.DecoderConfig(hidden=hidden, n_heads=2, n_kv_heads=1, ffn=ffn, n_layers=2, vocab=320, max_seq=max_seq, act_dtype=api.BF16))

    def weight(n, k, f=fmt):
        return api.DeviceWeight.from_device(b, f, torch.from_numpy(F.gen_weight(f, int(rng.integers(1 << 30)), n, k)[0]).cuda(), n, k)

    norm = lambda n: (1.0 + 0.1 * rng.standard_normal(n)).astype(np.float32)  # noqa: E731
    used, ws = 0, [weight(*s) for s in ((256, hidden), (128, hidden), (128, hidden), (hidden, 256), (ffn, hidden), (ffn, hidden), (hidden, ffn, Q.Q8_0))]
    for i in range(2):   # (both layers with the same weights)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        dec.set_layer(i, *ws, norm(hidden), norm(hidden), norm(128), norm(128))
        used += free - torch.cuda.mem_get_info()[0]
    dec.set_head(torch.from_numpy(rng.standard_normal((320, hidden)).astype(np.float32)).to(torch.bfloat16).cuda(), norm(hidden), weight(320, hidden))
    return dec, used


# (the last four large enough to be decoded through shared memory: rows of 18, 24 and 32 chunks)
@pytest.mark.parametrize("fmt,hidden,ffn", [(Q.Q4_K_GGML, 1280, 768), (Q.Q8_0, 576, 704), (Q.Q8_0, 576, 17024), (Q.Q6_K, 768, 12736), (Q.Q4_0, 1024, 9536), (Q.Q8_0, 1024, 9536)])
def test_same_bits_as_separate_products(fmt, hidden, ffn):
    """Both routes form every sum in the same order, round the same values and take the same activation: keys and values of the
    second layer, behind the first one's activation, have the same bits."""
    (dec, _), b = _model(fmt, hidden, ffn), api.gpu_backend()
    tokens = [int(t) for t in np.random.default_rng(3).integers(0, 320, 700)]
    got = []
    for path in (api.PATH_AUTO, api.PATH_TENSOR):
        b.set_path(path)
        try:
            dec.prefill(tokens)
        finally:
            b.set_path(api.PATH_AUTO)
        torch.cuda.synchronize()
        b.device_status()
        got.append([c[1, :, :700].clone() for c in dec.buffers()[:2]])
    for one, other in zip(*got):
        assert torch.isfinite(one).all() and torch.equal(one, other)
    dec.release()


def test_room_for_the_two_weights():
    """Setting the layers takes no room for the decoded pair, nor does a prompt where the context's scratch holds it; where it does not the
    first prompt takes the decoder's own. The same bits from both."""
    b = api.Backend(0)   # (a context whose scratch is as large as its largest weight)
    got, pair = [], 2 * 8192 * 1024 * 2
    tokens = [int(t) for t in np.random.default_rng(3).integers(0, 320, 700)]
    for roomy in (False, True):
        if roomy:
            big = api.DeviceWeight.from_device(b, Q.Q8_0, torch.zeros(16384 * 1024 // 32 * 34, dtype=torch.uint8, device="cuda"), 16384, 1024)
        dec, used = _model(Q.Q4_K_GGML, 1024, 8192, backend=b)
        assert used < pair // 2
        dec.prefill(tokens[:64])    # (the prompt buffers of 1024 rows)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        dec.prefill(tokens)
        torch.cuda.synchronize()
        b.device_status()
        assert (free - torch.cuda.mem_get_info()[0] < pair // 2) == roomy
        got.append([c[1, :, :700].clone() for c in dec.buffers()[:2]])
        dec.release()
    for one, other in zip(*got):
        assert torch.isfinite(one).all() and torch.equal(one, other)
    big.release()


@pytest.mark.parametrize("fmt,hidden,ffn", [(Q.Q4_K_GGML, 1280, 768), (Q.Q6_K, 512, 1280), (Q.Q8_0, 576, 704), (Q.Q4_0, 1024, 1088)])
@pytest.mark.parametrize("count", [513, 700])
def test_against_separate_products(fmt, hidden, ffn, count):
    b, rng = api.gpu_backend(), np.random.default_rng(hidden)
    dec = decoder.Decoder(b, decoder.DecoderConfig(hidden=hidden, n_heads=2, n_kv_heads=1, ffn=ffn, n_layers=2, vocab=320, max_seq=720, act_dtype=api.BF16))

    def weight(n, k, f=fmt):
        return api.DeviceWeight.from_device(b, f, torch.from_numpy(F.gen_weight(f, int(rng.integers(1 << 30)), n, k)[0]).cuda(), n, k)

    norm = lambda n: (1.0 + 0.1 * rng.standard_normal(n)).astype(np.float32)  # noqa: E731
    for i in range(2):
        ws = [weight(*s) for s in ((256, hidden), (128, hidden), (128, hidden))]
        dec.set_layer(i, *ws, weight(hidden, 256), weight(ffn, hidden), weight(ffn, hidden), weight(hidden, ffn, Q.Q8_0), norm(hidden), norm(hidden), norm(128), norm(128))
    dec.set_head(torch.from_numpy(rng.standard_normal((320, hidden)).astype(np.float32)).to(torch.bfloat16).cuda(), norm(hidden), weight(320, hidden))
    tokens = [int(t) for t in rng.integers(0, 320, count)]
    got = []
    for path in (api.PATH_AUTO, api.PATH_TENSOR):
        b.set_path(path)
        try:
            before = b.launch_count()
            dec.prefill(tokens)
            got.append((b.launch_count() - before, dec.buffers()[2].clone()))
        finally:
            b.set_path(api.PATH_AUTO)
    torch.cuda.synchronize()
    b.device_status()
    (n0, l0), (n1, l1) = got
    assert n0 != n1   # (another route)
    assert torch.isfinite(l0).all()
    assert (l0 - l1).norm() <= 1e-2 * l1.norm(), ((l0 - l1).norm() / l1.norm()).item()
