"""Large products on decoded weights: tiles of 256 x 256 by pairs of CTAs, of 128 x 256 and 128 x 128 by single ones, with edges
that leave the second CTA of a pair without rows or without weights. Against 64 bits: products of bf16 values are exact in f32,
so K roundings of partial sums are left (2^-24 each, of the magnitudes' sum) and, for bf16 results, half a unit of the last
place."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import rugesun_models as M
from nn_b200 import api, models
from nn_b200 import formats as F
from nn_b200.formats import QuantFormat as Q
from oracle import rugesun_ref as ref

pytestmark = pytest.mark.gpu


# rows and columns behind the last whole tile of 256: rows 1 and 76, columns 1, 40, 128 (a pair's second CTA has none); 129, 195, 255
@pytest.mark.parametrize("m,n", [(1025, 2817), (1100, 2600), (1281, 2500), (1153, 2755), (1535, 2689), (1281, 9000), (257, 12200), (300, 520), (640, 2815)])
@pytest.mark.parametrize("k", [64, 448])
@pytest.mark.parametrize("y_bf16,bias", [(False, False), (True, True)])
def test_product(m, n, k, y_bf16, bias):
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    w = torch.randn(n, k, device="cuda", generator=g).to(torch.bfloat16)
    x = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    b = torch.randn(n, device="cuda", generator=g) if bias else None
    t = api.DeviceWeight.from_device(api.gpu_backend(), Q.BF16_DENSE, w.view(torch.uint8).reshape(-1), n, k)
    y = api.quantized_linear(x, t, b, out_dtype=torch.bfloat16 if y_bf16 else torch.float32)
    torch.cuda.synchronize()
    t.backend.device_status()
    want, mag = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    if bias:
        want, mag = want + b.double(), mag + b.double().abs()
    bound = (k + 2) * 2.0 ** -24 * mag
    if y_bf16:
        bound = bound * (1 + 2.0 ** -8) + want.abs() * 2.0 ** -8
    assert bool(((y.double() - want).abs() <= bound).all())
    t.release()


@pytest.mark.parametrize("fmt,m", [(Q.Q4_K, 1025), (Q.Q6_K, 1281), (Q.Q8_0, 4100)])
def test_product_of_a_decoded_weight(fmt, m):
    """Both operands inside half of the L2 cache take single CTAs with 128 x 256 in their first wave, 4100 rows pairs."""
    n, k = 2817, 512
    raw, sc = F.gen_weight(fmt, 5, n, k)
    t = api.from_quantized(raw, fmt, [n, k], sc)
    w = t.dequantize().to(torch.bfloat16).double()
    x = torch.randn(m, k, device="cuda", generator=torch.Generator(device="cuda").manual_seed(m)).to(torch.bfloat16)
    y = api.quantized_linear(x, t, out_dtype=torch.float32)
    torch.cuda.synchronize()
    t.backend.device_status()
    want, mag = x.double() @ w.T, x.double().abs() @ w.abs().T
    assert bool(((y.double() - want).abs() <= (k + 2) * 2.0 ** -24 * mag).all())
    t.release()


def test_activation_in_the_epilogue_of_pairs(tmp_path):
    """800 rows through a feed-forward block of 1330: 4 x 11 tiles of pairs, the last without rows and without weights for their
    second CTA."""
    cfg = M.config([M.layer(heads=2, dim=32, rot_dim=16, vdim=32, window=40, mlp={"kind": "dense", "ff": 1330})], width=64, vocab=160)
    t = M.tensors(cfg, seed=9)
    ids = np.random.default_rng(2).integers(0, cfg["vocab"], 800).tolist()
    want = ref.forward(cfg, t, ids, np.float32)
    folder = tmp_path / "model"
    folder.mkdir()
    M.write_folder(folder, cfg, t)
    dec = models.load_model(str(folder), max_seq=800, act_dtype=api.BF16)
    d = dec.extend(ids, 0, list(range(len(ids)))).astype(np.float64) - want
    # (bf16 inputs of a layer's products on both ways: the bar of the bf16 tests of these models, at every row)
    assert np.max(np.sqrt((d * d).mean(-1))) <= 4e-2 * np.sqrt((want * want).mean())
    dec.release()
