"""Products with the weights in tensor memory (33..512 bf16 rows, f32 rows from 17): edges of the 128-row weight tiles and of
the token tiles, K of one unit, of several and of a broken one, one to eight ways to split it, every format it reads, and
several products of one call. Against the same product of the decoded weights and the activations rounded to bf16 in 64 bits:
the sums are f32, so what is left is K f32 roundings of partial sums (2^-24 each, of the magnitudes' sum) and, for bf16
results, half a unit of their last place."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from nn_b200 import api
from nn_b200 import formats as F
from nn_b200.formats import QuantFormat as Q
from oracle import cpu as orc

pytestmark = pytest.mark.gpu
FORMATS = [Q.Q4_K, Q.Q4_K_GGML, Q.Q4_0, Q.Q8_0, Q.Q6_K, Q.MXFP4_SPLIT]


def _bf16(a):
    return F.bf16_bits_to_f32(F.to_bf16_bits(np.ascontiguousarray(a))).reshape(a.shape).astype(np.float64)


def _weight(fmt, n, k, seed):
    w, sc = F.gen_weight(fmt, seed, n, k)
    return api.from_quantized(w, fmt, [n, k], sc), _bf16(orc.dequantize(fmt, w, n * k, sc).reshape(n, k))


def _check(y, x, w64, bias, k):
    x64 = _bf16(x)
    ref, mag = x64 @ w64.T, np.abs(x64) @ np.abs(w64).T
    if bias is not None:
        ref, mag = ref + bias, mag + np.abs(bias)
    got = y.double().cpu().numpy()
    bound = (k + 2) * 2.0 ** -24 * mag
    if y.dtype == torch.bfloat16:
        bound = bound * (1 + 2.0 ** -8) + np.abs(ref) * 2.0 ** -8
    assert np.all(np.abs(got - ref) <= bound), np.max(np.abs(got - ref) - bound)


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("n,k,m,x_bf16,y_bf16,bias", [(16, 256, 33, True, True, False), (130, 512, 128, True, False, True), (257, 2304, 129, True, True, True),
                                                      (128, 1024, 300, True, False, False), (40, 768, 17, False, False, True), (129, 2048, 145, False, True, False)])
def test_product(fmt, n, k, m, x_bf16, y_bf16, bias):
    t, w64 = _weight(fmt, n, k, 11)
    x = F.gen_activations(5, m, k, bf16=x_bf16)
    b = (F.Stream(7).normal(n) * 0.5).astype(np.float32) if bias else None
    xt = torch.from_numpy(x).cuda()
    y = api.quantized_linear(xt.to(torch.bfloat16) if x_bf16 else xt, t, torch.from_numpy(b).cuda() if bias else None, out_dtype=torch.bfloat16 if y_bf16 else torch.float32)
    torch.cuda.synchronize()
    t.backend.device_status()
    _check(y, x, w64, b, k)
    t.release()


@pytest.mark.parametrize("k", [64, 192, 320, 2880])
@pytest.mark.parametrize("x_bf16", [True, False])
def test_broken_unit(k, x_bf16):
    t, w64 = _weight(Q.MXFP4_SPLIT, 96, k, 3)
    x = F.gen_activations(4, 37, k, bf16=x_bf16)
    xt = torch.from_numpy(x).cuda()
    y = api.quantized_linear(xt.to(torch.bfloat16) if x_bf16 else xt, t)
    torch.cuda.synchronize()
    t.backend.device_status()
    _check(y, x, w64, None, k)
    t.release()


def test_several_products_of_one_call():
    """Jobs of one input share a launch, another input and another K start their own; results are those of single calls but for the
    rounding of sums (K may be split for all tiles of a launch)."""
    m, pairs = 70, []
    for i, (n, k) in enumerate([(300, 512), (64, 512), (128, 512), (200, 1024)]):
        pairs.append((_weight(Q.Q4_K, n, k, 20 + i), k))
    x = {k: F.gen_activations(k, m, k, bf16=True) for k in (512, 1024)}
    xt = {k: torch.from_numpy(v).cuda().to(torch.bfloat16) for k, v in x.items()}
    ys = api.linear_batch([xt[k] for _, k in pairs], [t for (t, _), _ in pairs], out_dtype=torch.float32)
    torch.cuda.synchronize()
    for y, ((t, w64), k) in zip(ys, pairs):
        _check(y, x[k], w64, None, k)
        one = api.quantized_linear(xt[k], t, out_dtype=torch.float32)
        torch.testing.assert_close(y, one, rtol=0, atol=float(k * 2.0 ** -24 * (np.abs(_bf16(x[k])) @ np.abs(w64).T).max()))   # (K may be split otherwise)
        t.release()

# The steady state: at least five units of 256 weights per CTA. 130 rows: two tiles, K over the eight CTAs of a cluster; 20000
# rows: 157 tiles, one CTA each. The rings of two raw and four operand stages turn at least twice.
@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("n,k,m", [(130, 10496, 37), (130, 10496, 128), (20001, 1280, 40)])
@pytest.mark.parametrize("x_bf16", [True, False])
def test_many_units(fmt, n, k, m, x_bf16):
    if fmt == Q.MXFP4_SPLIT:
        k += 64   # a broken last unit behind whole ones
    t, w64 = _weight(fmt, n, k, 13)
    x = F.gen_activations(6, m, k, bf16=x_bf16)
    xt = torch.from_numpy(x).cuda()
    y = api.quantized_linear(xt.to(torch.bfloat16) if x_bf16 else xt, t, out_dtype=torch.float32)
    torch.cuda.synchronize()
    t.backend.device_status()
    _check(y, x, w64, None, k)
    t.release()


@pytest.mark.parametrize("m", [64, 80, 81, 128, 160, 161, 241])
def test_q8_0_tiles_of_f32_rows(m):
    """Up to 80 tokens per tile, tiles of equal size, the last one ragged."""
    t, w64 = _weight(Q.Q8_0, 130, 1536, 17)
    x = F.gen_activations(8, m, 1536, bf16=False)
    y = api.quantized_linear(torch.from_numpy(x).cuda(), t)
    torch.cuda.synchronize()
    t.backend.device_status()
    _check(y, x, w64, None, 1536)
    t.release()
