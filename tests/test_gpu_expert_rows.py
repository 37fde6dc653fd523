"""Expert products with chosen numbers of routed rows per expert: none, one, the edges of the 32-column steps and of the 256-row tiles of
the prefill-sized product, and a reduction too long for the decode-sized kernel to hold its activations at once. Against float64 of the
oracle's weights; the bound counts the roundings: gate and up sums carry 2^-20 of their magnitudes (exact weights: MXFP4 in bf16) or
2^-8 (weights rounded to bf16 or f16 digits of their scales), |d silu| <= 1.1, h is rounded to bf16 (2^-8 with the rounding of the
down product's operands) and the second product adds as the first."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from nn_b200 import api, moe
from nn_b200 import formats as F
from nn_b200.formats import QuantFormat as Q
from test_gpu_moe import _make

pytestmark = pytest.mark.gpu


def _check(layout, fmt, counts, H, I, dtype, limit=7.0):
    E = len(counts)
    rw, rb, gu, gus, bgu, dn, dns, bd, w_gu, w_d = _make(layout, fmt, E, H, I, 31, fast=fmt in (Q.MXFP4_SPLIT, Q.MXFP4_GPTOSS))
    own = np.repeat(np.arange(E), counts)
    np.random.default_rng(5).shuffle(own)
    x = F.gen_activations(9, own.size, H, bf16=True)
    x[:, :E] = 0.0
    x[np.arange(own.size), own] = 4.0
    rw = np.zeros_like(rw)
    rw[np.arange(E), np.arange(E)] = 10.0
    blk = moe.MoeBlock(E, H, I, 1, limit, rw, np.zeros_like(rb), layout, fmt, gu, gus, bgu, dn, dns, bd)
    got = blk(torch.from_numpy(x).cuda().to(dtype)).double()
    torch.cuda.synchronize()
    api.gpu_backend().device_status()
    blk.release()
    exact = 2.0**-20 if fmt in (Q.MXFP4_SPLIT, Q.MXFP4_GPTOSS) else 2.0**-8
    for e in range(E):
        rows = np.flatnonzero(own == e)
        if not rows.size:
            continue
        xe, wg, wd = (torch.from_numpy(np.ascontiguousarray(a)).cuda().double() for a in (x[rows], w_gu[e], w_d[e]))
        gup, mag = xe @ wg + torch.from_numpy(bgu[e]).cuda().double(), exact * (xe.abs() @ wg.abs())
        g, u, eg, eu = gup[:, :I], gup[:, I:], mag[:, :I], mag[:, I:]
        s = (g * torch.sigmoid(g)).clamp(-limit, limit)
        h = s * u
        eh = 1.1 * eg * (u.abs() + eu) + s.abs() * eu + 2.0**-8 * h.abs()
        want = h @ wd + torch.from_numpy(bd[e]).cuda().double()
        bound = eh @ wd.abs() + exact * (h.abs() @ wd.abs()) + 1e-6
        err = ((got[torch.from_numpy(rows).cuda()] - want).abs() / bound).max().item()
        assert err <= 1.0, (e, rows.size, err)


@pytest.mark.parametrize("layout,fmt", [(moe.LAYOUT_NK, Q.MXFP4_SPLIT), (moe.LAYOUT_KN_GPTOSS, Q.MXFP4_GPTOSS), (moe.LAYOUT_NK, Q.Q4_0)])
@pytest.mark.parametrize("counts", [[0, 1, 31, 32, 33, 255, 256, 257, 700, 513, 0], [2050], [0, 0, 640, 1]])
def test_rows_of_prefill_sized_products(layout, fmt, counts):
    _check(layout, fmt, counts, 320, 192, torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("layout,fmt", [(moe.LAYOUT_NK, Q.MXFP4_SPLIT), (moe.LAYOUT_KN_GPTOSS, Q.MXFP4_GPTOSS), (moe.LAYOUT_NK, Q.Q8_0)])
@pytest.mark.parametrize("H,I", [(16384, 128), (128, 16384)])
def test_long_reductions_of_decode_sized_products(H, I, layout, fmt, dtype):
    _check(layout, fmt, [3, 0, 21], H, I, dtype)
