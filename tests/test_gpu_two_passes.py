"""Batches of products of 17 to 32 bf16 rows (9 to 16 f32 rows), whose two passes go out together, against each product alone: the same
kernel and order of sums, so the same bits; where one row is left for the second pass a batch may choose the one-row kernel, whose
sums come in another order: K 2^-24 of their magnitudes, 1e-5 in the 2-norm."""
import pytest

torch = pytest.importorskip("torch")

from nn_b200 import api
from nn_b200 import formats as F
from nn_b200.formats import QuantFormat as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [Q.Q4_K, Q.Q8_0, Q.Q6_K, Q.MXFP4_SPLIT])
@pytest.mark.parametrize("dtype,m", [(torch.bfloat16, m) for m in (17, 18, 31, 32)] + [(torch.float32, m) for m in (9, 10, 16)])
def test_batch_matches_single_products(fmt, dtype, m):
    b, k = api.gpu_backend(), 1024
    ws = []
    for i, n in enumerate((512, 40, 16)):
        data, scales = F.gen_weight(fmt, 3 + i, n, k)
        ws.append(api.DeviceWeight.from_device(b, fmt, torch.from_numpy(data).cuda(), n, k, None if scales is None else torch.from_numpy(scales).cuda()))
    x = torch.from_numpy(F.gen_activations(5, m, k, bf16=True)).cuda().to(dtype)
    before = b.launch_count()
    got = api.linear_batch([x] * 3, ws, out_dtype=torch.float32)
    launches = b.launch_count() - before
    want = [api.linear_batch([x], [w], out_dtype=torch.float32)[0] for w in ws]
    torch.cuda.synchronize()
    b.device_status()
    assert launches == 2
    for y, r in zip(got, want):
        if m in (17, 9):
            assert float((y.double() - r.double()).norm() / r.double().norm()) < 1e-5
        else:
            assert torch.equal(y, r)
