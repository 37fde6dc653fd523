"""Weights decoded to bf16 in front of the large GEMM: identity activations bring the decoded values back, which are the f32 decode
rounded to nearest even, bit for bit. Sizes whose chunks end inside a warp's 64, and whose bytes end inside a 16-byte unit."""
import pytest

torch = pytest.importorskip("torch")

from nn_b200 import api
from nn_b200 import formats as F
from nn_b200.formats import QuantFormat as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt,k", [(Q.Q4_0, 576), (Q.Q8_0, 576), (Q.Q8_0, 640), (Q.Q4_K, 768), (Q.Q4_K_GGML, 768), (Q.Q6_K, 768), (Q.Q4_1, 576), (Q.Q5_K, 768)])
@pytest.mark.parametrize("n", [1, 7, 333, 1040])
def test_values(fmt, k, n):
    b = api.gpu_backend()
    data, _ = F.gen_weight(fmt, n, n, k)
    w = api.DeviceWeight.from_device(b, fmt, torch.from_numpy(data).cuda(), n, k)
    x = torch.eye(k, device="cuda", dtype=torch.bfloat16)   # (more than 512 rows: the decode-once path)
    y = api.linear_batch([x], [w], out_dtype=torch.float32)[0]
    torch.cuda.synchronize()
    b.device_status()
    assert torch.equal(y.T.contiguous(), w.dequantize().view(n, k).to(torch.bfloat16).float())
    w.release()


@pytest.mark.parametrize("fmt,n,k", [(Q.Q4_0, 17001, 576), (Q.Q8_0, 17001, 576), (Q.Q6_K, 12701, 768), (Q.Q8_0, 15169, 640), (Q.Q4_0, 9473, 1024)])
def test_values_of_large_weights(fmt, n, k):
    """Weights of a unit of 64 chunks and more for each of 32 warps per SM, which are decoded through shared memory: chunks that end inside a
    unit, bytes that end inside a 16-byte piece, some warps with one unit and some with two."""
    b = api.gpu_backend()
    assert (n * (k // 32) + 63) // 64 >= 32 * torch.cuda.get_device_properties(0).multi_processor_count
    data, _ = F.gen_weight(fmt, n, n, k)
    w = api.DeviceWeight.from_device(b, fmt, torch.from_numpy(data).cuda(), n, k)
    y = api.linear_batch([torch.eye(k, device="cuda", dtype=torch.bfloat16)], [w], out_dtype=torch.float32)[0]
    torch.cuda.synchronize()
    b.device_status()
    assert torch.equal(y.T.contiguous(), w.dequantize().view(n, k).to(torch.bfloat16).float())
    w.release()
