"""Products of one input that share a GEMM (more than 512 bf16 rows, weights of one format behind one another), against each product alone:
every element is the same sum in the same order, so the same bits. Last weights whose rows end inside a tile, a bias for some, a
neighbour that cannot join (another format, a first weight that is no whole number of tiles)."""
import pytest

torch = pytest.importorskip("torch")

from nn_b200 import api
from nn_b200 import formats as F
from nn_b200.formats import QuantFormat as Q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmts,rows,launches", [
    ((Q.Q4_K, Q.Q4_K, Q.Q4_K), (1024, 256, 256), 4), ((Q.Q8_0, Q.Q8_0), (512, 300), 3), ((Q.Q6_K, Q.Q6_K, Q.Q4_K), (768, 40, 512), 5),
    ((Q.Q4_K, Q.Q4_K), (300, 512), 4), ((Q.Q4_0,) * 5, (256,) * 5, 7)])
@pytest.mark.parametrize("m,dt", [(513, torch.float32), (1100, torch.bfloat16)])
def test_against_single_products(fmts, rows, launches, m, dt):
    b, k = api.gpu_backend(), 768
    roomy = api.DeviceWeight.from_device(b, Q.Q8_0, torch.from_numpy(F.gen_weight(Q.Q8_0, 1, 2048, k)[0]).cuda(), 2048, k)   # (scratch for all of them)
    ws = [api.DeviceWeight.from_device(b, f, torch.from_numpy(F.gen_weight(f, 3 + i, n, k)[0]).cuda(), n, k) for i, (f, n) in enumerate(zip(fmts, rows))]
    g = torch.Generator(device="cuda").manual_seed(m)
    x = torch.randn(m, k, device="cuda", generator=g).to(torch.bfloat16)
    biases = [torch.randn(n, device="cuda", generator=g) if i != 1 else None for i, n in enumerate(rows)]
    before = b.launch_count()
    got = api.linear_batch([x] * len(ws), ws, biases=biases, out_dtype=dt)
    assert b.launch_count() - before == launches
    want = [api.linear_batch([x], [w], biases=[c], out_dtype=dt)[0] for w, c in zip(ws, biases)]
    torch.cuda.synchronize()
    b.device_status()
    for y, r in zip(got, want):
        assert torch.equal(y, r)
    for w in ws + [roomy]:
        w.release()
