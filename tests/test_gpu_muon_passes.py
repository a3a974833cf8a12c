"""The two memory passes of the fused Muon step (gradient -> momentum -> bf16 pack, update -> master and bf16 copy) against torch."""
import pytest
import torch

from gpt_moe_b200.ops import cuda_ops

pytestmark = pytest.mark.gpu


def table(tensors):
    return torch.tensor([t.data_ptr() for t in tensors], dtype=torch.int64, device="cuda")


# inside a tile, edges of tiles in both directions, odd row counts (no 4-byte pairs on the transposed side), a padded pitch
@pytest.mark.parametrize("rows,cols,pad", [(8, 4, 0), (64, 64, 0), (66, 68, 4), (63, 72, 0), (200, 132, 8), (129, 60, 0), (768, 768, 0)])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("nesterov", [False, True])
def test_prepare_and_apply(rows, cols, pad, transpose, nesterov):
    torch.manual_seed(rows + cols)
    n, ext = 3, cuda_ops.ext()
    grads, bufs, weights = ([torch.randn(rows, cols + pad, device="cuda") for _ in range(n)] for _ in range(3))
    copies = [torch.full((rows, cols + pad), 7.0, device="cuda", dtype=torch.bfloat16) for _ in range(n)]
    before = [b.clone() for b in bufs]
    if (rows * cols) % 8 == 0:
        packed = torch.empty((n, cols, rows) if transpose else (n, rows, cols), device="cuda", dtype=torch.bfloat16)
        sumsq = torch.zeros(n, device="cuda")
        ext.rs_muon_prepare(table(grads), table(bufs), packed, sumsq, rows, cols, cols + pad, cols + pad, 0.95, nesterov, transpose, [0], False)
        for i in range(n):
            g = grads[i][:, :cols]
            want = before[i][:, :cols] * 0.95 + g
            assert torch.allclose(bufs[i][:, :cols], want, rtol=1e-6, atol=1e-6)          # one fused multiply-add against two roundings
            assert torch.equal(bufs[i][:, cols:], before[i][:, cols:])
            u = g + 0.95 * bufs[i][:, :cols] if nesterov else bufs[i][:, :cols]
            got = (packed[i].t() if transpose else packed[i]).float()
            assert torch.allclose(got, u, rtol=2 ** -8, atol=1e-6)                         # one rounding to bf16
            assert abs(sumsq[i].item() - packed[i].double().pow(2).sum().item()) < 1e-4 * sumsq[i].item()
    update = torch.randn((n, cols, rows) if transpose else (n, rows, cols), device="cuda").bfloat16()
    old = [w.clone() for w in weights]
    ext.muon_apply_push(table(weights), table(copies), update, rows, cols, cols + pad, cols + pad, -0.02, transpose, [0])
    for i in range(n):
        o = (update[i].t() if transpose else update[i]).float()
        assert torch.allclose(weights[i][:, :cols], old[i][:, :cols] - 0.02 * o, rtol=1e-6, atol=1e-6)
        assert torch.equal(weights[i][:, cols:], old[i][:, cols:]) and (copies[i][:, cols:] == 7.0).all()
        assert torch.equal(copies[i][:, :cols], weights[i][:, :cols].bfloat16())
