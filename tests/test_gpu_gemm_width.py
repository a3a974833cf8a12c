"""bf16 products on 128-column tiles (`gemm_bf16_tile_width`) and at the line to 256-column ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def close(got, want):
    # one rounding to bf16 (2^-9 at most) over fp32 sums
    return ((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-3).all()


# one tile, ragged in every direction; a last tile of 8 columns; as many half tiles as pairs, one more column, one more row
@pytest.mark.parametrize("m,n,k", [(1, 136, 64), (300, 264, 200), (360, 2304, 768), (9472, 256, 64), (9472, 264, 64), (9473, 256, 64)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_dense(m, n, k, b_mn):
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(2)
    c = cuda_ops.ext()
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = torch.randn((k, n) if b_mn else (n, k), device="cuda").bfloat16()
    add = torch.randn(m, n, device="cuda").bfloat16()
    wide = torch.full((m + 1, n + 8), 3.0, device="cuda", dtype=torch.bfloat16)
    product = a.double() @ (b.double() if b_mn else b.double().t())
    c.gemm_bf16(a, b, wide[:m, :n], False, b_mn, 0.5)
    assert close(wide[:m, :n], 0.5 * product) and (wide[m] == 3).all() and (wide[:, n:] == 3).all()
    c.gemm_bf16(a, b, wide[:m, :n], False, b_mn, 1.0, -2.0, add)
    assert close(wide[:m, :n], product - 2 * add.double())
    row = torch.randn(1, n, device="cuda").bfloat16()                                 # an addend that the threads read
    c.gemm_bf16(a, b, wide[:m, :n], False, b_mn, 1.0, 1.0, row.expand(m, n))
    assert close(wide[:m, :n], product + row.double())
    cuda_ops.check_status()


def test_batched_and_by_expert():
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(3)
    c = cuda_ops.ext()
    a, b = torch.randn(5, 200, 96, device="cuda").bfloat16(), torch.randn(5, 328, 96, device="cuda").bfloat16()
    d = torch.empty(5, 200, 328, device="cuda", dtype=torch.bfloat16)
    c.gemm_bf16(a, b, d)
    assert close(d, torch.bmm(a.double(), b.double().transpose(1, 2)))
    counts, e, n, k = [256, 0, 512, 256], 4, 640, 136
    rows = sum(counts)
    x, w = torch.randn(rows + 256, k, device="cuda").bfloat16(), torch.randn(e, n, k, device="cuda").bfloat16()
    tiles = torch.tensor(sum([[i] * (cnt // 128) for i, cnt in enumerate(counts)], []) + [0, 0], dtype=torch.int32, device="cuda")
    meta = torch.tensor([rows // 128, rows], dtype=torch.int32, device="cuda")
    y = torch.zeros(rows + 256, n, device="cuda", dtype=torch.bfloat16)
    c.gemm_bf16(x, w, y, False, False, 1.0, 0.0, None, False, 1, tiles, meta)
    expert = torch.tensor(sum([[i] * cnt for i, cnt in enumerate(counts)], []), device="cuda")
    assert close(y[:rows], torch.einsum("rk,rnk->rn", x[:rows].double(), w.double()[expert]))
    assert y[rows:].abs().max().item() == 0.0                                       # tiles beyond num_m_tiles are not written
    cuda_ops.check_status()
