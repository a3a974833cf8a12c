"""MXFP8 products with a short contraction (`gemm_mxfp8_resident_kernel`) against the expanded operands."""
import pytest
import torch

from gpt_moe_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.float() - b).norm() / b.norm()).item()


# one strip and fewer tiles than CTA pairs; K of one block and of the most that stay resident; ragged rows and a last tile of 112 and of 176
# columns; ranges of a pair that begin and end inside a row and span several rows
@pytest.mark.parametrize("m,n,k", [(128, 384, 128), (300, 576, 1024), (129, 1840, 896), (520, 496, 256), (9000, 768, 768), (20001, 2288, 640)])
def test_resident_products(m, n, k):
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(4)
    c = cuda_ops.ext()
    a = torch.randn(m, k, device="cuda").bfloat16()
    b = (torch.randn(n, k, device="cuda") * torch.logspace(-2, 2, n, device="cuda")[:, None]).bfloat16()      # every row of B needs scales of its own
    (aq, asf), (bq, bsf) = c.mxfp8_quantize(a), c.mxfp8_quantize(b)
    d = torch.full((m + 1, n), 7.0, device="cuda", dtype=torch.bfloat16)
    c.gemm_mxfp8(aq, asf, bq, bsf, d[:m], 0.5)
    want = 0.5 * ref.mxfp8_linear(a.float(), b.float())
    assert rel(d[:m], want) < 4e-3                                    # one rounding to bf16
    columns = ((d[:m].float() - want).norm(dim=0) / want.norm(dim=0)).max().item()
    assert columns < 6e-3                                             # in every column: none took the scales of another
    assert (d[m] == 7.0).all()
    cuda_ops.check_status()


def test_resident_products_by_expert():
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(5)
    c = cuda_ops.ext()
    counts, e, n, k = [256, 0, 1280, 512, 0, 256], 6, 1536, 384
    rows = sum(counts)
    x = torch.randn(rows + 512, k, device="cuda").bfloat16()
    w = torch.randn(e, n, k, device="cuda").bfloat16()
    tiles = torch.tensor(sum([[i] * (cnt // 128) for i, cnt in enumerate(counts)], []) + [0] * 4, dtype=torch.int32, device="cuda")
    meta = torch.tensor([rows // 128, rows], dtype=torch.int32, device="cuda")
    (xq, xsf), (wq, wsf) = c.mxfp8_quantize(x, meta[1:2]), c.mxfp8_quantize(w)
    y = torch.zeros(rows + 512, n, device="cuda", dtype=torch.bfloat16)
    c.gemm_mxfp8(xq, xsf, wq, wsf, y, 1.0, tiles, meta)
    first = 0
    for i, cnt in enumerate(counts):
        if cnt:
            assert rel(y[first: first + cnt], ref.mxfp8_linear(x[first: first + cnt].float(), w[i].float())) < 4e-3
        first += cnt
    assert y[rows:].abs().max().item() == 0.0                         # tiles beyond num_m_tiles are not written
    cuda_ops.check_status()
