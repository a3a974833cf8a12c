"""D = alpha A B^T + beta C: the addend fetched by TMA against fp64 (edges of tiles and of the 64-column rounds, batches, symmetric results)."""
import pytest
import torch

from gpt_moe_b200.ops import cuda_ops

pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm()).item()


@pytest.mark.parametrize("batch,m,n,k", [(1, 8, 8, 8), (1, 130, 264, 64), (2, 256, 256, 192), (3, 384, 72, 128), (5, 520, 1096, 72), (40, 768, 768, 64)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_addend(batch, m, n, k, b_mn):
    torch.manual_seed(2)
    a, c = torch.randn(batch, m, k, device="cuda").bfloat16(), torch.randn(batch, m, n, device="cuda").bfloat16()
    b = torch.randn(batch, n, k, device="cuda").bfloat16()
    d = torch.empty(batch, m, n, device="cuda", dtype=torch.bfloat16)
    want = 0.7 * (a.double() @ b.double().transpose(1, 2)) - 1.3 * c.double()
    ext = cuda_ops.ext()
    ext.gemm_bf16(a, b.transpose(1, 2).contiguous() if b_mn else b, d, False, b_mn, 0.7, -1.3, c)
    assert rel(d, want) < 3e-3                                   # fp32 accumulation, one rounding to bf16 (1.1e-3 on average)
    wide = torch.full((batch, m, n + 8), float("nan"), device="cuda", dtype=torch.bfloat16)       # addend with a row pitch of its own
    wide[..., :n] = c
    again = torch.empty_like(d)
    ext.gemm_bf16(a, b.transpose(1, 2).contiguous() if b_mn else b, again, False, b_mn, 0.7, -1.3, wide[..., :n])
    assert torch.equal(again, d)
    ext.gemm_bf16(a, b.transpose(1, 2).contiguous() if b_mn else b, again, False, b_mn, 0.7, -1.3, c[0])      # broadcast: read by the threads
    assert rel(again, 0.7 * (a.double() @ b.double().transpose(1, 2)) - 1.3 * c[:1].double()) < 3e-3
    for spread in (c[:1].expand_as(c), c[:, :1].expand_as(c)):                                     # the same by a stride of zero
        ext.gemm_bf16(a, b.transpose(1, 2).contiguous() if b_mn else b, again, False, b_mn, 0.7, -1.3, spread)
        assert rel(again, 0.7 * (a.double() @ b.double().transpose(1, 2)) - 1.3 * spread.double()) < 3e-3
    cuda_ops.check_status()


def test_an_unaligned_addend_is_refused():
    a, b = torch.randn(16, 64, device="cuda").bfloat16(), torch.randn(24, 64, device="cuda").bfloat16()
    c = torch.randn(16 * 24 + 1, device="cuda").bfloat16()[1:].view(16, 24)
    with pytest.raises(RuntimeError, match="16-byte"):
        cuda_ops.ext().gemm_bf16(a, b, torch.empty(16, 24, device="cuda", dtype=torch.bfloat16), False, False, 1.0, 1.0, c)


@pytest.mark.parametrize("batch,m", [(1, 8), (3, 200), (2, 264), (30, 768), (1, 1096)])
def test_symmetric_addend(batch, m):
    torch.manual_seed(4)
    x = torch.randn(batch, m, 64, device="cuda") / 8
    s = (x @ x.transpose(1, 2)).bfloat16()
    assert torch.equal(s, s.transpose(1, 2).contiguous())
    d = torch.empty_like(s)
    cuda_ops.ext().gemm_bf16(s, s, d, False, False, 0.5, -0.25, s, symmetric=True)
    want = 0.5 * (s.double() @ s.double()) - 0.25 * s.double()
    assert rel(d, want) < 3e-3
    if m <= 256:                      # one tile: both halves are computed, equal up to the order of the sums
        assert rel(d, d.transpose(1, 2)) < 3e-3
    else:                             # off-diagonal tiles are copies
        assert torch.equal(d[:, :256, 256:], d[:, 256:, :256].transpose(1, 2))
    cuda_ops.check_status()
