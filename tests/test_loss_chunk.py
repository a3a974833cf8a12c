"""Rows of a chunk of the LM-head loss (`loss_chunk_rows` in ops/cuda_ops.py)."""
import pytest
import torch

from gpt_moe_b200.ops import cuda_ops
from gpt_moe_b200.ops import reference as ref


def test_chunks_follow_width_and_sm_count():
    rows = cuda_ops.loss_chunk_rows
    assert [rows(width, 50304, 148, True) for width in (512, 768, 1024, 2048)] == [9472, 12544, 9472, 9472]
    for width in (64, 256, 768, 1000, 1536, 4096):
        for sms in (2, 100, 132, 148, 160):
            waves = {r: -(-(r // 256) * -(-width // 256) // (sms // 2)) * (sms // 2) / r for r in range(8192, 12544 + 1, 256)}
            chosen = rows(width, 50304, sms, True)
            assert chosen in waves and waves[chosen] <= min(waves.values()) * (1 + 1e-9)
            assert rows(width, 50304, sms, False) == 8192


def test_chunks_of_a_large_vocabulary_hold_no_more_rows_than_others():
    for vocab in (50304, 60000, 81920, 128256, 262144):
        chunk = cuda_ops.loss_chunk_rows(768, vocab, 148, True)
        assert chunk == 8192 or chunk * vocab * 2 <= 5 << 28


# one chunk and a few rows, at a width with chunks of its own; two columns of tiles
@pytest.mark.gpu
@pytest.mark.parametrize("rows,width", [(9472 + 40, 1024), (12544 + 3, 768), (9472, 512)])
def test_loss_and_gradients_over_chunks(rows, width):
    torch.manual_seed(14)
    x = torch.randn(rows, width, device="cuda").bfloat16().requires_grad_()
    w = (torch.randn(1024, width, device="cuda") * 0.05).bfloat16().float().requires_grad_()
    y = torch.randint(0, 1024, (rows,), device="cuda")
    y[::7] = -100
    loss = cuda_ops.linear_cross_entropy(x, w, y)
    got = torch.autograd.grad(loss, (x, w))
    xd, wd = x.detach().double().requires_grad_(), w.detach().double().requires_grad_()
    want_loss = ref.cross_entropy(xd @ wd.t(), y)
    want = torch.autograd.grad(want_loss, (xd, wd))
    # logits and their gradients are bf16: 2^-9 / sqrt(3) each on average, and the result's own rounding
    assert abs(loss.item() - want_loss.item()) < 1e-3 * want_loss.item()
    for a, b in zip(got, want):
        assert ((a.double() - b).norm() / b.norm()).item() < 6e-3
    cuda_ops.check_status()
