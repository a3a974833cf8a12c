"""The embedding gradient that is added into the engine's buffer, against fp64 sums."""
import pytest
import torch

from gpt_moe_b200.ops import cuda_ops

pytestmark = pytest.mark.gpu


# windows of 32 sorted tokens: inside one, edges, runs over many windows, every token the same, widths around the block
@pytest.mark.parametrize("tokens,vocab,d", [(1, 5, 4), (31, 3, 64), (32, 1, 768), (33, 2, 1024), (500, 4, 260), (4096, 50304, 768), (3000, 7, 132)])
def test_gradient_is_added_row_by_row(tokens, vocab, d):
    torch.manual_seed(tokens)
    module = torch.nn.Embedding(vocab, d, device="cuda")
    weight = module.weight
    weight.main_grad = torch.randn(vocab, d, device="cuda")
    weight.grad_ready = True
    before = weight.main_grad.clone()
    # ids as words are: a few of them make up most of the text
    ids = torch.clamp((vocab ** torch.rand(tokens, device="cuda")).long() - 1, 0, vocab - 1).view(1, tokens)
    dy = torch.randn(1, tokens, d, device="cuda")
    out = cuda_ops.embedding(module, ids)
    assert torch.equal(out, weight.detach()[ids])
    out.backward(dy)
    assert weight.grad is None
    want = before.double().index_add_(0, ids.view(-1), dy[0].double())
    count = torch.bincount(ids.view(-1), minlength=vocab).max().item()
    # fp32 sums of `count` terms of size one: at most count * 2^-24 * sqrt(count), and one rounding of the row
    assert (weight.main_grad.double() - want).abs().max().item() < 2e-6 + count ** 1.5 * 6e-8
    again = before.clone()
    weight.main_grad = again
    cuda_ops.embedding(module, ids).backward(dy)
    first = before.clone()
    weight.main_grad = first
    cuda_ops.embedding(module, ids).backward(dy)
    assert torch.equal(first, again)                     # the same bits every time
    weight.main_grad, weight.grad_ready = torch.full((vocab, d), float("nan"), device="cuda"), False
    cuda_ops.embedding(module, ids).backward(dy)         # a buffer that has not been written in this step is overwritten
    assert (weight.main_grad.double() - (want - before.double())).abs().max().item() < 4e-6 + count ** 1.5 * 6e-8
