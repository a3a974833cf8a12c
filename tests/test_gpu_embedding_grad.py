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


def test_a_gradient_that_is_read_is_formed():
    torch.manual_seed(2)
    module = torch.nn.Embedding(11, 16, device="cuda")
    weight = module.weight
    ids = torch.randint(0, 11, (2, 9), device="cuda")
    dy = torch.randn(2, 9, 16, device="cuda")
    want = torch.zeros(11, 16, device="cuda").index_add_(0, ids.view(-1), dy.view(-1, 16))
    weight.grad = torch.zeros(11, 16, device="cuda")                  # as the fused engine lays it out: one buffer for both
    weight.main_grad, weight.grad_ready = weight.grad, True
    buffer = weight.main_grad
    (got,) = torch.autograd.grad(cuda_ops.embedding(module, ids), weight, dy)
    assert torch.allclose(got, want, atol=1e-5) and (buffer == 0).all()
    leaf = dy.clone().requires_grad_()
    (got,) = torch.autograd.grad(cuda_ops.embedding(module, ids), weight, leaf, create_graph=True)
    (back,) = torch.autograd.grad((got ** 2).sum(), leaf)             # 2 g, gathered at the positions
    assert torch.allclose(back, 2 * want[ids], atol=1e-4)
    seen = []
    hook = weight.register_hook(lambda g: seen.append(g.clone()))
    after = weight.register_post_accumulate_grad_hook(lambda p: seen.append(p.grad.clone()))
    cuda_ops.embedding(module, ids).backward(dy)
    hook.remove(), after.remove()
    assert len(seen) == 2 and all(torch.allclose(g, want, atol=1e-5) for g in seen)
    assert weight.grad.data_ptr() == buffer.data_ptr() and torch.allclose(buffer, want, atol=1e-5)
    cuda_ops.embedding(module, ids).backward(dy)                      # and without them straight into the buffer again
    assert weight.grad.data_ptr() == buffer.data_ptr() and torch.allclose(buffer, 2 * want, atol=2e-5)
    base = torch.randn(1 + dy.numel(), device="cuda")
    cuda_ops.embedding(module, ids).backward(base[1:].view(dy.shape))  # a gradient on no 16-byte boundary
    assert torch.allclose(buffer, 2 * want + torch.zeros_like(want).index_add_(0, ids.view(-1), base[1:].view(-1, 16)), atol=2e-5)


def test_tangents_and_traces_run_through_the_module():
    module = torch.nn.Embedding(7, 8, device="cuda")
    module.weight.main_grad, module.weight.grad_ready = torch.zeros(7, 8, device="cuda"), True
    ids = torch.tensor([[1, 2, 6]], device="cuda")
    from torch.autograd import forward_ad
    with forward_ad.dual_level():
        assert torch.equal(cuda_ops.embedding(module, ids), module(ids))

    class Lookup(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.table = module

        def forward(self, i):
            return cuda_ops.embedding(self.table, i)

    traced = torch.jit.trace(Lookup(), ids, check_trace=False)
    assert "PythonOp" not in str(traced.inlined_graph) and torch.equal(traced(ids.flip(1)), module(ids.flip(1)))
