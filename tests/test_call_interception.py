"""Calls without gradients skip the autograd node only where nothing looks at the ops themselves (no GPU needed)."""
import torch
from torch.autograd import forward_ad
from torch.utils._python_dispatch import TorchDispatchMode

from gpt_moe_b200.ops import attention_tc, cuda_ops


class _Double(torch.autograd.Function):
    """Opaque to a trace, as an extension call is."""

    @staticmethod
    def forward(ctx, x):
        return torch.from_numpy(2 * x.detach().numpy())

    @staticmethod
    def backward(ctx, g):
        return 2 * g


class _Watch(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def test_a_trace_records_the_call_and_not_its_result():
    with torch.no_grad():
        traced = torch.jit.trace(lambda x: cuda_ops.run_function(_Double, x) + 1, torch.ones(3), check_trace=False)
        assert torch.equal(traced(torch.full((3,), 5.0)), torch.full((3,), 11.0))


def test_what_the_attention_kernels_take():
    def qkv(b, t, s=None):
        return [torch.empty(b, n, 1, 64, dtype=torch.bfloat16) for n in (t, s or t, s or t)]

    assert attention_tc.supported(*qkv(1, 100), 0.0) and attention_tc.supported(*qkv(65535, 1), 0.0)
    assert not attention_tc.supported(*qkv(65536, 1), 0.0)          # sequences are a grid dimension
    assert not attention_tc.supported(*qkv(1, 100, 200), 0.0) and not attention_tc.supported(*qkv(2, 100, 50), 0.0)
    with forward_ad.dual_level():
        assert not attention_tc.supported(*qkv(1, 100), 0.0) and attention_tc.supported(*qkv(1, 128), 0.0)


def test_modules_with_hooks_or_a_forward_of_their_own_are_called():
    a, b = torch.nn.Linear(2, 2), torch.nn.Embedding(3, 2)
    assert cuda_ops.bypassable(a, b)
    for register in (a.register_forward_hook, a.register_forward_pre_hook, a.register_full_backward_hook, a.register_full_backward_pre_hook,
                     lambda f: torch.nn.modules.module.register_module_forward_hook(f),
                     lambda f: torch.nn.modules.module.register_module_full_backward_hook(f)):
        handle = register(lambda *args: None)
        assert not cuda_ops.bypassable(b, a)
        handle.remove()
        assert cuda_ops.bypassable(a, b)
    b.forward = lambda ids: torch.zeros(1)
    assert not cuda_ops.bypassable(a, b)


def test_plain_call_is_off_under_transforms_tangents_traces_and_modes():
    seen = []
    assert not cuda_ops.plain_call()                       # gradients are recorded
    with torch.no_grad():
        assert cuda_ops.plain_call()
        with forward_ad.dual_level():
            assert not cuda_ops.plain_call()
        torch.func.vmap(lambda x: (seen.append(cuda_ops.plain_call()), x)[1])(torch.ones(2))
        torch.jit.trace(lambda x: (seen.append(cuda_ops.plain_call()), x + 1)[1], torch.ones(2), check_trace=False)
        with _Watch():
            seen.append(cuda_ops.plain_call())
        assert cuda_ops.plain_call()
    assert seen == [False, False, False]
