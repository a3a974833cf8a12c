"""All blocks of a forward pass without gradients as one native call (`trunk`): the bits of the blocks' own calls, and only where they apply."""
import pytest
import torch
import torch.nn.utils.parametrize
import torch.nn.utils.prune

from gpt_moe_b200.config import get_preset
from gpt_moe_b200.models.gpt import GPT
from gpt_moe_b200.ops import cuda_ops

pytestmark = pytest.mark.gpu

# name: (model options, tokens, whether the one call serves it)
CASES = {
    "one token": ({}, 1, True),
    "odd length": ({}, 77, True),
    "grouped heads, full attention in one layer": (dict(n_kv_heads=4, full_attention_layers=[1], global_attn_dim=768, global_n_kv_heads=4), 300, True),
    "two experts a token, gates renormalised": (dict(moe_top_k=2), 130, True),
    "relu2": (dict(activation="relu2"), 40, True),
    "capped logits": (dict(use_attn_logit_softcapping=True, attn_logit_softcap=20.0), 128, True),
    "no rotation": (dict(pos_encoding_type="learned"), 64, True),
    "a scale on the residual": (dict(use_weighted_residual_path=True), 64, False),
    "dense feed-forward": (dict(use_moe=False), 64, False),
}


def _model(**options):
    torch.manual_seed(1)
    gc, tc = get_preset("small")
    gc.n_layers, gc.mlp_hidden_dim, gc.weighted_main_path_init = 3, 256, 0.3
    for name, value in options.items():
        assert hasattr(gc, name), name
        setattr(gc, name, value)
    tc.seq_len_train = tc.seq_len_val = 512
    tc.resolve(1)
    model = GPT(gc, tc).cuda().eval()
    model.set_sliding_window(48)
    model.set_precision_phase("evaluation")
    return model, gc


def _served(model):
    """Layers that went into the native call, one entry per call of the model's."""
    seen, inner = [], model._plain_blocks
    model._plain_blocks = lambda layers, *args: (seen.append(len(layers)), inner(layers, *args))[1]
    return seen


def _apart(model):
    model._plain_forward = lambda *args: False


@pytest.mark.parametrize("case", CASES)
def test_trunk_has_the_bits_of_the_blocks_own_calls(case):
    options, t, served = CASES[case]
    model, gc = _model(**options)
    ids = torch.randint(0, gc.vocab_size, (3, t), device="cuda")
    with torch.no_grad():
        seen = _served(model)
        got = model(ids)
        assert sum(seen) == (3 if served else 0)
        _apart(model)
        assert torch.equal(got, model(ids))
    cuda_ops.check_status()


@pytest.mark.parametrize("tokens", [1, 37, 130, 400])
def test_trunk_does_not_read_rows_that_hold_no_slot(tokens):
    """Pad rows of the experts' buffers are left as they are; here every byte the allocator has to give is part of a NaN."""
    model, gc = _model(moe_top_k=2)
    ids = torch.randint(0, gc.vocab_size, (1, tokens), device="cuda")
    with torch.no_grad():
        _apart(model)
        want = model(ids)
        del model._plain_forward
        torch.cuda.empty_cache()
        held = [torch.full((size,), 255, dtype=torch.uint8, device="cuda") for size in (1 << 10, 1 << 16, 1 << 19, 1 << 20, 12 << 20, 20 << 20, 40 << 20) for _ in range(12)]
        del held
        assert torch.equal(model(ids), want)
    cuda_ops.check_status()


def test_trunk_steps_aside_for_whoever_looks_at_a_block():
    model, gc = _model()
    ids = torch.randint(0, gc.vocab_size, (2, 33), device="cuda")
    with torch.no_grad():
        want, seen = model(ids), _served(model)
        for module, apart in ((model.transformer.h[1].attn, 1), (model.transformer.h[2].mlp, 1), (model.transformer.h[0].attn.out_proj, 1),
                              (model.transformer.h[0].mlp.router, 1)):
            calls = []
            handle = module.register_forward_hook(lambda *args: calls.append(1))
            seen.clear()
            assert torch.equal(model(ids), want) and sum(seen) == 3 - apart and calls      # the other blocks stay in the native call
            handle.remove()
        own = model.transformer.h[1].mlp.forward
        model.transformer.h[1].mlp.forward = lambda x: (0 * own(x)[0], None)
        seen.clear()
        assert not torch.equal(model(ids), want) and sum(seen) == 2
        del model.transformer.h[1].mlp.forward
        # weights changed in place are seen by the next call
        seen.clear()
        assert torch.equal(model(ids), want) and sum(seen) == 3
        model.transformer.h[1].attn.out_proj.weight.mul_(2)
        changed = model(ids)
        _apart(model)
        assert not torch.equal(changed, want) and torch.equal(changed, model(ids))
    cuda_ops.check_status()


class _Twice(torch.nn.Module):
    def forward(self, w):
        return 2 * w


def _parametrised_weight(block):
    torch.nn.utils.parametrize.register_parametrization(block.attn.k_proj, "weight", _Twice())


def _pruned_weight(block):
    torch.nn.utils.prune.random_unstructured(block.attn.q_proj, "weight", 0.5)


def _parametrised_bias(block):
    block.attn.q_proj.register_parameter("bias", torch.nn.Parameter(torch.randn(block.attn.attn_dim, device="cuda")))
    torch.nn.utils.parametrize.register_parametrization(block.attn.q_proj, "bias", _Twice())


def _rows_with_a_pitch(block):
    for module in (block.attn.out_proj, block.mlp.router):
        rows, cols = module.weight.shape
        wide = torch.zeros(rows, cols + 8, device="cuda", dtype=torch.bfloat16)
        wide[:, :cols] = module.weight.detach()
        module.weight = torch.nn.Parameter(wide[:, :cols])


def _own_step(block):
    inner = block.forward_prenormed
    block.forward_prenormed = lambda x, h, *rest: inner(x, 2 * h, *rest)


# change of the middle block: layers that stay in the native call
@pytest.mark.parametrize("change,served", [(_parametrised_weight, 3), (_pruned_weight, 3), (_parametrised_bias, 2), (_rows_with_a_pitch, 3), (_own_step, 2)])
def test_trunk_takes_modules_as_the_blocks_own_calls_do(change, served):
    model, gc = _model()
    ids = torch.randint(0, gc.vocab_size, (2, 40), device="cuda")
    with torch.no_grad():
        plain = model(ids)
        change(model.transformer.h[1])
        seen = _served(model)
        got = model(ids)
        assert sum(seen) == served
        _apart(model)
        assert torch.equal(got, model(ids))
        assert torch.equal(got, plain) == (change is _rows_with_a_pitch)
    cuda_ops.check_status()
