"""A forward pass without gradients takes composed calls (whole branches of a block): the same kernels, so the same bits."""
import pytest
import torch

from gpt_moe_b200.config import get_preset
from gpt_moe_b200.models.gpt import GPT
from gpt_moe_b200.ops import cuda_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("preset,t", [("small", 45), ("small", 256), ("wide_ep", 130), ("mla", 77)])
def test_no_grad_forward_equals_the_recorded_one(preset, t):
    torch.manual_seed(0)
    gc, tc = get_preset(preset)
    gc.n_layers, gc.num_experts, gc.weighted_main_path_init = 2, 8, 0.3
    tc.expert_parallel_size = 1
    tc.seq_len_train = tc.seq_len_val = 256
    tc.resolve(1)
    model = GPT(gc, tc).cuda().eval()
    model.set_sliding_window(64)
    model.set_precision_phase("evaluation")
    ids = torch.randint(0, gc.vocab_size, (2, t), device="cuda")
    recorded = model(ids)
    assert recorded.requires_grad
    with torch.no_grad():
        plain = model(ids)
        docs = torch.zeros(2, t, dtype=torch.long, device="cuda")
        docs[:, t // 2:] = 1
    assert torch.equal(plain, recorded.detach())
    model.use_doc_masking = True
    with torch.no_grad():
        masked = model(ids, document_ids=docs)
    assert torch.equal(masked, model(ids, document_ids=docs).detach())
    if preset != "mla":                       # hooks on a projection keep the modules' own path
        seen = []
        model.transformer.h[0].attn.out_proj.register_forward_hook(lambda *a: seen.append("out"))
        model.transformer.h[0].mlp.router.register_forward_hook(lambda *a: seen.append("router"))
        with torch.no_grad():
            assert torch.equal(model(ids, document_ids=docs), masked)
        assert seen == ["out", "router"]
        from torch.nn.modules.module import register_module_forward_hook
        handle = register_module_forward_hook(lambda m, *a: seen.append(type(m).__name__))
        try:
            with torch.no_grad():
                assert torch.equal(model(ids, document_ids=docs), masked)
        finally:
            handle.remove()
        assert sum(name == "Linear" for name in seen) >= 2 * 2                  # out_proj and router of both layers
    cuda_ops.check_status()
