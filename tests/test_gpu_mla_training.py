"""Latent attention from its projections (one autograd node) and the shared expert's activation against fp32 definitions."""
import copy

import pytest
import torch

from gpt_moe_b200.config import get_preset
from gpt_moe_b200.models.attention import AttentionContext
from gpt_moe_b200.models.mla import MLAttention
from gpt_moe_b200.ops import api, cuda_ops
from gpt_moe_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def rel(a, b):
    return ((a.detach().double() - b.detach().double()).norm() / b.detach().double().norm().clamp_min(1e-30)).item()


# rotary widths, odd head counts (a warp's second head is empty), grouped heads, ragged lengths, window, no QK-norm, clamped scales
@pytest.mark.parametrize("b,t,hq,hk,dr,window,norm", [(2, 256, 4, 4, 64, None, True), (1, 200, 3, 3, 64, 50, True), (2, 45, 4, 2, 32, None, True),
                                                      (1, 130, 2, 1, 8, None, False), (3, 1, 2, 2, 64, None, True)])
def test_node_matches_reference(b, t, hq, hk, dr, window, norm):
    torch.manual_seed(9)
    content = 128 - dr
    q = torch.randn(b, t, hq * 128, device="cuda").bfloat16().requires_grad_()
    kv = torch.randn(b, t, hk * (content + 64), device="cuda").bfloat16().requires_grad_()
    low = torch.randn(b, t, 16 + dr, device="cuda").bfloat16().requires_grad_()
    qs = torch.tensor([0.8, 1.3, 6.0, 1.0][:hq], device="cuda").view(1, hq, 1, 1).requires_grad_() if norm else None       # 6 is clamped to 5
    ks = torch.linspace(0.7, 1.2, hk, device="cuda").view(1, hk, 1, 1).requires_grad_() if norm else None
    cos, sin = ref.rope_tables(dr, 10000, t + 3)
    cos, sin = cos.cuda(), sin.cuda()
    scale = 128 ** -0.5
    out = cuda_ops.mla_rope_attention(q, kv, low[..., 16:], cos, sin, qs, ks, hq, hk, 1e-6, True, float("-inf"), 5.0, window, scale)
    g = torch.randn_like(out)
    leaves = [x for x in (q, kv, low, qs, ks) if x is not None]
    grads = torch.autograd.grad(out, leaves, g)

    want_leaves = [x.detach().float().requires_grad_() for x in leaves]
    wq, wkv, wlow = want_leaves[:3]
    wqs, wks = want_leaves[3:] if norm else (None, None)
    query = wq.view(b, t, hq, 128)
    kvh = wkv.view(b, t, hk, content + 64)
    rope = ref.apply_rope(wlow[..., 16:].reshape(b, t, 1, dr), cos, sin)
    query = torch.cat((query[..., :content], ref.apply_rope(query[..., content:], cos, sin)), dim=-1)
    key = torch.cat((kvh[..., :content], rope.expand(-1, -1, hk, -1)), dim=-1)
    if norm:
        # one copy of a scale per token: their gradients are the terms of the scale's, and the terms cancel
        tqs, tks = (w.clamp(max=5.0).view(1, 1, -1, 1).expand(b, t, -1, 1).clone() for w in (wqs, wks))
        tqs.retain_grad(), tks.retain_grad()
        query = query * torch.rsqrt(query.pow(2).mean(-1, keepdim=True) + 1e-6) * tqs
        key = key * torch.rsqrt(key.pow(2).mean(-1, keepdim=True) + 1e-6) * tks
    want = ref.attention(query, key, kvh[..., content:], causal=True, window=window, scale=scale)
    want.backward(g.float())
    want_grads = [x.grad for x in want_leaves]
    # rotated heads, probabilities and results are rounded to bf16, 1.1e-3 on average each
    assert rel(out, want) < 8e-3
    for got, exp, name in zip(grads, want_grads, ("q", "kv", "low", "q_scale", "k_scale")):
        # a scale's gradient is a sum of terms many times its size, each as exact as a gradient (rounding the rotated heads alone moves the
        # sum by up to 3e-3 of the terms' norm)
        size = exp.norm() if name not in ("q_scale", "k_scale") else (tqs if name == "q_scale" else tks).grad.norm()
        if size > 1e-2:                       # one position: the scores have no gradient
            assert (got.float() - exp).norm() < 1.5e-2 * size, name
    cuda_ops.check_status()


@pytest.mark.parametrize("name", ["gelu", "relu", "relu2", "silu", "swiglu"])
@pytest.mark.parametrize("shape", [(3, 5, 16), (300, 1024), (7, 6)])
def test_activation_entry_point(name, shape):
    torch.manual_seed(4)
    x = (3 * torch.randn(*shape, device="cuda")).bfloat16().requires_grad_()
    y = api.activate(x, name)
    g = torch.randn_like(y)
    (dx,) = torch.autograd.grad(y, x, g)
    xf = x.detach().float().requires_grad_()
    want = ref.activate(xf, name)
    (dwant,) = torch.autograd.grad(want, xf, g.float())
    tol = 4e-3 if shape[-1] % 16 == 0 else 8e-3          # one rounding in the kernel; torch's ops round every intermediate
    assert rel(y, want) < tol and rel(dx, dwant) < tol


@pytest.mark.parametrize("name", ["gelu", "relu", "relu2", "silu", "swiglu"])
def test_activation_keeps_nan_and_infinities(name):
    x = torch.tensor([float("nan"), float("inf"), -float("inf"), 0.0, -0.0, 1.0, -1.0, 3.0e38] * 4, device="cuda").bfloat16()
    x = torch.stack((x, x.flip(0))).requires_grad_()
    y = api.activate(x, name)
    (dx,) = torch.autograd.grad(y, x, torch.ones_like(y))
    xf = x.detach().float().requires_grad_()
    want = ref.activate(xf, name)
    (dwant,) = torch.autograd.grad(want, xf, torch.ones_like(want))
    assert torch.equal(torch.isnan(y), torch.isnan(want))
    if name in ("relu", "relu2"):
        assert torch.allclose(y.float(), want.bfloat16().float(), equal_nan=True) and torch.allclose(dx.float(), dwant.bfloat16().float(), equal_nan=True)


@pytest.mark.parametrize("shape,name", [((3, 17), "swiglu"), ((2, 15), "swiglu"), ((4, 8), "unknown")])
def test_activation_refuses_what_torch_refuses(shape, name):
    x = torch.randn(*shape, device="cuda").bfloat16()
    with pytest.raises((RuntimeError, ValueError)):
        ref.activate(x, name)
    with pytest.raises((RuntimeError, ValueError)):
        api.activate(x, name)


@pytest.mark.parametrize("name", ["gelu", "relu2", "swiglu"])
def test_activation_of_empty_scalar_and_unaligned_tensors(name):
    for shape in ((0, 16), (3, 0), (0,)):
        assert api.activate(torch.empty(*shape, device="cuda", dtype=torch.bfloat16), name).shape == ref.activate(torch.empty(*shape), name).shape
    if name != "swiglu":
        assert api.activate(torch.tensor(2.0, device="cuda", dtype=torch.bfloat16), name).dim() == 0
    base = torch.randn(1 + 5 * 32, device="cuda").bfloat16()
    x = base[1:].view(5, 32).requires_grad_()                 # contiguous, on no 16-byte boundary
    y = api.activate(x, name)
    g = torch.randn(1 + y.numel(), device="cuda").bfloat16()[1:].view(y.shape)
    (dx,) = torch.autograd.grad(y, x, g)
    xf = x.detach().float().requires_grad_()
    want = ref.activate(xf, name)
    (dwant,) = torch.autograd.grad(want, xf, g.float())
    assert rel(y, want) < 4e-3 and rel(dx, dwant) < 4e-3


@pytest.mark.parametrize("name", ["gelu", "relu2", "silu", "swiglu"])
def test_activation_second_derivatives_tangents_and_vmap(name):
    torch.manual_seed(8)
    x = torch.randn(6, 64, device="cuda").bfloat16()
    v = torch.randn(6, 64, device="cuda").bfloat16()

    def second(leaf, f):
        (g,) = torch.autograd.grad((f(leaf, name).float() ** 2).sum(), leaf, create_graph=True)
        return torch.autograd.grad((g.float() * v.to(g.dtype).float()).sum(), leaf)[0]

    want = second(x.float().requires_grad_(), ref.activate)
    assert rel(second(x.clone().requires_grad_(), api.activate), want) < 2e-2                        # bf16 steps of torch's own derivatives
    t = x.t().contiguous().t().requires_grad_()                                                     # the gradient reaches the strided input itself
    assert rel(second(t, api.activate), want) < 2e-2
    out, tangent = torch.func.jvp(lambda y: api.activate(y, name), (x,), (v,))
    assert rel(tangent, torch.func.jvp(lambda y: ref.activate(y, name), (x.float(),), (v.float(),))[1]) < 2e-2
    assert torch.equal(torch.func.vmap(lambda y: api.activate(y, name))(x), ref.activate(x, name))
    traced = torch.jit.trace(lambda y: api.activate(y, name), x, check_trace=False)
    assert torch.equal(traced(v), ref.activate(v, name))


# rotary widths that are no whole 16-byte pieces; tables that were cast with the model
@pytest.mark.parametrize("dr,hk,t,cast", [(36, 4, 128, False), (4, 2, 75, False), (64, 4, 128, True), (20, 4, 130, True)])
def test_every_128_wide_head_takes_the_fused_path(dr, hk, t, cast, monkeypatch):
    torch.manual_seed(10)
    gc, tc = get_preset("mla")
    gc.hidden_size, gc.n_heads, gc.n_kv_heads = 256, 4, hk
    gc.mla_kv_rank, gc.mla_qk_rope_dim, gc.mla_qk_content_dim, gc.mla_value_dim, gc.mla_q_rank = 128, dr, 128 - dr, 64, 0
    tc.seq_len_train = tc.seq_len_val = 256
    tc.resolve(1)
    cpu = MLAttention(gc, tc)
    for p in cpu.parameters():
        if p.dim() == 2:
            torch.nn.init.normal_(p, std=0.05)
            p.data = p.data.bfloat16().float()
    gpu = copy.deepcopy(cpu).cuda()
    if cast:
        for m in (cpu, gpu):
            m.rotary.cos_cached, m.rotary.sin_cached = m.rotary.cos_cached.bfloat16(), m.rotary.sin_cached.bfloat16()
        cpu.rotary.float()                                   # the same rounded values
    monkeypatch.setattr(gpu, "_project", lambda *a: pytest.fail("general path"))
    x = torch.randn(2, t, 256).bfloat16()
    ctx = AttentionContext(40, None, None)
    xg, xc = x.cuda().requires_grad_(), x.float().requires_grad_()
    got, want = gpu(xg, ctx), cpu(xc, ctx)
    g = torch.randn_like(want).bfloat16()
    got.backward(g.cuda()), want.backward(g.float())
    # one rounding to bf16 for each of projections, rotated heads, probabilities, output and their gradients, 1.1e-3 on average
    assert rel(got.cpu(), want) < 1.2e-2 and rel(xg.grad.cpu(), xc.grad) < 2e-2
    for (name, a), (_, b) in zip(gpu.named_parameters(), cpu.named_parameters()):
        if a.dim() == 2:
            assert rel(a.grad.cpu(), b.grad) < 2e-2, name
    cuda_ops.check_status()


def test_swiglu_of_a_gate_far_below_zero():
    """exp(88) is a float and its reciprocal is not a normal one; the products are within bf16's range all the same."""
    x = torch.zeros(2, 32, device="cuda").bfloat16()
    x[0, :16], x[1, :16], x[:, 16:] = -87.5, -88.0, 1.0
    x.requires_grad_()
    y = api.activate(x, "swiglu")
    (dx,) = torch.autograd.grad(y, x, torch.ones_like(y))
    xd = x.detach().double().requires_grad_()
    want = ref.activate(xd, "swiglu")
    (dwant,) = torch.autograd.grad(want, xd, torch.ones_like(want))
    assert (y.double() / want - 1).abs().max() < 1e-2 and (dx.double() / dwant - 1).abs().max() < 1e-2       # single values: 2^-8 and exp's share
