"""The attention kernels at sequence lengths that are no multiple of a tile, against the fp32 definition."""
import pytest
import torch

from gpt_moe_b200.ops import attention_cuda, cuda_ops
from gpt_moe_b200.ops import reference as ref

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = a.detach().double(), b.detach().double()
    return ((a - b).norm() / b.norm().clamp_min(1e-30)).item()


# one row, inside a tile, edges of one and two tiles, odd and even numbers of tiles
@pytest.mark.parametrize("t,window,hq,hk,d", [(1, None, 2, 2, 64), (45, None, 4, 4, 64), (127, 20, 2, 1, 64), (129, None, 4, 2, 64),
                                               (184, 64, 2, 2, 64), (300, None, 2, 2, 64), (1000, 256, 3, 3, 64), (1100, None, 2, 1, 64),
                                               (45, None, 2, 2, 128), (333, 100, 2, 1, 128)])
def test_any_length_forward_and_backward(t, window, hq, hk, d):
    torch.manual_seed(5)
    b = 3
    q, k, v = (torch.randn(b, t, h, w, device="cuda").bfloat16() for h, w in ((hq, d), (hk, d), (hk, 64)))
    g = torch.randn(b, t, hq, 64, device="cuda").bfloat16()
    for x in (q, k, v, g):
        x[1] = float("nan")                       # a tile that reaches past a sequence's end must not see the next sequence
    q, k, v = (x.requires_grad_() for x in (q, k, v))
    before = cuda_ops.path_counts().get("attention:tcgen05", 0)
    out = attention_cuda.attention(q, k, v, window=window)
    assert cuda_ops.path_counts()["attention:tcgen05"] == before + 1
    grads = torch.autograd.grad(out, (q, k, v), g)
    keep = [0, 2]
    want_in = [x.detach()[keep].float().requires_grad_() for x in (q, k, v)]
    want = ref.attention(*want_in, causal=True, window=window)
    want_grads = torch.autograd.grad(want, want_in, g[keep].float())
    # bf16 probabilities and results: a rounding is 2^-9 / sqrt(3) = 1.1e-3 on average, two to three of them on the way to each output
    assert rel(out[keep], want) < 6e-3
    for got, exp in zip(grads, want_grads):
        if exp.norm() > 1e-3:                     # a single row attends to itself alone: its score gradients vanish
            assert rel(got[keep], exp) < 1e-2
        else:
            assert got[keep].float().norm() < 1e-1
    cuda_ops.check_status()


@pytest.mark.parametrize("t", [200, 300])
def test_any_length_with_document_mask(t):
    torch.manual_seed(6)
    q, k, v = (torch.randn(2, t, 2, 64, device="cuda").bfloat16().requires_grad_() for _ in range(3))
    g = torch.randn(2, t, 2, 64, device="cuda").bfloat16()
    docs = (torch.rand(2, t, device="cuda") < 0.02).int().cumsum(1)
    out = attention_cuda.attention(q, k, v, document_ids=docs)
    grads = torch.autograd.grad(out, (q, k, v), g)
    want_in = [x.detach().float().requires_grad_() for x in (q, k, v)]
    want = ref.attention(*want_in, causal=True, document_ids=docs)
    assert rel(out, want) < 6e-3
    for got, exp in zip(grads, torch.autograd.grad(want, want_in, g.float())):
        assert rel(got, exp) < 1e-2
    cuda_ops.check_status()


# lengths outside whole pairs of tiles: both forward kernels follow the row maximum exactly
@pytest.mark.parametrize("t,window", [(184, 50), (184, None), (1000, 256), (1152, 256), (1500, None), (300, None), (1100, None)])
def test_ragged_outputs_are_as_exact_as_the_single_tile_kernels(t, window):
    torch.manual_seed(7)
    q, k = (torch.nn.functional.rms_norm(torch.randn(2, t, 4, 64, device="cuda"), (64,)).bfloat16() for _ in range(2))
    v = torch.randn(2, t, 4, 64, device="cuda").bfloat16()
    w = t if window is None else window
    out = cuda_ops.ext().attn_fwd(q, k, v, w, 0.125)[0]
    single = cuda_ops.ext().attn_fwd(q, k, v, w, 0.125, single_tile=True)[0]
    want = ref.attention(q.double(), k.double(), v.double(), causal=True, window=window)
    # the same probabilities in bf16; another order of the sums moves the error's fourth digit, a lagging maximum its second
    assert rel(out, want) < 1.003 * rel(single, want)
    cuda_ops.check_status()


@pytest.mark.parametrize("t", [257, 384])
def test_three_tiles_without_a_window_take_the_single_tile_kernel(t):
    """Of three query tiles the two-tile kernel idles in a quarter of its work (64 x 300 tokens: 109 us against 103)."""
    torch.manual_seed(10)
    q, k, v = (torch.randn(2, t, 4, 64, device="cuda").bfloat16() for _ in range(3))
    out, lse = cuda_ops.ext().attn_fwd(q, k, v, t, 0.125)
    single, single_lse = cuda_ops.ext().attn_fwd(q, k, v, t, 0.125, single_tile=True)
    assert torch.equal(out, single) and torch.equal(lse, single_lse)


@pytest.mark.parametrize("t", [200, 256])
@pytest.mark.parametrize("scale", [1e-12, 1e-6, 4.0])
def test_gradients_at_any_scale(t, scale):
    """Rows past the end of the last tile have no probabilities, however small the scale that their statistics are divided by."""
    torch.manual_seed(11)
    q, k, v = (torch.randn(2, t, n, 64, device="cuda").bfloat16().requires_grad_() for n in (4, 2, 2))
    g = torch.randn(2, t, 4, 64, device="cuda").bfloat16()
    out = attention_cuda.attention(q, k, v, scale=scale)
    grads = torch.autograd.grad(out, (q, k, v), g)
    want_in = [x.detach().double().requires_grad_() for x in (q, k, v)]
    want = ref.attention(*want_in, causal=True, scale=scale)
    assert rel(out, want) < 6e-3
    for got, exp in zip(grads, torch.autograd.grad(want, want_in, g.double())):
        assert rel(got, exp) < 1e-2
    cuda_ops.check_status()


# twelve key tiles and more, where the two query tiles take turns at their exponentials: B with as many key tiles as A and with one more
@pytest.mark.parametrize("softcap", [0.0, 15.0])
@pytest.mark.parametrize("t,window", [(2048, 2048), (2304, 1536), (3072, 1700)])
def test_turns_of_the_query_tiles(t, window, softcap):
    torch.manual_seed(12)
    q, k = (2 * torch.nn.functional.rms_norm(torch.randn(1, t, 2, 64, device="cuda"), (64,)).bfloat16() for _ in range(2))
    v = torch.randn(1, t, 2, 64, device="cuda").bfloat16()
    out, lse = cuda_ops.ext().attn_fwd(q, k, v, window, 0.125, softcap)
    want = ref.attention(q.double(), k.double(), v.double(), causal=True, window=window, scale=0.125, softcap_value=softcap)
    # bf16 probabilities and result; the cap is the hardware's tanh (2^-11 of the cap, an exponent of e)
    assert rel(out, want) < (6e-3 if softcap else 3e-3)
    word = torch.tensor([window], dtype=torch.int32, device="cuda")           # the kernel's own look-back, shorter than the one the host decides by
    again, again_lse = cuda_ops.ext().attn_fwd(q, k, v, t, 0.125, softcap, window_tensor=word)
    assert torch.equal(out, again) and torch.equal(lse, again_lse)
    cuda_ops.check_status()


def test_a_longer_look_back_on_the_device_keeps_the_exact_maximum():
    """The reference of the exponentials may lag only where the look-back in use is short, not where the host's bound alone is."""
    torch.manual_seed(13)
    t = 2304
    q, k = (torch.nn.functional.rms_norm(torch.randn(1, t, 4, 64, device="cuda"), (64,)).bfloat16() for _ in range(2))
    q, v = 3 * q, torch.randn(1, t, 4, 64, device="cuda").bfloat16()
    word = torch.tensor([t], dtype=torch.int32, device="cuda")
    out, single = (cuda_ops.ext().attn_fwd(q, k, v, 1024, 0.125, single_tile=one, window_tensor=word)[0] for one in (False, True))
    want = ref.attention(q.double(), k.double(), v.double(), causal=True, window=None)
    assert rel(out, want) < 1.003 * rel(single, want)                 # bound as above
    cuda_ops.check_status()
