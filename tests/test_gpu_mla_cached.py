"""The cached step of multi-head latent attention (`MLAttention.forward_cached`) on the GPU against the plain fp32 path on the CPU."""
import copy

import pytest
import torch

from gpt_moe_b200.config import get_preset
from gpt_moe_b200.models.mla import MLAttention

pytestmark = pytest.mark.gpu


def rel(a, b):
    a, b = a.detach().double().cpu(), b.detach().double().cpu()
    return ((a - b).norm() / b.norm().clamp_min(1e-30)).item()


# batch, new tokens, heads, kv heads, latent rank, rope width, content width, tokens already there, window, QK-norm, query rank
CASES = [
    (3, 1, 16, 16, 512, 64, 64, 333, None, True, 0),         # one token, cache no multiple of the tile
    (1, 1, 16, 16, 512, 64, 64, 0, None, True, 0),           # first token of an empty cache
    (33, 1, 16, 4, 512, 64, 64, 65, 40, True, 0),            # more rows than the skinny projection takes; groups of heads; window
    (2, 16, 16, 16, 512, 64, 64, 31, None, True, 0),         # 32 rows: largest skinny projection, tokens straddle tiles
    (1, 37, 8, 8, 256, 16, 48, 100, 20, True, 0),            # two tokens to a 16-row tile, odd count, narrow rotary part
    (2, 3, 32, 8, 256, 10, 54, 62, None, False, 0),          # 32 heads, rotary width no multiple of 8, no QK-norm
    (1, 70, 16, 16, 768, 32, 32, 5, None, True, 64),         # wide latent, low-rank queries, many tokens per weight pass
    (2, 1, 8, 2, 1024, 64, 64, 200, 64, True, 0),            # widest latent
    (3, 256, 16, 16, 512, 64, 64, 0, None, True, 0),         # expanded keys and values from here on: an empty cache, whole tiles
    (1, 200, 16, 4, 512, 64, 64, 333, None, True, 0),        # groups of heads, ragged queries and positions
    (4, 129, 8, 8, 256, 64, 64, 500, 100, True, 0),          # a window shorter than a tile: expansion starts inside the cache
    (4, 130, 16, 16, 768, 64, 64, 126, 300, False, 0),       # a window longer than a tile, no QK-norm
    (1, 300, 16, 16, 512, 64, 64, 1, None, True, 64),        # low-rank queries
]


@pytest.mark.parametrize("b,t,h,hkv,r,dr,c,start,window,norm,q_rank", CASES)
def test_cached_step_matches_the_plain_path(b, t, h, hkv, r, dr, c, start, window, norm, q_rank):
    torch.manual_seed(11)
    gc, tc = get_preset("mla")
    gc.hidden_size, gc.n_heads, gc.n_kv_heads, gc.use_qk_norm = 256, h, hkv, norm
    gc.mla_kv_rank, gc.mla_qk_rope_dim, gc.mla_qk_content_dim, gc.mla_value_dim, gc.mla_q_rank = r, dr, c, 64 if t >= 128 else 32, q_rank
    tc.resolve(1)
    cpu = MLAttention(gc, tc).eval()
    for p in cpu.parameters():
        if p.dim() == 2:
            torch.nn.init.normal_(p, std=0.05)
            p.data = p.data.bfloat16().float()                # both sides then project with the same weights
    gpu = copy.deepcopy(cpu).cuda()
    x = torch.randn(b, t, 256).bfloat16()
    cache = gpu.allocate_cache(b, start + t + 3, device="cuda", dtype=torch.bfloat16)
    cache.latent.normal_(), cache.rope.normal_(), cache.key_gain.uniform_(0.5, 2.0)
    poison = start + t
    for part in (cache.latent, cache.rope, cache.key_gain):
        part[:, poison:] = float("nan")                       # rows past the new tokens are not read
    cache.length = start
    plain = cpu.allocate_cache(b, start + t + 3, device="cpu", dtype=torch.float32)
    for mine, theirs in ((plain.latent, cache.latent), (plain.rope, cache.rope), (plain.key_gain, cache.key_gain)):
        mine.copy_(theirs.float().cpu())
        mine[:, poison:] = 0.0
    plain.length = start
    from gpt_moe_b200.ops import cuda_ops
    before = cuda_ops.path_counts().get("mla_decode:kernel", 0)
    got = gpu.forward_cached(x.cuda(), cache, window)
    assert cuda_ops.path_counts().get("mla_decode:kernel", 0) == before + 1
    if t >= 128:
        assert cuda_ops.ext().mla_prefill_wanted(b, t, h, hkv, start + t, -1 if window is None else window, r, dr, c, 64, 0.0)
    want = cpu.forward_cached(x.float(), plain, window)
    assert got.dtype == torch.bfloat16 and cache.length == plain.length == start + t
    new = slice(start, start + t)
    # one rounding to bf16 is 2^-9 / sqrt(3) = 1.1e-3 on average.  Cache entries: the projection's, the norm's and the stored one.
    # Output: those of query, latent and attention output (several thousand roundings average out in the sums) and its own; the
    # scores are the exponents of the probabilities, which doubles the share of query and key
    for name in ("latent", "rope", "key_gain"):
        assert rel(getattr(cache, name)[:, new], getattr(plain, name)[:, new]) < 5e-3, name
    assert rel(got, want) < 1.2e-2, rel(got, want)
    cuda_ops.check_status()


# an exactly full cache, one with room; a window that starts inside it; a rank whose contraction is long for its few tiles
@pytest.mark.parametrize("start,t,r,window", [(1000, 200, 512, None), (633, 512, 256, 200), (1000, 128, 1024, None)])
def test_a_batch_expands_as_its_sequences_do(start, t, r, window):
    torch.manual_seed(14)
    gc, tc = get_preset("mla")
    gc.hidden_size, gc.n_heads, gc.n_kv_heads, gc.mla_kv_rank = 256, 8, 4, r
    tc.resolve(1)
    attn = MLAttention(gc, tc).cuda().eval()
    x = torch.randn(3, t, 256, device="cuda").bfloat16()
    old = [torch.randn(3, start, n, device="cuda").bfloat16() for n in (r, 64)] + [torch.rand(3, start, 4, device="cuda").bfloat16() + 0.5]

    def call(rows, spare):
        cache = attn.allocate_cache(rows.stop - rows.start, start + t + spare, device="cuda", dtype=torch.bfloat16)
        for part, past in zip((cache.latent, cache.rope, cache.key_gain), old):
            part[:, :start] = past[rows]
            part[:, start + t:] = float("nan")
        cache.length = start
        return attn.forward_cached(x[rows], cache, window)

    from gpt_moe_b200.ops import cuda_ops
    assert cuda_ops.ext().mla_prefill_wanted(1, t, 8, 4, start + t, -1 if window is None else window, r, 64, 64, 64, 0.0)
    full, roomy = call(slice(0, 3), 0), call(slice(0, 3), 77)
    alone = torch.cat([call(slice(i, i + 1), 5) for i in range(3)])
    assert torch.equal(full, roomy) and torch.equal(full, alone)
    cuda_ops.check_status()


@pytest.mark.parametrize("t", [1, 40, 256])                    # one native call; absorbed; expanded
def test_a_weight_written_behind_torchs_back_is_seen(t):
    torch.manual_seed(13)
    gc, tc = get_preset("mla")
    gc.hidden_size, gc.n_heads, gc.n_kv_heads = 256, 8, 8
    tc.resolve(1)
    attn = MLAttention(gc, tc).cuda().eval()
    x = torch.randn(1, t, 256, device="cuda").bfloat16()

    def call(module):
        return module.forward_cached(x, module.allocate_cache(1, 300, device="cuda", dtype=torch.bfloat16))

    first = call(attn)
    attn.kv_up_proj.weight.data.mul_(-0.5)                     # bumps no version counter
    second = call(attn)
    assert not torch.equal(first, second)
    assert torch.equal(second, call(copy.deepcopy(attn)))


# sequences, new tokens, heads, kv heads, positions, rank: where one form was measured to be at least 1.3 times as fast as the other
@pytest.mark.parametrize("b,t,h,hkv,end,r,expanded", [(1, 64, 16, 16, 7000, 512, False), (2, 96, 16, 16, 1500, 512, True), (4, 48, 16, 16, 300, 512, True),
                                                      (16, 16, 16, 16, 4000, 512, False), (16, 16, 16, 2, 4000, 512, True), (4, 32, 16, 2, 4000, 512, True),
                                                      (2, 48, 8, 8, 1500, 256, False), (4, 48, 8, 8, 4000, 256, False), (1, 128, 8, 8, 7000, 256, False),
                                                      (2, 48, 32, 32, 1500, 512, True), (32, 8, 16, 4, 1000, 768, True), (1, 48, 16, 16, 2000, 512, False),
                                                      (16, 8, 16, 16, 4000, 1024, False), (16, 32, 16, 16, 500, 1024, True)])
def test_the_form_follows_heads_and_rank(b, t, h, hkv, end, r, expanded):
    from gpt_moe_b200.ops import cuda_ops
    assert cuda_ops.ext().mla_prefill_wanted(b, t, h, hkv, end, -1, r, 64, 64, 64, 0.0) == expanded


def test_a_tangent_is_not_dropped():
    gc, tc = get_preset("mla")
    gc.hidden_size, gc.n_heads, gc.n_kv_heads = 256, 8, 8
    tc.resolve(1)
    attn = MLAttention(gc, tc).cuda().eval()
    x = torch.randn(1, 4, 256, device="cuda").bfloat16()
    with torch.no_grad(), pytest.raises(RuntimeError):          # the projections have no rule for forward mode and say so
        torch.func.jvp(lambda y: attn.forward_cached(y, attn.allocate_cache(1, 8, device="cuda", dtype=torch.bfloat16)), (x,), (x,))


# grids of more than 65535 groups of rows or sequences; a window of zero positions keeps the work small
@pytest.mark.parametrize("b,t,h,r", [(1, 131072, 16, 768), (1, 65600, 32, 256), (65600, 1, 8, 256)])
def test_more_rows_than_a_grid_dimension_holds(b, t, h, r):
    torch.manual_seed(12)
    gc, tc = get_preset("mla")
    gc.hidden_size, gc.n_heads, gc.n_kv_heads = 128, h, h
    gc.mla_kv_rank, gc.mla_qk_rope_dim, gc.mla_qk_content_dim, gc.mla_value_dim, gc.mla_q_rank = r, 32, 32, 32, 0
    tc.seq_len_train = tc.seq_len_val = t + 64
    tc.resolve(1)
    attn = MLAttention(gc, tc).cuda().eval()
    x = torch.randn(b, t, 128, device="cuda").bfloat16()
    whole = attn.allocate_cache(b, t + 2, device="cuda", dtype=torch.bfloat16)
    got = attn.forward_cached(x, whole, 0)
    parts = attn.allocate_cache(b, t + 2, device="cuda", dtype=torch.bfloat16)
    if t > 1:                                                # the same tokens in calls of 32768
        want = torch.cat([attn.forward_cached(x[:, i: i + 32768], parts, 0) for i in range(0, t, 32768)], dim=1)
    else:
        want = torch.empty_like(got)
        for i in range(0, b, 32768):
            part = attn.allocate_cache(min(32768, b - i), t + 2, device="cuda", dtype=torch.bfloat16)
            want[i: i + 32768] = attn.forward_cached(x[i: i + 32768], part, 0)
            parts.latent[i: i + 32768] = part.latent
    assert whole.latent[:, :t].abs().sum(dim=-1).min() > 0 and torch.equal(whole.latent, parts.latent)
    assert torch.equal(got, want)
    from gpt_moe_b200.ops import cuda_ops
    cuda_ops.check_status()


# one and two tiles of rows, every rank
@pytest.mark.parametrize("b,t,h,hkv,r,dr,s", [(2, 1, 16, 16, 512, 64, 777), (4, 1, 16, 16, 512, 64, 4022), (1, 5, 8, 2, 256, 32, 300), (2, 1, 32, 32, 512, 64, 130), (1, 2, 16, 4, 768, 64, 500), (1, 1, 8, 8, 1024, 10, 90)])
def test_a_context_in_fp32_has_the_bits_of_fp32(b, t, h, hkv, r, dr, s):
    from gpt_moe_b200.models.mla import api_mla_decode
    torch.manual_seed(15)
    q, qr = 0.3 * torch.randn(b, t, h, r, device="cuda"), torch.randn(b, t, h, dr, device="cuda")
    lat, rope = torch.randn(b, s, r, device="cuda").bfloat16(), torch.randn(b, s, dr, device="cuda").bfloat16()
    gain = (torch.rand(b, s, hkv, device="cuda") + 0.5).bfloat16()
    got = api_mla_decode(q, qr, lat, rope, gain, s - t, 0.08, 0.0, "exact", None)
    score = torch.einsum("bthr,bsr->bhts", q.double(), lat.double()) + torch.einsum("bthd,bsd->bhts", qr.double(), rope.double())
    score = score * gain.double().permute(0, 2, 1).repeat_interleave(h // hkv, dim=1)[:, :, None, :] * 0.08
    keep = torch.arange(s, device="cuda")[None, :] <= torch.arange(s - t, s, device="cuda")[:, None]
    want = torch.einsum("bhts,bsr->bthr", torch.softmax(score.masked_fill(~keep, float("-inf")), dim=-1), lat.double())
    assert rel(got, want) < 6e-7                                  # 2e-7 to 4e-7 with fp32 products and sums throughout


# low ranks and few positions, measured in us absorbed / expanded: 150 / 85, 320 / 177, 93 / 73, 50 / 38, 138 / 110; and the other way: 297 / 357, 39 / 78
@pytest.mark.parametrize("b,t,h,hkv,end,r,expanded", [(4, 24, 32, 8, 1524, 256, True), (4, 24, 32, 8, 4024, 256, True), (1, 64, 32, 8, 1564, 256, True),
                                                      (4, 16, 16, 4, 16, 512, True), (4, 32, 16, 16, 1532, 512, True), (2, 48, 16, 16, 8048, 512, False),
                                                      (1, 16, 16, 16, 1516, 512, False)])
def test_the_form_follows_what_the_expansion_costs(b, t, h, hkv, end, r, expanded):
    from gpt_moe_b200.ops import cuda_ops
    assert cuda_ops.ext().mla_prefill_wanted(b, t, h, hkv, end, -1, r, 64, 64, 64, 0.0) == expanded


@pytest.mark.parametrize("expanded", [True, False])
@pytest.mark.parametrize("b,t,h,hkv,r,start", [(1, 500, 8, 8, 256, 300), (2, 130, 16, 4, 512, 360)])
def test_only_the_output_is_rounded_to_bf16(b, t, h, hkv, r, start, expanded):
    """Against 64 bits on what lies in the cache afterwards: queries, keys, probabilities and values keep more bits than bf16 in both forms."""
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(16)
    end = start + t
    width = h * 128 + (0 if expanded else 2)                        # rows on no 8-byte boundary stay with the absorbed form
    query = (2 * torch.randn(b * t, width, device="cuda")).bfloat16()[:, :h * 128]
    low = torch.randn(b * t, r + 64, device="cuda").bfloat16()
    w = torch.randn(hkv * 128, r, device="cuda") * r ** -0.5
    cos, sin = torch.rand(end, 32, device="cuda"), torch.rand(end, 32, device="cuda")
    qs, ks = torch.linspace(0.5, 3.0, h, device="cuda"), torch.linspace(0.5, 2.0, hkv, device="cuda")
    lat, rope = torch.randn(b, end, r, device="cuda").bfloat16(), torch.randn(b, end, 64, device="cuda").bfloat16()
    gain = (torch.rand(b, end, hkv, device="cuda") + 0.5).bfloat16()
    assert cuda_ops.ext().mla_prefill_wanted(b, t, h, hkv, end, -1, r, 64, 64, 64, 0.0)
    got = cuda_ops.ext().mla_cached(query, low, w, None, 1e-6, cos, sin, qs, ks, 1e-6, True, -3e38, 3e38, lat, rope, gain, start, h, 64, 64, 128 ** -0.5, 0.0, -1)
    q = query.double().view(b, t, h, 128)
    norm = torch.rsqrt(q.pow(2).mean(-1, keepdim=True) + 1e-6) * qs.double().view(1, 1, -1, 1)
    x0, x1 = q[..., 64::2], q[..., 65::2]
    c, s = (m[start:].double()[None, :, None] for m in (cos, sin))
    q = torch.cat((q[..., :64], torch.stack((x0 * c - x1 * s, x0 * s + x1 * c), dim=-1).flatten(-2)), dim=-1) * norm
    kv = torch.einsum("bsr,hdr->bshd", lat.double(), w.double().view(hkv, 128, r))
    key = torch.cat((kv[..., :64], rope.double()[:, :, None].expand(-1, -1, hkv, -1)), dim=-1) * gain.double()[..., None]
    score = torch.einsum("bthd,bshd->bhts", q, key.repeat_interleave(h // hkv, dim=2)) * 128 ** -0.5
    keep = torch.arange(end, device="cuda")[None, :] <= torch.arange(start, end, device="cuda")[:, None]
    want = torch.einsum("bhts,bshd->bthd", torch.softmax(score.masked_fill(~keep, float("-inf")), dim=-1), kv[..., 64:].repeat_interleave(h // hkv, dim=2))
    assert rel(got.view(b, t, h, 64), want) < 1.8e-3                # the rounding itself: 1.65e-3 of the norm; one of the queries alone adds as much
    cuda_ops.check_status()


@pytest.mark.parametrize("rows,n,k", [(1, 16, 32), (8, 576, 1024), (9, 8, 96), (17, 2624, 1024), (32, 24, 64)])
def test_rows_linear_matches_matmul(rows, n, k):
    from gpt_moe_b200.ops import cuda_ops
    torch.manual_seed(3)
    x, w = torch.randn(rows, k, device="cuda").bfloat16(), torch.randn(n, k, device="cuda").bfloat16()
    want = x.double() @ w.double().t()
    assert rel(cuda_ops.ext().rows_linear(x, w), want) < 3e-3         # fp32 sums, one rounding of the result
