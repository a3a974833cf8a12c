"""What this framework is used for, as cases whose speed and results can be measured.

Five kinds, each through the call that a user makes:

  train      one optimizer step, `Trainer.train_step` on a pinned host batch: forward, backward, Muon with Polar Express, AdamW
  validate   the loss of one validation batch, `GPT.forward` with targets in eval mode
  logits     the logits of a padded batch of prompts, `GPT.forward` without targets: every token of `sampling.sample`, and
             HellaSwag scoring, which then takes the continuation's log-probabilities from them
  mla        new tokens against the latent cache, `MLAttention.forward_cached`: one token a call is decoding, many are prefill
  attention  forward and backward of the attention op alone, `ops.api.attention`: long contexts, grouped heads, soft-capping, odd lengths

Widths, head counts, experts and windows are those of the presets "small", "wide_ep" and "mla"; layers, experts and batch are
scaled so that a model fits one GPU without its expert-parallel peers.

The models have random weights, with one thing of a trained model put in: a router that tells tokens apart.  Token embeddings
carry a component that names the token's cluster and the router rows point along those components, so that the top choices
stand well clear of the rest (as they do in training once experts have specialised) and experts get unequal shares of the
tokens.  With a random router thousands of tokens are near ties, and the last bit of a bf16 logit would decide them.
"""
from __future__ import annotations

import gc as garbage
import math

import torch

from gpt_moe_b200.config import get_preset
from gpt_moe_b200.evaluation.hellaswag import continuation_scores
from gpt_moe_b200.models.gpt import GPT
from gpt_moe_b200.models.mla import MLAttention
from gpt_moe_b200.ops import api, cuda_ops
from gpt_moe_b200.runtime import trainer as trainer_module
from gpt_moe_b200.runtime.precision import precision_context
from gpt_moe_b200.runtime.trainer import Trainer
from gpt_moe_b200.schedules.token import custom_schedule

VOCAB = 50304


# ---- the cases ------------------------------------------------------------------------------------------------------------
def _train(name, model, layers, experts, batch, seq, window, precision, docs=False):
    return dict(name=name, kind="train", model=model, layers=layers, experts=experts, batch=batch, seq=seq, window=window,
                precision=precision, docs=docs)


def _logits(name, batch, seq, score, layers=12):
    return dict(name=name, kind="logits", model="small", layers=layers, experts=8, batch=batch, seq=seq, window=1024, score=score)


def _mla(name, batch, start, new, window=-1):
    return dict(name=name, kind="mla", batch=batch, start=start, new=new, window=window)


def _attention(name, batch, seq, heads, kv_heads, qk_dim, window, softcap=0.0):
    return dict(name=name, kind="attention", batch=batch, seq=seq, heads=heads, kv_heads=kv_heads, qk_dim=qk_dim, window=window,
                softcap=softcap)


def listed():
    return [
        # the benchmark's own configuration and batch, projections in MXFP8: what a training run repeats a hundred thousand times
        _train("train_small", "small", 12, 8, 16, 2048, 1024, "mxfp8"),
        # 32 narrow experts, two per token, every GEMM in bf16, documents kept apart, a batch that is no power of two
        _train("train_wide_docs", "wide_ep", 4, 32, 3, 1280, 512, "default", docs=True),
        # latent attention over 4096 tokens, one rank's share of the routed experts beside the shared one
        _train("train_mla", "mla", 3, 8, 2, 4096, 4096, "mxfp8"),
        # a short step on a shallow model (first trials, smoke runs): optimizer and launches outweigh the tokens
        _train("train_short", "small", 2, 8, 2, 512, 1024, "mxfp8"),
        # the validation batch of the same run
        dict(name="validate_small", kind="validate", model="small", layers=12, experts=8, batch=16, seq=2048, window=1024),
        # 16 HellaSwag examples with their four endings, one-shot prompt, padded to a multiple of 8
        _logits("score_hellaswag", 64, 184, True),
        # a token of eight sampled texts, mid-way through
        _logits("sample_step", 8, 45, False),
        # decoding one token for eight sequences, cache filled to 4000 and something
        _mla("mla_decode", 8, 4021, 1),
        # a chunk of a prompt appended to a cache that already holds 1500 tokens
        _mla("mla_prefill", 2, 1500, 512),
        # full causal attention over a long context with four query heads to a key head
        _attention("attention_long", 1, 16384, 16, 4, 64, 0),
        # a length that is no multiple of any tile
        _attention("attention_ragged", 5, 1000, 12, 12, 64, 256),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("train", "train", "train", "validate", "logits", "logits", "mla", "mla", "attention", "attention"))
    if kind == "train":
        model = rng.choice(("small", "small", "wide_ep", "mla"))
        layers = _log_int(rng, 2, 12) if model == "small" else rng.randint(2, 4)
        experts = {"small": 8, "wide_ep": rng.choice((16, 32)), "mla": 8}[model]
        batch = _log_int(rng, 1, 16 if model != "mla" else 4)
        # sequence lengths are multiples of the mask block of 128 in training configurations, and now and then they are not
        seq = 128 * _log_int(rng, 2, 16) if rng.random() < 0.8 else 8 * rng.randint(20, 200)
        docs = model != "mla" and seq % 128 == 0 and rng.random() < 0.3
        window = seq if model == "mla" else 128 * rng.randint(1, 8)
        case = _train("", model, layers, experts, batch, seq, window, rng.choice(("mxfp8", "mxfp8", "default")), docs)
    elif kind == "validate":
        case = dict(kind="validate", model=rng.choice(("small", "small", "wide_ep")), layers=rng.randint(2, 12), experts=8,
                    batch=_log_int(rng, 1, 16), seq=128 * _log_int(rng, 2, 16), window=128 * rng.randint(1, 8))
    elif kind == "logits":
        score = rng.random() < 0.5
        case = _logits("", 4 * _log_int(rng, 4, 16) if score else _log_int(rng, 1, 16), 8 * rng.randint(14, 30) if score else _log_int(rng, 6, 1000),
                       score, rng.randint(4, 12))
    elif kind == "mla":
        new = 1 if rng.random() < 0.6 else _log_int(rng, 2, 512)
        case = _mla("", _log_int(rng, 1, 32 if new == 1 else 4), _log_int(rng, 30, 8000), new, rng.choice((-1, -1, 1024)))
    else:
        seq = rng.choice((128 * _log_int(rng, 1, 96), rng.randint(100, 6000)))
        heads, kv_heads = rng.choice(((12, 12), (16, 4), (16, 16), (16, 1)))
        qk_dim = 128 if seq % 128 == 0 and rng.random() < 0.25 else 64
        batch = _log_int(rng, 1, max(1, min(8, 16384 // seq)))
        window = rng.choice((0, 128 * rng.randint(1, 8)))
        case = _attention("", batch, seq, heads, heads if qk_dim == 128 else kv_heads, qk_dim, window,
                          15.0 if qk_dim == 64 and seq % 128 == 0 and rng.random() < 0.15 else 0.0)
    case.pop("name", None)
    return case


# ---- models and inputs ----------------------------------------------------------------------------------------------------
def _configs(case, seed):
    preset = case["model"]
    gc, tc = get_preset(preset, precision=case.get("precision", "mxfp8"))
    gc.n_layers, gc.num_experts = case["layers"], case["experts"]
    gc.weighted_main_path_init = 0.15                   # every branch takes part, as after some training
    gc.use_doc_masking = bool(case.get("docs", False))
    tc.gpu_batch_size_train = tc.gpu_batch_size_val = case["batch"]
    tc.seq_len_train = tc.seq_len_val = max(case["seq"], 64)
    tc.expert_parallel_size = 1
    tc.kernel_warmup_train_steps = 0
    tc.adamw_max_lr = tc.adamw_hard_min_lr              # the late, long part of the learning-rate schedule
    tc.base_seed = seed
    tc.batch_size_values_schedule = {"fn": custom_schedule, "kwargs": {"values": [case["batch"]]}}
    tc.swa_values_schedule = {"fn": custom_schedule, "kwargs": {"values": [case["window"]]}}
    return gc, tc


@torch.no_grad()
def _specialise_router(model, gc, seed):
    """Clusters of tokens, and routers that see them (see the head of the file)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    d, experts = gc.hidden_size, gc.num_experts
    axes = torch.linalg.qr(torch.randn(d, experts, generator=gen, device="cuda"))[0].t()          # orthonormal rows
    share = 1.0 / (torch.arange(experts, device="cuda") + experts / 2.0)                          # unequal shares, at most 3 to 1
    first = torch.multinomial(share, gc.vocab_size, replacement=True, generator=gen)
    second = (first + torch.randint(1, experts, (gc.vocab_size,), generator=gen, device="cuda")) % experts
    wte = model.transformer.wte.weight
    wte.copy_(0.6 * torch.randn(wte.shape, generator=gen, device="cuda") + 10.0 * axes[first] + 6.0 * axes[second])
    for block in model.transformer.h:
        order = torch.randperm(experts, generator=gen, device="cuda")
        block.mlp.router.weight.copy_(0.35 * axes[order])


def _tokens(case, seed, columns):
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    return torch.randint(0, VOCAB, (case["batch"], columns), generator=gen, device="cuda")


def _gpt_on_gpu(*args, **kwargs):
    """The model with its parameters drawn on the GPU: on the host that takes ten seconds for the large ones."""
    with torch.device("cuda"):
        return GPT(*args, **kwargs)


def _prepare_train(case, seed):
    gc, tc = _configs(case, seed)
    try:
        trainer_module.GPT = _gpt_on_gpu
        trainer = Trainer(gc, tc, device_type="cuda", quiet=True)
    finally:
        trainer_module.GPT = GPT
    _specialise_router(trainer.raw_gpt_model, gc, seed)
    trainer.engine.refresh_from_parameters()
    ids = _tokens(case, seed, case["seq"] + 1).cpu()
    docs = None
    if case["docs"]:                                    # documents of some 300 tokens
        gen = torch.Generator().manual_seed(seed)
        ends = torch.rand(case["batch"], case["seq"], generator=gen) < 1 / 300
        docs = (ends.int().cumsum(1) - ends.int()).int().pin_memory()
    state = dict(trainer=trainer, batch=[(ids[:, :-1].contiguous().pin_memory(), ids[:, 1:].contiguous().pin_memory(), docs)])
    for _ in range(3):                                  # a run that is under way: momentum is there, the step's graph captured
        trainer.train_step(state["batch"])
    return state


def _prepare_model(case, seed):
    gc, tc = _configs(case, seed)
    tc.resolve(1)
    torch.manual_seed(seed)
    model = _gpt_on_gpu(gc, tc)
    _specialise_router(model, gc, seed)
    model.set_sliding_window(case["window"])
    model.eval()
    model.set_precision_phase("validation" if case["kind"] == "validate" else "evaluation")
    state = dict(model=model, ctx=precision_context(tc, "cuda"))
    ids = _tokens(case, seed, case["seq"] + 1)
    state["x"], state["y"] = ids[:, :-1].contiguous(), ids[:, 1:].contiguous()
    if case.get("score"):                               # endings of 8 to 40 tokens; rows are padded on the right
        gen = torch.Generator().manual_seed(seed)
        true = torch.randint(case["seq"] - 24, case["seq"] + 1, (case["batch"],), generator=gen)
        state["true"] = true.tolist()
        state["prefix"] = (true - torch.randint(8, 40, (case["batch"],), generator=gen)).tolist()
    return state


def _prepare_mla(case, seed):
    gc, tc = get_preset("mla")
    tc.seq_len_train = tc.seq_len_val = max(64, case["start"] + case["new"])
    tc.resolve(1)
    torch.manual_seed(seed)
    with torch.device("cuda"):
        attn = MLAttention(gc, tc)
        for p in attn.parameters():
            if p.dim() == 2:
                torch.nn.init.normal_(p, std=0.02)
    attn.requires_grad_(False).eval()
    cache = attn.allocate_cache(case["batch"], case["start"] + case["new"], device="cuda", dtype=torch.bfloat16)
    # what earlier calls have left there: a normalised latent, a rope key, the gain of the QK-norm
    cache.latent.normal_()
    cache.rope.normal_(std=0.5)
    cache.key_gain.uniform_(1.0, 3.0)
    x = torch.randn(case["batch"], case["new"], gc.hidden_size, device="cuda").bfloat16()          # rows of a preceding RMSNorm
    return dict(attn=attn, cache=cache, x=x, start=case["start"], window=None if case["window"] < 0 else case["window"])


def _prepare_attention(case, seed):
    torch.manual_seed(seed)
    b, t, h, hk, d = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "qk_dim"))
    # queries and keys as QK-norm leaves them: unit mean square
    q, k = (torch.nn.functional.rms_norm(torch.randn(b, t, n, d, device="cuda"), (d,)).bfloat16().requires_grad_() for n in (h, hk))
    v = torch.randn(b, t, hk, 64, device="cuda").bfloat16().requires_grad_()
    d_out = torch.randn(b, t, h, 64, device="cuda").bfloat16()
    return dict(q=q, k=k, v=v, d_out=d_out, window=case["window"] or None, softcap=case["softcap"])


def prepare(case, seed):
    # one process goes through many models: let go of what is left of those that are gone
    garbage.collect()
    cuda_ops.clear_weight_cache()
    kind = case["kind"]
    if kind == "train":
        state = _prepare_train(case, seed)
    elif kind == "mla":
        state = _prepare_mla(case, seed)
    elif kind == "attention":
        state = _prepare_attention(case, seed)
    else:
        state = _prepare_model(case, seed)
    state["kind"] = kind
    return state


def run(state):
    kind = state["kind"]
    if kind == "train":
        trainer = state["trainer"]
        stats = trainer.train_step(state["batch"])
        engine = trainer.engine
        return dict(loss=stats["loss"], token_loss=stats["token_loss"], balance=stats["balance_term"],
                    matrix_grads=engine.grad_muon.tensor, other_grads=engine.adamw_grad.tensor,
                    matrix_weights=engine.compute.tensor, other_weights=engine.adamw_param.tensor)
    if kind == "mla":
        cache, x = state["cache"], state["x"]
        start = cache.length = state["start"]
        out = state["attn"].forward_cached(x, cache, state["window"])
        end = cache.length
        return out, cache.latent[:, start:end], cache.rope[:, start:end], cache.key_gain[:, start:end]
    if kind == "attention":
        q, k, v = state["q"], state["k"], state["v"]
        out = api.attention(q, k, v, window=state["window"], softcap_value=state["softcap"], tanh_backend="ptx")
        return (out,) + torch.autograd.grad(out, (q, k, v), state["d_out"])
    model = state["model"]
    with torch.no_grad(), state["ctx"]:
        if kind == "validate":
            return model(state["x"], state["y"])
        logits = model(state["x"], attn_mask=None, ignore_doc_mask=True)
        if "true" not in state:
            return logits
        return logits, continuation_scores(logits, state["x"], state["prefix"], state["true"])


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------
def _pairs(seq, window):
    """Query-key pairs of one causal head."""
    w = seq if window <= 0 else min(window, seq)
    return sum(min(i, w) + 1 for i in range(seq))


def _shapes(case):
    """(rows, cols, how many, how many of them one token meets) of the matrices of one layer."""
    gc, _ = get_preset(case["model"])
    d, e, k = gc.hidden_size, case["experts"], gc.moe_top_k
    m = gc.mlp_hidden_dim
    shapes = [(2 * m, d, e, k), (d, m, e, k), (e, d, 1, 1)]
    if gc.use_mla:
        head = gc.mla_qk_content_dim + gc.mla_qk_rope_dim
        s = gc.moe_shared_expert_hidden_dim
        shapes += [(gc.n_heads * head, d, 1, 1), (gc.mla_kv_rank + gc.mla_qk_rope_dim, d, 1, 1),
                   (gc.n_heads * (gc.mla_qk_content_dim + gc.mla_value_dim), gc.mla_kv_rank, 1, 1),
                   (d, gc.n_heads * gc.mla_value_dim, 1, 1), (2 * s, d, 1, 1), (d, s, 1, 1)]
        return gc, shapes, head
    return gc, shapes + [(gc.attn_dim, d, 4, 4)], gc.head_size


def work(case):
    if case["kind"] == "attention":
        b, t, h, hk, d = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "qk_dim"))
        pairs = b * h * _pairs(t, case["window"])
        values = b * t * (h * d + hk * d + hk * 64 + h * 64)
        # forward reads q, k, v and writes the output; backward reads those and the output's gradient and writes three gradients
        return dict(bytes=2 * (values + values + b * t * h * 64 + b * t * (h * d + hk * d + hk * 64)), flops=pairs * 2 * (4 * d + 3 * 64))
    if case["kind"] == "mla":
        gc, _ = get_preset("mla")
        b, t, s = case["batch"], case["new"], case["start"] + case["new"]
        r, dr, h, c, v = gc.mla_kv_rank, gc.mla_qk_rope_dim, gc.n_heads, gc.mla_qk_content_dim, gc.mla_value_dim
        seen = min(s, case["window"] + t) if case["window"] >= 0 else s
        weights = gc.hidden_size * (h * (c + dr) + r + dr) + h * (c + v) * r + h * v * gc.hidden_size
        rows = b * t
        return dict(bytes=2 * weights + 2 * b * seen * (r + dr + h) + 4 * rows * gc.hidden_size,
                    flops=rows * (2 * weights + 2 * h * c * r) + b * t * h * seen * 2 * (2 * r + dr))
    gc, shapes, head = _shapes(case)
    layers, tokens = case["layers"], case["batch"] * case["seq"]
    value = gc.mla_value_dim if gc.use_mla else head
    per_token = layers * sum(r * c * met for r, c, _, met in shapes) + gc.hidden_size * VOCAB
    matrices = layers * sum(r * c * n for r, c, n, _ in shapes)
    pairs = layers * case["batch"] * gc.n_heads * _pairs(case["seq"], case["window"])
    if case["kind"] != "train":
        logits = 2 * tokens * VOCAB if case["kind"] == "logits" else 0
        return dict(bytes=2 * matrices + 2 * gc.hidden_size * VOCAB + logits + 4 * tokens * gc.hidden_size,
                    flops=2 * tokens * per_token + pairs * 2 * (head + value))
    # Polar Express in its cheapest form: one Gram product, five quintic steps on the small side, one product back
    polar = layers * sum(n * (3 * min(r, c) ** 2 * max(r, c) + 15 * min(r, c) ** 3) for r, c, n, _ in shapes)
    # every matrix: master and momentum read and written, gradient written and read, bf16 copy written; embedding and head: AdamW
    return dict(bytes=matrices * (8 + 8 + 8 + 2) + 2 * gc.hidden_size * VOCAB * 32,
                flops=6 * tokens * per_token + pairs * 2 * (4 * head + 3 * value) + polar)


# ---- the same in 64 bits -------------------------------------------------------------------------------------------------
def _visible(rows, cols, start, window):
    """rows x cols truth values: query i sits at position start + i and looks `window` positions back (None: all the way)."""
    q = torch.arange(start, start + rows, device="cuda")[:, None]
    k = torch.arange(cols, device="cuda")[None, :]
    keep = k <= q
    return keep if window is None else keep & (q - k <= window)


def _exact_attention(case, seed):
    state = _prepare_attention(case, seed)
    q, k, v, d_out = (state[n].detach().double() for n in ("q", "k", "v", "d_out"))
    b, t, h, d = q.shape
    group, window, cap = h // k.shape[2], state["window"], state["softcap"]
    out, dq, dk, dv = torch.empty_like(d_out), torch.empty_like(q), torch.zeros_like(k), torch.zeros_like(v)
    step = max(1, min(t, (1 << 27) // t))                # rows at a time: a gigabyte of scores
    for i in range(b):
        for j in range(h):
            kj, vj = k[i, :, j // group], v[i, :, j // group]
            for r in range(0, t, step):
                rows = slice(r, min(r + step, t))
                s = q[i, rows, j] @ kj.t() * d ** -0.5
                slope = None
                if cap:
                    th = torch.tanh(s / cap)
                    s, slope = cap * th, 1 - th * th
                p = torch.softmax(s.masked_fill(~_visible(s.shape[0], t, r, window), -math.inf), dim=-1)
                o, g = p @ vj, d_out[i, rows, j]
                out[i, rows, j] = o
                dv[i, :, j // group] += p.t() @ g
                ds = p * (g @ vj.t() - (g * o).sum(-1, keepdim=True)) * d ** -0.5
                if slope is not None:
                    ds = ds * slope
                dq[i, rows, j] = ds @ kj
                dk[i, :, j // group] += ds.t() @ q[i, rows, j]
    return out, dq, dk, dv


def _exact_mla(case, seed):
    state = _prepare_mla(case, seed)
    gc, _ = get_preset("mla")
    attn, cache, x, start = state["attn"], state["cache"], state["x"].double(), state["start"]
    par = {name: p.detach().double() for name, p in attn.named_parameters()}
    b, t, _ = x.shape
    h, r, dr, c, dv = gc.n_heads, gc.mla_kv_rank, gc.mla_qk_rope_dim, gc.mla_qk_content_dim, gc.mla_value_dim

    def rotate(y):                                       # [b, t, heads, dr], pairs of neighbours
        freq = gc.rope_base_theta ** (-torch.arange(0, dr, 2, device="cuda", dtype=torch.float64) / dr)
        angle = torch.arange(start, start + t, device="cuda", dtype=torch.float64)[:, None] * freq
        cos, sin = angle.cos()[None, :, None], angle.sin()[None, :, None]
        a, o = y[..., 0::2], y[..., 1::2]
        return torch.stack((a * cos - o * sin, a * sin + o * cos), dim=-1).flatten(-2)

    def gain(y, scale):
        return torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + gc.qk_eps) * scale.clamp(gc.qk_scale_min, gc.qk_scale_max).view(1, 1, -1, 1)

    q = (x @ par["q_proj.weight"].t()).view(b, t, h, c + dr)
    q = torch.cat((q[..., :c], rotate(q[..., c:])), dim=-1)
    low = x @ par["kv_down_proj.weight"].t()
    lat = low[..., :r]
    lat = lat * torch.rsqrt(lat.pow(2).mean(-1, keepdim=True) + gc.mla_norm_eps) * par["kv_norm.weight"]
    rope = rotate(low[..., None, r:])
    w = par["kv_up_proj.weight"].view(h, c + dv, r)
    key = torch.cat((torch.einsum("btr,hdr->bthd", lat, w[:, :c]), rope.expand(-1, -1, h, -1)), dim=-1)
    new_gain = gain(key, par["k_scale"])[..., 0]
    q = q * gain(q, par["q_scale"])
    q_lat = torch.einsum("bthd,hdr->bthr", q[..., :c], w[:, :c])
    context = torch.empty(b, t, h, r, device="cuda", dtype=torch.float64)
    for i in range(b):
        ci, ri, gi = (torch.cat((old[i, :start].double(), new[i]), dim=0) for old, new in ((cache.latent, lat), (cache.rope, rope[:, :, 0]), (cache.key_gain, new_gain)))
        keep = _visible(t, start + t, start, state["window"])
        for j in range(h):
            s = (q_lat[i, :, j] @ ci.t() + q[i, :, j, c:] @ ri.t()) * gi[:, j] * (c + dr) ** -0.5
            context[i, :, j] = torch.softmax(s.masked_fill(~keep, -math.inf), dim=-1) @ ci
    out = torch.einsum("bthr,hdr->bthd", context, w[:, c:]).flatten(-2) @ par["out_proj.weight"].t()
    return out, lat, rope[:, :, 0], new_gain


def exact(case, seed):
    """The single layers in 64 bits; a whole model has no such answer that its roundings would not hide."""
    with torch.no_grad():
        return _exact_attention(case, seed) if case["kind"] == "attention" else _exact_mla(case, seed) if case["kind"] == "mla" else None


def tolerance(case):
    """About four times what was measured between correct ways of computing the same: attention by another kernel with another
    order of its sums, or in fp32 on whole score matrices.  Training compares the fourth step of a run, gradients included."""
    if case["kind"] == "train":
        # the e4m3 payload of a value near a rounding boundary flips with the last bit of what came before: 1.0e-2, single
        # elements 0.56; in bf16 2.1e-3, 0.10
        return {"rel": 3e-2, "max": 0.99} if case["precision"] == "mxfp8" else {"rel": 1e-2, "max": 0.4}
    if case["kind"] == "validate":
        return {"rel": 5e-5}                            # a mean over the tokens: 2e-7 at 32768 of them, 1e-5 at a few hundred
    if case["kind"] == "logits":
        return {"rel": 1e-2, "max": 0.06}               # 2.4e-3, 0.014: bf16 activations through twelve layers
    if case["kind"] == "mla":
        return {"rel": 1e-2, "max": 0.1}                # two roundings to bf16 (attention output, projection), 2e-3 each
    return {"rel": 1.2e-2, "max": 0.3}                  # 2.8e-3, 0.076: probabilities and results in bf16
