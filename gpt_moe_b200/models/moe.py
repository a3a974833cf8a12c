"""Dropless token-choice mixture of experts.

Router in fp32, top-k selection, Switch-style load-balance loss, then sort-by-expert grouped
expert computation and a gate-weighted combine — no capacity factor, no dropped tokens
(reference `model/feedforward/moe.py:21-134`).  Parameter layout is the reference's:
`router.weight [E, hidden]`, `experts.{e}.up_proj.weight`, `experts.{e}.down_proj.weight`.

New here: an optional always-on shared expert (`shared_expert`, its own width) and expert
parallelism — with `expert_parallel_size > 1` each rank holds `num_experts / ep` experts and the
tokens travel by a counted all-to-all (see `parallel/ep.py`); the module's parameters are then
only the local experts, named by their GLOBAL index so checkpoints stay in the unsharded layout.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch.nn as nn
from torch import Tensor

from ..ops import api
from .linear import Linear
from .mlp import MLP


class MoE(nn.Module):
    def __init__(self, gpt_config, training_config, num_experts: int, top_k: int = 2,
                 ep_rank: int = 0, ep_size: int = 1) -> None:
        super().__init__()
        assert num_experts % ep_size == 0, "expert_parallel_size must divide num_experts"
        self.num_experts, self.top_k = num_experts, top_k
        self.ep_rank, self.ep_size = ep_rank, ep_size
        self.experts_per_rank = num_experts // ep_size
        self.first_expert = ep_rank * self.experts_per_rank
        self.full_softmax_gating = gpt_config.moe_full_softmax_gating
        self.load_balance_weight = training_config.moe_load_balance_weight
        self.router = Linear(gpt_config.hidden_size, num_experts, role="router", bias=False)
        # keys are global expert indices: experts.{e}.up_proj.weight.  All experts are constructed so that the
        # initial weights do not depend on the sharding; `keep_local_experts()` drops the others after init.
        self.experts = nn.ModuleDict({str(e): MLP(gpt_config, training_config) for e in range(num_experts)})
        self.shared_expert = (MLP(gpt_config, training_config, hidden_dim=gpt_config.moe_shared_expert_hidden_dim)
                              if gpt_config.moe_shared_expert_hidden_dim > 0 else None)
        self.ep_group = None            # set by parallel.ep.attach_expert_parallel

    def keep_local_experts(self) -> None:
        for e in range(self.num_experts):
            if not self.first_expert <= e < self.first_expert + self.experts_per_rank:
                del self.experts[str(e)]

    def local_experts(self):
        return [self.experts[str(e)] for e in range(self.first_expert, self.first_expert + self.experts_per_rank)]

    def _forward_plain(self, hidden: Tensor) -> Optional[Tensor]:
        """The routed experts without gradients as one call (`moe_branch`): same launches, a fraction of the host time.  None when an
        option or shape needs the general path."""
        from ..ops import cuda_ops
        if not cuda_ops.plain_call() or self.ep_size > 1 or (self.training and self.load_balance_weight > 0):
            return None
        router = self.router
        # straight from the modules' tables: attribute access on a module costs a microsecond, and there are four per expert
        experts = self.experts._modules
        mlps = [experts[str(e)]._modules for e in range(self.num_experts)]
        ups, downs = [m["up_proj"] for m in mlps], [m["down_proj"] for m in mlps]
        for m in (router, ups[0], downs[0]):
            if type(m) is not Linear or m.bias is not None or m.precision != "default":
                return None
        w_up, w_down = [m._parameters.get("weight") for m in ups], [m._parameters.get("weight") for m in downs]
        d, up_n = w_up[0].shape[1] if w_up[0] is not None else 0, w_up[0].shape[0] if w_up[0] is not None else 0
        if (any(w is None for w in w_up) or any(w is None for w in w_down) or not cuda_ops.bypassable(router)
                or self.num_experts % 8 or self.num_experts > 128 or self.top_k > 8 or d % 8 or up_n % 16 or w_down[0].shape[0] % 8):
            return None
        renormalise = not (self.top_k == 1 or self.full_softmax_gating)
        out = cuda_ops.ext().moe_branch(
            cuda_ops._as_bf16_2d(hidden), cuda_ops.bf16_weight((router.weight,)), self.top_k, renormalise, cuda_ops.stacked_weight(w_up),
            cuda_ops.stacked_weight(w_down), experts["0"].activation_name)
        return out if hidden.dtype == out.dtype else out.to(hidden.dtype)

    def forward(self, x: Tensor) -> Tuple[Tensor, Optional[Tensor]]:
        shape = x.shape
        hidden = x.reshape(-1, shape[-1])
        if hidden.is_cuda:
            out = self._forward_plain(hidden)
            if out is not None:
                if self.shared_expert is not None:
                    out = out + self.shared_expert(hidden)
                return out.reshape(shape), None
        logits = self.router(hidden)
        want_balance = bool(self.training and self.load_balance_weight > 0)
        top_idx, gates, balance = api.router(logits, self.top_k, self.full_softmax_gating, want_balance, self.num_experts)
        experts = self.local_experts()
        first = experts[0]
        args = dict(
            up_weights=[m.up_proj.weight for m in experts], down_weights=[m.down_proj.weight for m in experts],
            up_biases=None if first.up_proj.bias is None else [m.up_proj.bias for m in experts],
            down_biases=None if first.down_proj.bias is None else [m.down_proj.bias for m in experts],
            activation=first.activation_name, up_precision=first.up_proj.precision,
            down_precision=first.down_proj.precision)
        if self.ep_size > 1:
            from ..parallel.ep import expert_parallel_moe
            out = expert_parallel_moe(self, hidden, top_idx, gates, args)
        else:
            out = api.moe_experts(hidden, top_idx, gates, **args)
        if self.shared_expert is not None:
            out = out + self.shared_expert(hidden)
        return out.reshape(shape), balance
