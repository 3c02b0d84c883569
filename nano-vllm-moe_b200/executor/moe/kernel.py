"""prepare -> experts -> finalize (reference: executor/moe/kernel.py:14-78)."""
from __future__ import annotations

import torch
import torch.distributed as dist

from ... import _lib
from .config import MoEParallelConfig
from .experts import Fp8Experts, Fp8ExpertWeights
from .prepare_finalize import NoEPPrepareFinalize


class MoEKernel:
    def __init__(self, *, prepare_finalize, experts: Fp8Experts, parallel_config: MoEParallelConfig) -> None:
        self.prepare_finalize = prepare_finalize
        self.experts = experts
        self.parallel_config = parallel_config

    def __call__(self, x: torch.Tensor, topk_weights: torch.Tensor, topk_ids: torch.Tensor, weights: Fp8ExpertWeights,
                 *, model_dtype: torch.dtype, reduce_tp: bool = True) -> torch.Tensor:
        if (type(self.prepare_finalize) is NoEPPrepareFinalize and type(self.experts) is Fp8Experts and model_dtype == torch.bfloat16
                and x.is_cuda and x.dtype == torch.bfloat16 and topk_ids.dim() == 2 and weights.hidden_size % 8 == 0):
            # every expert is local and nothing moves: grouping, both projections and the k-slot sum are one native call
            out = _lib.host().moe_block(x, topk_weights, topk_ids, weights.w13_packed, weights.w13_scale, weights.w13_input_scale,
                                        weights.w2_packed, weights.w2_scale, weights.w2_input_scale, weights.num_experts,
                                        weights.inter_size)
            if reduce_tp and self.prepare_finalize.parallel_config.tp_size > 1:
                dist.all_reduce(out, group=self.prepare_finalize.parallel_config.tp_group)
            return out
        prepared = self.prepare_finalize.prepare(x, topk_weights, topk_ids)
        local = self.experts.apply(prepared.hidden_states, prepared.topk_ids, prepared.topk_weights, weights,
                                   x_div=prepared.ctx.get("x_div", 1))
        return self.prepare_finalize.finalize(local, prepared, output_shape=(x.shape[0], x.shape[1]),
                                              model_dtype=model_dtype, reduce_tp=reduce_tp)
