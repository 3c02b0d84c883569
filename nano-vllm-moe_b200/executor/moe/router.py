"""Softmax top-k router (reference: executor/moe/router.py:9-34), on the CUDA router kernel."""
from __future__ import annotations

from abc import ABC, abstractmethod

import torch

from ... import _lib


class MoERouter(ABC):
    @abstractmethod
    def select_experts(self, hidden_states: torch.Tensor, router_logits: torch.Tensor) -> tuple[torch.Tensor, torch.Tensor]:
        ...


class SoftmaxTopKRouter(MoERouter):
    def __init__(self, top_k: int, renormalize: bool) -> None:
        self.top_k = top_k
        self.renormalize = renormalize

    def select_experts(self, hidden_states, router_logits):
        """-> (weights float32 [T, k], expert ids int64 [T, k]); softmax in fp32 over all experts, then top-k."""
        del hidden_states
        return _lib.host().moe_route(router_logits, self.top_k, self.renormalize)
