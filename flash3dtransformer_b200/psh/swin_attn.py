"""Output buffers of the bucketed attention operators (reference: flash3dxfmr/psh/swin_attn.py:13-43)."""
from __future__ import annotations

from dataclasses import dataclass

import torch

from . import plan as f3dplan


def lse_rows(b: int, l: int, h: int, device) -> torch.Tensor:
    """Log-sum-exp rows that nobody reads: inside plan.level_buffers() one buffer per shape."""
    return f3dplan.pooled(("lse", b, l, h, str(device)), lambda: torch.empty(b, l, h, dtype=torch.float32, device=device))


@dataclass(slots=True)
class BuckSwinFwdBuffers:
    O: torch.Tensor
    LSE: torch.Tensor

    @staticmethod
    def create_buckswin_fwd_buff(Q: torch.Tensor):
        b, l, h, _ = Q.shape
        if f3dplan.enabled():
            return BuckSwinFwdBuffers(torch.empty_like(Q), lse_rows(b, l, h, Q.device))
        return BuckSwinFwdBuffers(torch.empty_like(Q), torch.zeros(b, l, h, dtype=torch.float32, device=Q.device))


@dataclass(slots=True)
class BuckSwinBwdBuffers:
    O: torch.Tensor
    dQ: torch.Tensor
    dK: torch.Tensor
    dV: torch.Tensor
    Scope_buckets: torch.Tensor
    Delta: torch.Tensor
    buck_size: int

    @staticmethod
    def create_buckswin_buffers(O: torch.Tensor, Scope_buckets: torch.Tensor, buck_size: int, fill: bool = True):
        """`fill` False leaves the buffers as allocated: the backward writes Delta and dQ whole, dK and dV for the tokens of
        listed buckets."""
        b, l, h, _ = O.shape
        if not fill:
            return BuckSwinBwdBuffers(O, torch.empty_like(O), torch.empty_like(O), torch.empty_like(O), Scope_buckets,
                                      torch.empty(b, l, h, dtype=torch.float32, device=O.device), buck_size)
        return BuckSwinBwdBuffers(O, torch.zeros_like(O), torch.zeros_like(O), torch.zeros_like(O), Scope_buckets,
                                  torch.zeros(b, l, h, dtype=torch.float32, device=O.device), buck_size)
