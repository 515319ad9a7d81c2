"""Norms over the rows of the residual: RMSNorm, and a weighted layer norm without a shift.

``y = (x * rsqrt(mean(x^2) + eps)) * w`` with float32 statistics
(src/backend/cpu/scalar/quants.c:1489-1512).  The input is the float32
residual; the output has the compute dtype (it feeds a matrix product).

``layernorm``: ``y = (x - mean(x)) * rsqrt(var(x) + eps) * w`` with the variance
taken about the mean (the mean of the squared deviations), float32 statistics,
no bias.
"""
from __future__ import annotations

from typing import Dict, Optional

import torch

from ..ops import kernels as K
from ..ops.linear import NormedRows
from .base import Part, WeightSpec, register_part


class RMSNorm(Part):
    category = "norm"
    graph_safe = True

    def __init__(self, params, env):
        super().__init__(params, env)
        self.size = int(self._p("size"))
        self.eps = float(self._p("eps"))
        self.weight: Optional[torch.Tensor] = None

    def weight_specs(self) -> Dict[str, WeightSpec]:
        return {"weight": WeightSpec((self.size,), "norm")}

    def bind(self, w):
        self.weight = w["weight"].to(torch.float32).contiguous()

    def forward(self, x: torch.Tensor, rows: Optional[torch.Tensor] = None) -> torch.Tensor:
        n = x.shape[0] if rows is None else rows.numel()
        out = torch.empty((n, self.size), dtype=self.env.dtype, device=x.device)
        return K.rmsnorm_rows(x, self.weight, self.eps, out, rows)

    def forward_for(self, part, x: torch.Tensor):
        """The norm as ``part``'s input: in a bfloat16 step of few rows left to the part's first product, if the part's forward is
        marked as one that takes :class:`NormedRows` (a subclass with a forward of its own is not) and the norm is this one (and
        not a subclass's, with a forward of its own)."""
        if (x.shape[0] <= K.ROWS_MAX_M and self.env.dtype == torch.bfloat16 and getattr(part.forward, "takes_normed_rows", False)
                and getattr(self.forward, "__func__", None) is _RMS_FORWARD):
            return NormedRows(x, self.weight, self.eps)
        return self.forward(x)


_RMS_FORWARD = RMSNorm.forward


class LayerNorm(RMSNorm):
    """Same sizes, weight and interface as :class:`RMSNorm`; the rows are centred first."""

    def forward(self, x: torch.Tensor, rows: Optional[torch.Tensor] = None) -> torch.Tensor:
        n = x.shape[0] if rows is None else rows.numel()
        out = torch.empty((n, self.size), dtype=self.env.dtype, device=x.device)
        return K.layernorm_rows(x, self.weight, self.eps, out, rows)


register_part("norm", "rmsnorm", RMSNorm)
register_part("norm", "layernorm", LayerNorm)
