"""Calibration of channel orders and residual widths from activations, on whatever device they live on.

The reference derives both from forward passes over a calibration set: the per-channel maximum of
|x| at the input of every projection (``get_act_stats`` with the max metric, utilize.py:80-116 of
ARCQuant, running maximum over the samples), the channel order = ascending argsort of that statistic
(reorder_indices.py), and the number of residual channels from the share of elements that exceed an
eighth of their row's maximum, rounded up to a multiple of 64 (``search_select_proportions``,
utilize.py:546-551).  The same rules here, as three small functions that a caller hooks onto the
inputs of its linears; the results feed `llama_layer.PackedLinear` / `checkpoint`.
"""
from __future__ import annotations

import math

import torch

from . import ops


class ChannelAbsMax:
    """Running per-channel max |x| over any number of batches [..., channels], and with it the running
    count behind the residual-width rule.  bf16 batches on a CUDA device take one pass of
    `arcq_calib_stats_bf16` (both statistics at once, accumulated on the device); anything else takes the
    eager torch formulation."""

    def __init__(self):
        self.value: torch.Tensor | None = None
        self._above: torch.Tensor | None = None      # elements larger than an eighth of their row's maximum
        self._seen = 0                               # elements seen

    def update(self, x: torch.Tensor) -> None:
        k = x.shape[-1]
        native = x.is_cuda and x.dtype == torch.bfloat16 and k % 8 == 0 and k <= 32768
        if native and not x.is_contiguous():
            x = x.detach().reshape(-1, k)
            native = x.is_contiguous()
        if native:
            if self.value is None and self._above is None:      # (one allocation: one launch that clears it)
                both = torch.zeros(k + 2, dtype=torch.float32, device=x.device)
                self.value, self._above = both[:k], both[k:].view(torch.int64).reshape(())
            if self.value is None:                   # (a caller has taken the maxima away)
                self.value = torch.zeros(k, dtype=torch.float32, device=x.device)
            if self._above is None:                  # (a caller has put maxima here)
                self._above = torch.zeros((), dtype=torch.int64, device=x.device)
            ops.calib_stats(x, self.value, self._above)
            self._seen += x.numel()
        else:
            self._update_eager(x.detach().reshape(-1, k))

    @torch.no_grad()
    def _update_eager(self, x2: torch.Tensor) -> None:
        cur = x2.abs().amax(dim=0).float()
        self.value = cur if self.value is None else torch.maximum(self.value, cur.to(self.value.device))
        thr = x2.max(dim=-1, keepdim=True)[0] * 0.125
        n = (x2 > thr).sum().to(torch.int64)
        self._above = n if self._above is None else self._above + n.to(self._above.device)
        self._seen += x2.numel()

    def reorder_index(self) -> torch.Tensor:
        """int16 [channels]: channels by ascending statistic - the largest (critical) channels last."""
        if self.value is None:
            raise RuntimeError("no batch seen")
        if self.value.numel() > 32752:
            raise ValueError("more channels than an int16 order can hold")
        # (its work grows with the square of the width, us against torch's sort: 4096 8.6 / 45.7, 8192 16 / 63, 14 336 50 / 62,
        # 28 672 167 / 67)
        if (self.value.is_cuda and self.value.dtype == torch.float32 and self.value.dim() == 1 and self.value.is_contiguous()
                and 0 < self.value.numel() <= 14336):
            return ops.channel_order(self.value)
        return torch.argsort(self.value).to(torch.int16)

    def select_num(self, granule: int = 64) -> int:
        """The residual width the rule of `select_num_rule` gives for everything seen so far."""
        if self.value is None:
            raise RuntimeError("no batch seen")
        k = self.value.numel()
        ratio = float(self._above) / self._seen
        return min(math.ceil(k * ratio / granule) * granule, k)


@torch.no_grad()
def select_num_rule(x: torch.Tensor, reorder_index: torch.Tensor | None = None, granule: int = 64) -> int:
    """Residual channels for activations x [..., channels]: the share of elements larger than an eighth
    of their row's (signed) maximum decides how many channels get a residual, in units of `granule`.
    The statistic does not depend on the channel order; `reorder_index` is accepted for symmetry with
    the reference, which applies it first."""
    keys = x.detach().reshape(-1, x.shape[-1])
    if reorder_index is not None:
        keys = keys[:, reorder_index.to(keys.device).long()]
    in_features = keys.shape[1]
    threshold = keys.max(dim=-1, keepdim=True)[0] * 0.125
    ratio = float((keys > threshold).sum()) / keys.numel()
    select_num = math.ceil(in_features * ratio / granule) * granule
    return min(select_num, in_features)


def average_bits(in_features: int, select_num: int) -> float:
    """4.5 bits per stored element (e2m1 + a ue4m3 scale per 16) over the augmented width."""
    return 4.5 * (in_features + select_num) / in_features
