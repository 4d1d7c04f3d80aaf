"""Rows of the residual stream whose RMSNorm is still to be applied, and the forms in which the contraction kernels take them."""
from __future__ import annotations

from typing import Optional, Union

import torch

from .. import kernels


class NormedRows:
    """RMSNorm(x) * weight that is computed when somebody needs it as a tensor."""

    def __init__(self, x: torch.Tensor, weight: torch.Tensor, eps: float, dtype: torch.dtype,
                 scaled: Optional["kernels.NormEmit"] = None):
        self.x, self.weight, self.eps, self.dtype = x, weight, eps, dtype
        self.scaled = scaled          # what the kernel that summed x wrote for this norm, if it did
        self._tensor: Optional[torch.Tensor] = None

    @property
    def shape(self):
        return self.x.shape

    def tensor(self) -> torch.Tensor:
        if self._tensor is None:
            self._tensor = kernels.rmsnorm(self.x, self.weight, self.eps, self.dtype)
        return self._tensor

    def kernel_input(self) -> "kernels.NormInput":
        return kernels.NormInput(self.x, self.weight, self.eps)


def as_tensor(a: Union[torch.Tensor, NormedRows]) -> torch.Tensor:
    return a.tensor() if isinstance(a, NormedRows) else a


def scaled_or_tensor(a: Union[torch.Tensor, NormedRows]):
    """For a kernel that takes a `kernels.ScaledInput`: that, if the rows came prepared and nobody
    has asked for the normalised tensor yet; else the tensor."""
    if isinstance(a, NormedRows) and a.scaled is not None and a._tensor is None and a.dtype == torch.bfloat16:
        return kernels.ScaledInput(a.scaled.xw, a.scaled.ssq, a.eps)
    return as_tensor(a)


# A block that applies the norm itself reads all M rows again, so fusing the norm pays only while
# few blocks do so (about one per SM) or the rows are very few; measured on the LFM2-1.2B shapes:
# fused 12.5 us against 14.5 us for the short convolution's in_proj (128 blocks, 8 rows), but
# 75 us against 50 us for the head (2048 blocks).  A whole step with every norm fused against the
# rule below: 0.673 against 0.680 ms at 4 rows, 0.723 against 0.714 ms at 8 rows.
NORM_FUSION_MAX_BLOCKS = 160
NORM_FUSION_ANY_BLOCKS_ROWS = 4


def fused_input(a: Union[torch.Tensor, NormedRows], w: torch.Tensor, need_fused_rows: bool = False,
                blocks: Optional[int] = None):
    """What a skinny kernel should be given for `a`, or None if it does not take it: the pending
    norm itself when the kernel can apply it and that is the faster way (`blocks` = thread blocks
    the kernel will run, default one per 16 weight rows), else the (materialised) bfloat16 tensor."""
    takes = kernels.gemm_skinny_fused_takes if need_fused_rows else kernels.gemm_skinny_takes
    if isinstance(a, NormedRows):
        if a.dtype != torch.bfloat16:
            return None
        if a._tensor is None:
            if a.scaled is not None:
                si = kernels.ScaledInput(a.scaled.xw, a.scaled.ssq, a.eps)
                if takes(si, w):
                    return si
            ki = a.kernel_input()
            n_blocks = blocks if blocks is not None else -(-w.shape[0] // 16)
            worth = n_blocks <= NORM_FUSION_MAX_BLOCKS or a.shape[0] <= NORM_FUSION_ANY_BLOCKS_ROWS
            if worth and takes(ki, w):
                return ki
            max_rows = kernels.gemm_skinny_fused_max_m() if need_fused_rows else kernels.gemm_skinny_max_m()
            if a.shape[0] > max_rows:
                return None             # too many rows for these kernels: the norm stays pending for another
        a = a.tensor()
    return a if takes(a, w) else None
