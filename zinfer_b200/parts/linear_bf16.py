"""Tensor-core contractions of the bfloat16 path.  `try_linear` returns None for a shape no
tensor-core kernel takes; the caller then uses the CUDA-core kernel.

Few rows (single-token steps): the weight-streaming mma.sync kernel, which can also apply a
pending RMSNorm itself.  More rows (prompt steps): the TMA-fed tcgen05 kernel with its
accumulator in tensor memory."""
from __future__ import annotations

from .. import kernels
from .rows import as_tensor, fused_input, scaled_or_tensor


# From 17 to 64 rows the tcgen05 kernel with the weights on its 128-row side beats the mma.sync
# kernel (measured at 64 rows on the LFM2-1.2B shapes: 17 us against 44 us for N = 16384, 10 against
# 22 for N = 6144, 7 against 12 for N = 2048, 12 against 38 for N = 2048 with K = 8192).  Up to 16
# rows the mma.sync kernel needs no cluster and applies pending norms itself.  Whole steps of 9 / 12 / 16 sequences at
# 500 tokens, ms, mma.sync against tcgen05 (the short convolution fused in both): the 350M shape 0.43 / 0.47 / 0.49 against
# 0.54 / 0.56 / 0.57; LFM2-1.2B 0.72 / 0.76 / 0.80 against 0.83 / 0.86 / 0.86; the 2.6B shape 1.51 / 1.59 / 1.66 against
# 1.58 / 1.61 / 1.64.
TC_SWAPPED_MIN_ROWS = 17


def swapped_splits(n_weight_rows: int, sm_count: int) -> int:
    """In how many parts K is cut (one per block of a cluster): the fewest that give 7 of 10 SMs a block.
    Two blocks fit an SM: up to one per SM, the blocks of the next kernel all find a place and request their first
    weights while this one runs; a second round of parts takes those places and adds partial sums to exchange.
    Fewer blocks than that leave too few loads under way.  Whole single-token steps (ms) with parts until 0.6 / 0.7 /
    1.0 x SMs: LFM2-1.2B with 64 rows 1.21 / 1.16 / 1.19, 32 rows 1.01 / 0.97 / 0.99; the 350M shape with 64 rows
    0.87 / 0.85 / 0.92, 24 rows 0.62 / 0.60 / 0.65; the 2.6B shape with 24 rows 1.88 / 1.80 / 1.80."""
    tiles = -(-n_weight_rows // 128)
    s = 1
    while s < 8 and 10 * tiles * s < 7 * sm_count:
        s *= 2
    return s


def try_linear(a, w, out, out_dtype, accumulate, bias, sink=None):
    if TC_SWAPPED_MIN_ROWS <= a.shape[0] <= kernels.gemm_skinny_max_m():
        t = scaled_or_tensor(a)
        if not kernels.gemm_tc_takes(t, w, out):
            t = as_tensor(a)
        if kernels.gemm_tc_takes(t, w, out):
            emit = None
            if sink is not None and kernels.gemm_tc_emits(t, out):
                emit = kernels.NormEmit(sink.norm_weight)
            y = kernels.gemm_tc(t, w, out=out, out_dtype=out_dtype, accumulate=accumulate, bias=bias,
                                splits=swapped_splits(w.shape[0], kernels.sm_count(w.device)), emit=emit)
            if emit is not None:
                sink.emit = emit
            return y
    x = fused_input(a, w)
    if x is not None:
        emit = None
        if sink is not None and kernels.gemm_skinny_emits(x, out):
            emit = kernels.NormEmit(sink.norm_weight)
        y = kernels.gemm_skinny(x, w, out=out, out_dtype=out_dtype, accumulate=accumulate, bias=bias, emit=emit, _taken=True)
        if emit is not None:
            sink.emit = emit
        return y
    a = as_tensor(a)
    if kernels.gemm_tc_takes(a, w, out):
        return kernels.gemm_tc(a, w, out=out, out_dtype=out_dtype, accumulate=accumulate, bias=bias)
    return None
