"""A matrix product ``y = x W^T (+ b)`` with ``W`` stored ``[out, in]``.

The reference issues one cuBLAS call per projection with float32 accumulation
(runtime/backends/cuda/native/cublas_gemm.cpp:84-102, ``C[M,N] = A[M,K] *
B[N,K]^T``).  Here a float32 weight goes through the products of the 32-bit
path (gemm_f32.cu, gemm_f32_umma.cu); a bfloat16 weight goes through the library (cuBLAS via ``torch.mm``) for
many rows, through the weight-streaming kernel (gemv_bf16.cu) for up to 8
rows, and through the tcgen05 kernel with the operands' places changed
(gemm_umma.cu) for 9 to 128 rows where the consumer adds partial sums and K is
long or the host launches the step, and for a vocabulary's float32 logits.
This is not a registered part: mixers and feed-forwards own their Linears.
"""
from __future__ import annotations

from typing import Optional

import torch

from ..kernels import ops
from .base import PartialSums


GEMV_ROWS = 8     # up to this many rows go to the weight-streaming kernel (it matches the library there)
# From 9 to 128 rows a product is still bound by reading W once: the tcgen05 kernel with the weights as the tiles' rows.  It
# leaves float32 partial sums, so it serves consumers that add such up.  Product and consumer together, us, kernel / library:
# with a long K (down) 3B sizes 15 to 17 / 18 to 23, 7B 28 to 33 / 31 to 37, 14B 30 to 37 / 30 to 38 (a tenth behind at 128 rows);
# with a short K it is behind everywhere: q, k, v 3B 8.5 at 9 rows to 11.0 at 128 / 7.8 to 8.2, 7B 13.9 to 14.6 / 10.5 to 11.5,
# 14B 18.9 to 21.6 / 16.4 to 19.0; o 3B 7.5 to 10.1 / 7.4 to 8.0, 7B 10.5 to 14.9 / 10.2 to 11.5, 14B 18.4 to 19.7 / 14.8 to 17.7.
# But a launch of the library costs the host more, and a step that the host launches waits for its launches: prompts of 12 to
# 128 tokens and steps of 28 to 121 rows with prompts among them take 0.86 to 0.91 of the time at the 3B sizes, 0.88 to 0.96 at
# the 7B, 0.89 to 1.03 at the 14B ones (6 layers; above 1 where 40 rows and more of the larger sizes keep the GPU behind).  So short
# K goes to the kernel in such steps only; a captured step of 64 single tokens (7B sizes, 6 layers) took 1,210 us with it, 1,158 without.
FEW_ROWS, FEW_ROWS_MIN_K = 128, 8192
# A vocabulary's float32 logits for 9 to 128 rows: the same kernel with K in one piece (152,064 x 3,584: 23 rows 164 us against
# the library's 180, 64 rows 172 / 188, 128 rows 192 / 212; 151,936 x 2,048: 99 / 105 and 114 / 127; 152,064 x 5,120: 236 / 260
# and 271 / 288).  At 32,768 columns the two are level, below the library is ahead (14,336: 21.7 / 20.1 at 64 rows).
WIDE_COLUMNS = 65536


def stack_rows(mats) -> torch.Tensor:
    """The matrices below one another, zero rows behind them up to a multiple of eight.  The library takes a product with
    any other number of columns through a kernel of an older kind (2,048 rows, K 3,584: 4,636 columns 221 us, 4,640 48 us)."""
    fill = -sum(m.shape[0] for m in mats) % 8
    return torch.cat([*mats, mats[0].new_zeros((fill, mats[0].shape[1]))] if fill else list(mats), dim=0)


class Linear:
    def __init__(self, weight: torch.Tensor, bias: Optional[torch.Tensor] = None):
        if weight.dim() != 2:
            raise ValueError("Linear wants a [out, in] matrix")
        self.weight = weight.contiguous()
        self.out_features, self.in_features = weight.shape
        self.bias = None if bias is None else bias.to(torch.float32).contiguous()

    def forward(self, x: torch.Tensor, out_dtype: Optional[torch.dtype] = None, allow_partials: bool = False,
                f32_sums: bool = False, launched: bool = False):
        """x [M, in] -> [M, out] in ``out_dtype`` (default: x's type).  With
        ``allow_partials`` the result may be a :class:`PartialSums` (the
        weight-streaming kernel cuts K between blocks when a matrix has too few
        rows to fill the GPU).  With ``f32_sums`` on top of that, a bfloat16
        product always comes as float32 sums (one slice from the library): for
        a consumer that computes on with the sums, to which a rounding to
        bfloat16 in between would only add error.  ``launched``: the step's launches are the host's, not a graph's, so that
        9 to 128 rows against a short K go to the kernel that is the cheaper one to launch."""
        m = x.shape[0]
        out_dtype = out_dtype or x.dtype
        w = self.weight
        if w.dtype == torch.float32:
            # 32-bit weights: true float32 product whatever the activations are
            if x.dtype != torch.float32:
                x = ops.convert(x.contiguous(), torch.empty(x.shape, dtype=torch.float32, device=x.device))
            y = torch.empty((m, self.out_features), dtype=torch.float32, device=x.device)
            ops.gemm_f32(x, w, self.bias, y, w_fixed=True)
            if out_dtype != torch.float32:
                y = ops.convert(y, torch.empty(y.shape, dtype=out_dtype, device=x.device))
            return y
        if x.dtype != torch.bfloat16:
            raise ops.KernelError(f"Linear: bfloat16 weights need bfloat16 activations, got {x.dtype}")
        if m <= GEMV_ROWS and self.in_features % 8 == 0:
            # a few rows: bound by reading the weights once -> the weight-streaming kernel
            splits = self._k_splits() if allow_partials else 1
            if splits > 1:
                y = torch.empty((splits, m, self.out_features), dtype=torch.float32, device=x.device)
                return PartialSums(ops.gemv_bf16(x, w, self.bias, y, k_splits=splits))
            if allow_partials and f32_sums:
                y = torch.empty((m, self.out_features), dtype=torch.float32, device=x.device)
                return PartialSums(ops.gemv_bf16(x, w, self.bias, y).unsqueeze(0))
            y = torch.empty((m, self.out_features), dtype=out_dtype, device=x.device)
            return ops.gemv_bf16(x, w, self.bias, y)
        if (allow_partials and self.bias is None and m <= FEW_ROWS and (launched or self.in_features >= FEW_ROWS_MIN_K)
                and self.in_features % 8 == 0 and x.stride(1) == 1 and x.stride(0) % 8 == 0
                and not (x.data_ptr() | w.data_ptr()) & 15):                    # (the library takes any)
            parts = ops.gemm_umma_skinny_parts(self.out_features, self.in_features, m)
            y = torch.empty((parts, m, self.out_features), dtype=torch.float32, device=x.device)
            return PartialSums(ops.gemm_umma_skinny(x, w, y, True))
        if (out_dtype == torch.float32 and self.bias is None and m <= FEW_ROWS and self.out_features >= WIDE_COLUMNS
                and self.in_features % 8 == 0 and x.stride(1) == 1 and x.stride(0) % 8 == 0
                and not (x.data_ptr() | w.data_ptr()) & 15):
            y = torch.empty((1, m, self.out_features), dtype=torch.float32, device=x.device)
            y = ops.gemm_umma_skinny(x, w, y, True)
            return PartialSums(y) if allow_partials and f32_sums else y[0]
        if allow_partials and f32_sums and self.bias is None:
            return PartialSums(ops.matmul_library(x, w, torch.float32).unsqueeze(0))
        y = ops.matmul_library(x, w, torch.float32 if (out_dtype == torch.float32 or self.bias is not None)
                               else torch.bfloat16)
        if self.bias is not None:
            y += self.bias
        return y if y.dtype == out_dtype else y.to(out_dtype)

    def _k_splits(self) -> int:
        """Into how many parts the weight-streaming kernel cuts K (it knows its
        block shapes and how many blocks the GPU holds; the number depends on
        the matrix only, never on the batch)."""
        return ops.gemv_k_splits(self.out_features, self.in_features)
