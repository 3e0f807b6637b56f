"""y = x W^T (+ b) with W stored [out, in], as the reference's linears
(src/paged/qwen3.rs:120-132, 226-239).

The one place where a matrix product is chosen:
  float32   the engine's own kernels, true 32-bit: multiply-adds on the CUDA cores, or the
            tensor cores with every operand in three bfloat16 parts (24 bits, no less exact);
            N and K say which, and every output element is summed over k in an order that K alone
            fixes, so a row's result does not depend on the rows beside it.
  bfloat16  the tensor-core product (see `matmul`).
"""
from __future__ import annotations

from typing import Optional

import torch

from ..csrc import ops


def matmul(x: torch.Tensor, weight: torch.Tensor, bias: Optional[torch.Tensor] = None,
           out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
    """`weight` belongs to a model: nothing that a kernel of the step writes (the products may fetch it ahead of earlier kernels)."""
    out_dtype = out_dtype or x.dtype
    if x.dtype == torch.float32:
        return ops.gemm_nt_simt(x, weight, bias, out_dtype, w_ready=True)
    return ops.gemm_bf16(x, weight, bias, out_dtype, w_ready=True)


class Linear:
    """A weight [out, in] and an optional float32 bias, already on the device."""

    def __init__(self, weight: torch.Tensor, bias: Optional[torch.Tensor] = None):
        self.weight, self.bias = weight, bias

    def __call__(self, x: torch.Tensor, out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
        return matmul(x, self.weight, self.bias, out_dtype)
