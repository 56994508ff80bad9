"""x @ W^T for a weight ``[out, in]`` (the reference's one path from a weight
name to a matmul, crates/models/qwen/src/forward/projection.rs:257-265).

float32 runs on the hand-written CUDA-core kernel (true 32-bit, fixed order),
or, for large products of a prompt's rows, on the tensor cores in three
bfloat16 parts a number (``Runtime.ordered_sums``).
bfloat16 runs on the hand-written tcgen05 kernel where its shape rules hold,
else on the library product (the reference itself calls a library matmul
here), or on the plain CUDA-core kernel when asked.
"""
from __future__ import annotations

from typing import Optional, Sequence

import torch

from .. import ops
from .registry import Runtime


class Linear:
    def __init__(self, weight: torch.Tensor, runtime: Runtime):
        if weight.dim() != 2:
            raise ValueError(f"a linear weight must be [out, in], got {tuple(weight.shape)}")
        self.weight = weight.to(device=runtime.device, dtype=runtime.dtype).contiguous()
        self.out_features, self.in_features = self.weight.shape
        self.dtype = runtime.dtype
        self.backend = runtime.gemm_backend
        self.runtime = runtime   # a part that is built later may change what it says of sums, a step what it says of rows

    @classmethod
    def stacked(cls, weights: Sequence[torch.Tensor], runtime: Runtime) -> "Linear":
        """Several weights over the same input, rows one after another, so
        that one product yields all their outputs side by side."""
        return cls(torch.cat([w.to(runtime.device) for w in weights], dim=0), runtime)

    def forward(self, x: torch.Tensor, out_dtype: Optional[torch.dtype] = None,
                out: Optional[torch.Tensor] = None) -> torch.Tensor:
        out_dtype = out_dtype or self.dtype
        if self.dtype == torch.float32:
            return self._float32(x, out)
        return ops.gemm_bf16(x, self.weight, out_dtype=out_dtype, backend=self.backend, out=out)

    def _float32(self, x: torch.Tensor, out: Optional[torch.Tensor]) -> torch.Tensor:
        """Single tokens in ascending order; rows of portions, where large enough matrices make that faster, on the tensor
        cores. Both give a row the same bits whatever other rows come with it, so a request's do not depend on what else a
        step holds, nor on how its prompt was cut into portions of several tokens."""
        runs = self.runtime.runs
        if runs is None or runs[-1][1] != x.shape[0] or self.backend != "auto" or not ops.gemm_float_takes(x, self.weight):
            return ops.gemm_simple(x, self.weight, out_dtype=torch.float32, out=out)
        if out is None:
            out = torch.empty((x.shape[0], self.out_features), dtype=torch.float32, device=x.device)
        for begin, end, several in runs:
            (ops.gemm_float if several else ops.gemm_simple)(x[begin:end], self.weight, out=out[begin:end])
        return out

    def rows_are_short(self) -> bool:
        """Whether this is a weight of the kind whose decode-step products are
        short, overlapped kernels (rows of at most ``ops.STREAM_K`` values, the
        kernel chosen by this library), where a hand-over between kernels costs
        as much as the work."""
        return self.dtype == torch.bfloat16 and self.backend == "auto" and self.in_features <= ops.STREAM_K

    def weight_bytes(self) -> int:
        return self.weight.numel() * self.weight.element_size()


def stacked_rows(matrices: Sequence[torch.Tensor], runtime: Runtime, multiple: int = 8) -> Linear:
    """One product over the same input, with rows of zeros at the end so that a
    row of the result starts on the boundary that vector accesses need."""
    rows = sum(m.shape[0] for m in matrices)
    extra = -rows % multiple
    if extra:
        matrices = list(matrices) + [torch.zeros((extra, matrices[0].shape[1]), dtype=matrices[0].dtype,
                                                 device=matrices[0].device)]
    return Linear.stacked(matrices, runtime)
