"""A bias-free linear layer over one or several stored matrices.

The matrices named in ``sources`` ([out_i, in] each, row-major as stored) are
stacked along the output axis at load, so that projections that read the same
input (q, k, v; gate, up) run as one product.  The reference keeps them apart
and reads them under their stored names
(crates/llm-backend/src/core/qwen/ops/attention_full.rs:586-609).
"""
from __future__ import annotations

from typing import Dict, List, Optional, Sequence, Tuple

import torch

from .base import FusedNormSpec, Part, Runtime, UnscaledNorm, WeightSpec


class Linear(Part):
    capture_safe = True
    kernels_only = True

    def __init__(self, sources: Sequence[Tuple[str, int]], in_features: int, *, side_by_side: bool = False,
                 column_groups: Optional[Tuple[int, int, int]] = None, row_order: Optional[torch.Tensor] = None):
        """``side_by_side``: the sources [out, in_i] share the output axis and are laid next to each other along the
        input axis (``in_features`` is then the common OUTPUT size and the numbers in ``sources`` are input sizes), so
        that one product sums what each matrix makes of its share of the input columns.  ``column_groups`` =
        (groups, used, padded): the input arrives as ``groups`` groups of ``padded`` columns of which the first
        ``used`` are real (heads whose rows are narrower than the cache's); the stored matrix [out, groups * used]
        gets zero columns at load.  ``row_order`` [out_features]: the stacked rows are taken in this order (output column
        j is stored row ``row_order[j]``), for a consumer that wants a projection's columns in another order than the
        stored one."""
        self.row_order = row_order
        self.sources: List[Tuple[str, int]] = list(sources)
        self.side_by_side = side_by_side
        self.column_groups = column_groups
        total = sum(n for _, n in self.sources)
        if side_by_side:
            self.out_features, self.in_features = in_features, total
        else:
            self.out_features, self.in_features = total, in_features
        if row_order is not None and (side_by_side or row_order.numel() != self.out_features):
            raise ValueError(f"a row order of {row_order.numel()} entries does not fit {self.out_features} stacked rows")
        if column_groups is not None:
            groups, used, padded = column_groups
            if side_by_side or groups * used != in_features or padded < used:
                raise ValueError(f"column groups {column_groups} do not fit {in_features} input columns")
            self.in_features = groups * padded
        self.weight: Optional[torch.Tensor] = None

    def weight_specs(self) -> Dict[str, WeightSpec]:
        if self.side_by_side:
            return {name: WeightSpec((self.out_features, n), "linear") for name, n in self.sources}
        stored_in = self.in_features if self.column_groups is None else self.column_groups[0] * self.column_groups[1]
        return {name: WeightSpec((n, stored_in), "linear") for name, n in self.sources}

    def load(self, weights, rt: Runtime) -> None:
        self.rt = rt
        parts = [weights.stored(name).to(device=rt.device, dtype=rt.dtype) for name, _ in self.sources]
        stacked = parts[0].contiguous() if len(parts) == 1 else torch.cat(parts, dim=1 if self.side_by_side else 0).contiguous()
        if self.row_order is not None:
            stacked = stacked[self.row_order.to(stacked.device)].contiguous()
        if self.column_groups is not None and self.column_groups[1] != self.column_groups[2]:
            groups, used, padded = self.column_groups
            wide = torch.zeros((stacked.shape[0], groups, padded), dtype=stacked.dtype, device=stacked.device)
            wide[:, :, :used] = stacked.view(stacked.shape[0], groups, used)
            stacked = wide.view(stacked.shape[0], groups * padded)
        # the tensor-core product streams weights fastest from its own box layout (``ops.TiledWeight``)
        self.weight = rt.ops.tile_weight(stacked) if self.on_tensor_cores() else stacked

    def load_matrix(self, matrix: torch.Tensor, rt: Runtime) -> None:
        """Takes a ready matrix [out_features, in_features] (one that a part worked out from stored tensors) in place
        of stored ones."""
        self.rt = rt
        if tuple(matrix.shape) != (self.out_features, self.in_features):
            raise ValueError(f"matrix {tuple(matrix.shape)} does not fit a layer of {self.out_features} x {self.in_features}")
        matrix = matrix.to(device=rt.device, dtype=rt.dtype).contiguous()
        self.weight = rt.ops.tile_weight(matrix) if self.on_tensor_cores() else matrix

    def forward(self, x, out_dtype: Optional[torch.dtype] = None) -> torch.Tensor:
        if isinstance(x, UnscaledNorm):
            return self.rt.ops.linear_tcgen05(x.rows, self.weight, out_dtype, row_scale=x.row_scale())
        return self.rt.ops.linear(x, self.weight, out_dtype, constant=True)

    # Largest batch for which a norm is folded into the products around it: every batch that the weight-streaming
    # products take.  Measured on the 8B layer sizes (ms a decode step, folded against separate): one request 4 %
    # faster, 24 requests of 2,048 tokens 4.42, 32 requests 4.70 against 4.83, 48 of 1,024 tokens 4.84 against 4.97,
    # 64 of 4,096 tokens 9.51 against 9.54.  (Before the epilogue stored through shared memory it took 2.4 to 3.8 us a
    # product and lost from 17 rows on.)  The many-token kernel's epilogue of this kind is slower than the separate
    # norm kernel, beside which the next product already loads its first weight tiles.
    FUSED_NORM_MAX_ROWS = 64

    def on_tensor_cores(self) -> bool:
        """Whether this layer's products run on the tensor-core kernel, which alone has the fused epilogues."""
        return self.rt.dtype == torch.bfloat16 and self.in_features % 8 == 0

    def fuses_norms(self, rows: int) -> bool:
        """Whether a batch of ``rows`` tokens should have the norms next to this product folded into it."""
        return self.on_tensor_cores() and rows <= self.FUSED_NORM_MAX_ROWS

    def forward_into_norm(self, x: torch.Tensor, resid: torch.Tensor, spec: FusedNormSpec) -> UnscaledNorm:
        """resid += x W^T in place; returns the sum's rows under the norm ``spec`` without their 1 / rms factor."""
        rows, sumsq = self.rt.ops.linear_residual_norm(x, self.weight, resid, spec.weight)
        return UnscaledNorm(rows, sumsq, spec.width, spec.eps)
