"""Grouped (mixture-of-experts) packed-weight matmul and the fused gate/up pair: Python surface of
``torch_ggml_ops::grouped_mmq`` and ``torch_ggml_ops::grouped_mmq_pair``.

Same contract as the reference (torch_ggml_ops/grouped_mmq.py:4-250).  Rows are pre-sorted by
expert; ``expert_indices`` (int64) names the expert of each group and ``expert_offsets`` (int32)
the cumulative end row of each group; both stay on the device.  Backward of the pair has three
cases: both cotangents present -> one fused ``grouped_mmq_pair_grad_input`` (the two Jacobian
products are summed in fp32 before one bf16 rounding); only one present -> the single-projection
``grouped_mmq_grad_input`` with that projection's weight (``csrc/torch_ext.cpp``).
"""
import torch

from .mmq import _NS


def _rows_by(like: torch.Tensor, width: int) -> torch.Tensor:
    return like.new_empty((like.shape[0], width))


@torch.library.register_fake(f"{_NS}::grouped_mmq")
def _(input, packed_weight, expert_indices, expert_offsets, quant_type, out_features):
    return _rows_by(input, out_features)


@torch.library.register_fake(f"{_NS}::grouped_mmq_grad_input")
def _(grad_output, packed_weight, expert_indices, expert_offsets, quant_type, in_features):
    return _rows_by(grad_output, in_features)


@torch.library.register_fake(f"{_NS}::grouped_mmq_pair")
def _(input, first_packed_weight, second_packed_weight, expert_indices, expert_offsets, quant_type, out_features):
    return _rows_by(input, out_features), _rows_by(input, out_features)


@torch.library.register_fake(f"{_NS}::grouped_mmq_pair_grad_input")
def _(first_grad_output, second_grad_output, first_packed_weight, second_packed_weight, expert_indices,
      expert_offsets, quant_type, in_features):
    return _rows_by(first_grad_output, in_features)


def grouped_mmq(input, packed_weight, expert_indices, expert_offsets, quant_type: int, out_features: int):
    """Per-group ``input[rows_g] @ W[expert_g].T`` over expert-sorted bf16 rows."""
    return torch.ops.torch_ggml_ops.grouped_mmq.default(
        input, packed_weight, expert_indices, expert_offsets, int(quant_type), int(out_features))


def grouped_mmq_pair(input, first_packed_weight, second_packed_weight, expert_indices, expert_offsets,
                     quant_type: int, out_features: int):
    """Gate and up projections of the same rows in one launch: ``(x @ W1[e].T, x @ W2[e].T)``."""
    return torch.ops.torch_ggml_ops.grouped_mmq_pair.default(
        input, first_packed_weight, second_packed_weight, expert_indices, expert_offsets,
        int(quant_type), int(out_features))


__all__ = ["grouped_mmq", "grouped_mmq_pair"]
