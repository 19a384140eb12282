"""Dense packed-weight matmul: Python surface of ``torch_ggml_ops::mmq``.

Same contract as the reference (torch_ggml_ops/mmq.py:4-80): a fake (meta) kernel per operator so
the ops trace under ``torch.compile``; an autograd formula for ``mmq`` that saves only the packed
weight and calls ``mmq_grad_input`` on a contiguous cotangent; and a guard that makes second-order
differentiation of ``mmq_grad_input`` an error (both in ``csrc/torch_ext.cpp``).  The packed weight
never receives a gradient.
"""
import torch

_NS = "torch_ggml_ops"


def _swap_last_dim(like: torch.Tensor, width: int) -> torch.Tensor:
    return like.new_empty((*like.shape[:-1], width))


@torch.library.register_fake(f"{_NS}::mmq")
def _(input, packed_weight, quant_type, out_features):
    return _swap_last_dim(input, out_features)


@torch.library.register_fake(f"{_NS}::mmq_grad_input")
def _(grad_output, packed_weight, quant_type, in_features):
    return _swap_last_dim(grad_output, in_features)


def mmq(input: torch.Tensor, packed_weight: torch.Tensor, quant_type: int, out_features: int) -> torch.Tensor:
    """``input[..., K] @ W[N, K].T`` with ``W`` given as raw GGUF super-blocks (uint8).

    bf16 in, bf16 out; ``quant_type`` is the GGML type id (IQ2_S, Q3_K, Q4_K, Q5_K, Q6_K)."""
    return torch.ops.torch_ggml_ops.mmq.default(input, packed_weight, int(quant_type), int(out_features))


__all__ = ["mmq"]
