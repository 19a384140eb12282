"""Operators either side of the reference's surface (they have no reference schema, so they are
registered under this package's own namespace ``torch_ggml_ops_b200::``):

* ``mmq_multi``: several dense projections of one activation tensor in one call (the reference's
  own "remaining work" for the dense forward, docs/mmq_fwd_optimization.md:299-307);
* ``swiglu``: ``silu(gate) * up``, the step a caller runs between ``grouped_mmq_pair`` and the down
  projection (README.md:3 leaves it to the caller);
* ``moe_mlp``: the single-GPU MoE feed-forward block built from the grouped operators;
* ``lm_head_loss``: the chunked LM-head loop (forward -> cross entropy -> input gradient over
  chunks of rows) that the reference's other production consumer runs
  (docs/mmq_bwd_optimization.md:502-524), which never materialises the full logits.

Everything here calls the same native kernels as the six reference operators; nothing has a CPU or
eager fallback.  The operators and their autograd formulas are registered in ``csrc/torch_ext.cpp``.
"""
from __future__ import annotations

import torch

_NS = "torch_ggml_ops_b200"
_ops = torch.ops.torch_ggml_ops_b200


@torch.library.register_fake(f"{_NS}::mmq_multi")
def _(input, packed_weights, quant_type, out_features):
    return [input.new_empty((*input.shape[:-1], out_features)) for _ in packed_weights]


@torch.library.register_fake(f"{_NS}::swiglu")
def _(gate, up):
    return torch.empty_like(gate)


@torch.library.register_fake(f"{_NS}::swiglu_grad")
def _(grad, gate, up):
    return torch.empty_like(gate), torch.empty_like(gate)


@torch.library.register_fake(f"{_NS}::lm_head_loss")
def _(hidden, packed_weight, quant_type, vocab, targets, chunk_rows, grad_scale):
    return hidden.new_empty((), dtype=torch.float32), torch.empty_like(hidden)


@torch.library.register_fake(f"{_NS}::lm_head_loss_f32")   # with the gradient before its rounding, for autograd
def _(hidden, packed_weight, quant_type, vocab, targets, chunk_rows, grad_scale):
    return hidden.new_empty((), dtype=torch.float32), torch.empty_like(hidden), hidden.new_empty(hidden.shape, dtype=torch.float32)


def mmq_multi(input: torch.Tensor, packed_weights, quant_type: int, out_features: int):
    """``[input @ W_i.T for W_i in packed_weights]`` (1 to 4 weights of one quant type and shape
    [out_features, in_features]) with two weight sets per kernel launch (few tokens: all of them); every
    result is bit-identical to ``mmq`` on that weight alone."""
    return tuple(_ops.mmq_multi.default(input, list(packed_weights), int(quant_type), int(out_features)))


def swiglu(gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    """``silu(gate) * up`` on bf16 tensors (fp32 arithmetic, one rounding), differentiable."""
    return _ops.swiglu.default(gate, up)


def moe_mlp(input, gate_weight, up_weight, down_weight, expert_indices, expert_offsets, quant_type_gate_up: int,
            quant_type_down: int, ffn_features: int):
    """MoE feed-forward block over expert-sorted rows on one GPU:
    ``grouped_mmq(swiglu(*grouped_mmq_pair(x, Wg, Wu)), Wd)``; differentiable with respect to ``input``.
    ``gate_weight`` / ``up_weight``: [E, ffn, row bytes]; ``down_weight``: [E, hidden, row bytes]."""
    from .grouped_mmq import grouped_mmq, grouped_mmq_pair

    gate, up = grouped_mmq_pair(input, gate_weight, up_weight, expert_indices, expert_offsets, quant_type_gate_up, ffn_features)
    return grouped_mmq(swiglu(gate, up), down_weight, expert_indices, expert_offsets, quant_type_down, input.shape[-1])


def lm_head_loss(hidden: torch.Tensor, packed_weight: torch.Tensor, quant_type: int, vocab: int, targets: torch.Tensor,
                 chunk_rows: int = 256, grad_scale: float = 1.0):
    """Sum of the token cross entropies of ``softmax(hidden @ W.T)`` against ``targets`` and its
    gradient with respect to ``hidden``, computed over chunks of ``chunk_rows`` rows so that only
    one chunk of logits ([chunk_rows, vocab], bf16) exists at a time.  Per chunk: forward product
    (bf16 logits) -> fp32 log-softmax and loss, cotangent ``(softmax - onehot) * grad_scale`` in
    bf16 over the logits -> input gradient.  Returns ``(loss_sum fp32 scalar tensor, d_hidden bf16
    like hidden)``.

    The loss is differentiable with respect to ``hidden``, once; the returned gradient is not.

    The reference's production consumer runs this loop with chunk_rows = 256 for a Q6_K head of
    248320 x 2048 (docs/mmq_bwd_optimization.md:502-524); rows = hidden.numel() / K."""
    if chunk_rows < 1:
        raise ValueError(f"chunk_rows must be positive; got {chunk_rows}")
    h2 = hidden.reshape(-1, hidden.shape[-1])
    t1 = targets.reshape(-1)
    if t1.numel() != h2.shape[0]:
        raise ValueError("targets must have one entry per row of hidden")
    if h2.shape[0] == 0:
        return torch.zeros((), dtype=torch.float32, device=hidden.device), torch.empty_like(h2).reshape(hidden.shape)
    loss, d_hidden = _ops.lm_head_loss.default(h2, packed_weight, int(quant_type), int(vocab), t1.long().contiguous(), int(chunk_rows),
                                               float(grad_scale))
    return loss, d_hidden.reshape(hidden.shape)


__all__ = ["lm_head_loss", "mmq_multi", "moe_mlp", "swiglu"]
