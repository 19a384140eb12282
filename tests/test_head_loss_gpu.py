"""``lm_head_loss`` on the GPU beyond its plain call (test_extras_gpu.py): what autograd gets from it and its
element-wise kernels at awkward inputs."""
import numpy as np
import pytest
import torch

from oracle import blocks, ref
from helpers import ALL_TYPES, dense_case, to_dev

pytestmark = pytest.mark.gpu


def _inputs(qt, V, K, T, seed=8):
    w, W, _ = dense_case(qt, V, K, seed)
    hidden = (blocks.gaussian_bf16((T, K), 9).float() * 0.02).to(torch.bfloat16)   # logits with a spread of about one
    targets = torch.from_numpy(np.random.default_rng(1).integers(0, V, size=T))
    return w, W, hidden, targets


def _fp64(W, hidden, targets):
    h = hidden.double().requires_grad_(True)
    loss = torch.nn.functional.cross_entropy(h @ torch.from_numpy(W).double().t(), targets, reduction="sum")
    loss.backward()
    return loss.detach(), h.grad


# input gradient in one range, cut into ranges, and over several token tiles
@pytest.mark.parametrize("V,K,T,chunk", [(1000, 512, 90, 32), (8200, 512, 70, 256), (1000, 512, 1100, 1100)])
@pytest.mark.parametrize("name,qt", ALL_TYPES)
def test_gradient_through_autograd(cuda, name, qt, V, K, T, chunk):
    import torch_ggml_ops_b200 as tgo

    w, W, hidden, targets = _inputs(qt, V, K, T)
    wd, td = to_dev(w), to_dev(targets)
    want_loss, want = _fp64(W, hidden, targets)
    plain = tgo.lm_head_loss(to_dev(hidden), wd, qt, V, td, chunk_rows=chunk)[1]
    loss, d, d32 = torch.ops.torch_ggml_ops_b200.lm_head_loss_f32(to_dev(hidden), wd, qt, V, td, chunk, 1.0)
    assert torch.equal(d, plain) and torch.equal(d, d32.to(torch.bfloat16))
    for scale, cotangent in ((1.0, 0.37), (0.5, 1.0), (0.0, -2.0)):
        x = to_dev(hidden).requires_grad_(True)
        out, dh = tgo.lm_head_loss(x, wd, qt, V, td, chunk_rows=chunk, grad_scale=scale)
        (out * cotangent).backward()
        assert torch.equal(x.grad, (d32 * cotangent).to(torch.bfloat16))   # powers of two: the scale leaves no trace
        assert ref.rel_frobenius(x.grad.double().cpu(), want * cotangent) < 1e-2
        assert abs(float(out) - float(want_loss)) < 2e-3 * float(want_loss)
        assert ref.rel_frobenius(dh.detach().double().cpu(), want * scale) < 1e-2 if scale else not dh.detach().any()
