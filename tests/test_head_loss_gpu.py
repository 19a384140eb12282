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
        assert abs(float(out.detach()) - float(want_loss)) < 2e-3 * float(want_loss)
        assert ref.rel_frobenius(dh.detach().double().cpu(), want * scale) < 1e-2 if scale else not dh.detach().any()


def _q6_rows(d):
    """Q6_K rows of one block whose 256 weights are all d (quants 33 - 32, scales 1), d a list of fp16 values."""
    b = np.zeros((len(d), 210), dtype=np.uint8)
    b[:, :128], b[:, 128:192], b[:, 192:208] = 0x11, 0xAA, 1
    b[:, 208:] = np.asarray(d, dtype=np.float16).view(np.uint8).reshape(-1, 2)
    return b


@pytest.mark.parametrize("at", [0, 8, 504, 992])
@pytest.mark.parametrize("bad", [[np.nan] * 8, [np.inf] * 7 + [np.nan], [np.inf] * 8, [-np.inf] * 8])
def test_non_finite_logits(cuda, bad, at):
    """x = -1: eight neighbouring columns are NaN, -inf or +inf, those that one thread of the statistics reads
    first among them; loss and gradient as log_softmax defines them."""
    import torch_ggml_ops_b200 as tgo

    V, K, T = 1000, 256, 40
    w, W, _ = dense_case(ref.Q6_K, V, K, 3)
    w = w.reshape(V, 210).copy()
    w[at:at + 8] = _q6_rows(bad)
    targets = torch.full((T,), 20)
    x = torch.full((T, K), -1.0, dtype=torch.bfloat16)
    logits = (x.double() @ torch.from_numpy(W).double().t())
    logits[:, at:at + 8] = -torch.tensor(bad, dtype=torch.float64)
    want = torch.nn.functional.cross_entropy(logits, targets, reduction="sum")
    loss, dh = tgo.lm_head_loss(to_dev(x), to_dev(w), ref.Q6_K, V, to_dev(targets))
    if torch.isnan(want):
        assert torch.isnan(loss) and torch.isnan(dh).all()
    else:   # the columns have no probability; 0 * inf leaves no gradient
        assert abs(float(loss) - float(want)) < 2e-3 * abs(float(want))


def test_strided_hidden(cuda):
    """Rows that lie apart are taken, columns that do are refused; the gradient has the layout that the fake
    kernel promises."""
    import torch_ggml_ops_b200 as tgo

    qt, V, K, T = ref.Q6_K, 1000, 256, 50
    w, _, hidden, targets = _inputs(qt, V, K, T)
    wd, td = to_dev(w), to_dev(targets)
    padded = to_dev(torch.nn.functional.pad(hidden, (3, 5)))[:, 3:3 + K]
    across = to_dev(hidden.t().contiguous()).t()
    for x, chunk in ((padded, 256), (padded, 16), (across, 1)):
        compiled = torch.compile(lambda h: tgo.lm_head_loss(h, wd, qt, V, td, chunk_rows=chunk), backend="aot_eager", fullgraph=True)
        loss, d = tgo.lm_head_loss(to_dev(hidden), wd, qt, V, td, chunk_rows=chunk)
        for got_loss, got in (tgo.lm_head_loss(x, wd, qt, V, td, chunk_rows=chunk), compiled(x)):
            assert got.stride() == torch.empty_like(x).stride()
            assert torch.equal(got, d) and torch.equal(got_loss, loss)
    for chunk in (256, 20, 49):
        with pytest.raises(RuntimeError, match="contiguous"):
            tgo.lm_head_loss(across, wd, qt, V, td, chunk_rows=chunk)
