"""The autograd side of ``lm_head_loss`` (csrc/torch_ext.cpp) without a GPU: the operator's CUDA kernel is
stood in for by a plain CPU one, everything above it is the package's own."""
import pytest
import torch

V, K, T = 40, 16, 12


def _weight(w):
    return w.view(-1).float()[: V * K].reshape(V, K) / 128 - 1


def _loss(h, w, quant_type, vocab, targets, chunk_rows, grad_scale):
    lp = torch.log_softmax(h.float() @ _weight(w).t(), -1)
    loss = -lp.gather(1, targets[:, None]).sum()
    d = lp.exp().scatter_add_(1, targets[:, None], torch.full((h.shape[0], 1), -1.0)) * grad_scale
    d = d @ _weight(w)
    return loss, d.to(h.dtype), d


@pytest.fixture
def head():
    import torch_ggml_ops_b200 as tgo

    lib = torch.library.Library("torch_ggml_ops_b200", "IMPL")
    lib.impl("lm_head_loss", lambda *a: _loss(*a)[:2], "CPU")
    lib.impl("lm_head_loss_f32", _loss, "CPU")
    g = torch.Generator().manual_seed(1)
    w = torch.randint(0, 256, (V * K,), dtype=torch.uint8, generator=g)
    hidden = torch.randn(T, K, generator=g).to(torch.bfloat16)
    targets = torch.randint(0, V, (T,), generator=g)
    yield hidden, lambda h, **kw: tgo.lm_head_loss(h, w, 14, V, targets, **kw)
    lib._destroy()


def test_second_derivatives_are_refused(head):
    """The loss is not linear in hidden: a gradient without a graph would silently lose its Hessian."""
    hidden, loss_of = head
    x = hidden.clone().requires_grad_()
    (dx,) = torch.autograd.grad(loss_of(x)[0], x, create_graph=True)
    assert dx.requires_grad
    with pytest.raises(RuntimeError, match="higher-order"):
        torch.autograd.grad((x ** 2).sum().float() + (dx.float() ** 2).sum(), x)
    # neither with respect to the cotangent
    y = hidden.clone().requires_grad_()
    with pytest.raises(RuntimeError, match="higher-order"):
        (dy,) = torch.autograd.grad(loss_of(y)[0] ** 2, y, create_graph=True)
        dy.float().sum().backward()
    # a first derivative is not affected, and hidden may change once the loss has been computed
    z = hidden.clone().requires_grad_()
    h = z * 1
    loss = loss_of(h)[0]
    h.add_(1)
    loss.backward()
    assert torch.equal(z.grad, dx.detach())


def test_a_derivative_of_the_returned_gradient_is_refused(head):
    hidden, loss_of = head
    x = hidden.clone().requires_grad_()
    loss, d = loss_of(x)
    assert d.requires_grad
    with pytest.raises(RuntimeError, match="higher-order"):
        torch.autograd.grad(loss + d.float().sum(), x)


@pytest.mark.parametrize("grad_scale", [1.0, 0.3, 3.0, 0.0, 1e-45, 1e38])
def test_the_gradient_is_rounded_once(head, grad_scale):
    """cotangent * gradient in fp32, then one rounding: at most half a unit in the last of bf16's 8 significant
    bits, 2^-9 of a value's power of two (a thousandth of it is left to the fp32 products)."""
    hidden, loss_of = head
    for cotangent in (1.0, 0.37, -1.0 / 3.0, 1e-3):
        x = hidden.clone().requires_grad_()
        loss, d = loss_of(x, grad_scale=grad_scale)
        with torch.no_grad():
            d.mul_(2)   # the caller's copy is the caller's
        (loss * cotangent).backward()
        y = hidden.double().requires_grad_()
        w = _weight(torch.randint(0, 256, (V * K,), dtype=torch.uint8, generator=torch.Generator().manual_seed(1)))
        g = torch.Generator().manual_seed(1)
        torch.randint(0, 256, (V * K,), dtype=torch.uint8, generator=g), torch.randn(T, K, generator=g)
        targets = torch.randint(0, V, (T,), generator=g)
        (torch.nn.functional.cross_entropy(y @ w.double().t(), targets, reduction="sum") * cotangent).backward()
        unit = torch.exp2(torch.floor(torch.log2(y.grad.abs())) - 7)
        assert bool(((x.grad.double() - y.grad).abs() <= 0.501 * unit + 1e-6 * y.grad.abs().max()).all())


def test_no_rows(head):
    """Nothing to compute: a loss of zero and an empty gradient, whatever the weight and the device."""
    import torch_ggml_ops_b200 as tgo

    for hidden in (torch.empty(0, K, dtype=torch.bfloat16), torch.empty(2, 0, K), torch.empty(0, K, dtype=torch.bfloat16, requires_grad=True)):
        loss, d = tgo.lm_head_loss(hidden, torch.empty(0, dtype=torch.uint8), 14, V, torch.empty(0, dtype=torch.long))
        assert loss.dtype == torch.float32 and float(loss) == 0.0 and not loss.requires_grad
        assert d.shape == hidden.shape and d.dtype == hidden.dtype
