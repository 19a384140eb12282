"""``mmq_multi`` in traced programs, without a GPU (a plain CPU kernel stands in for the CUDA one)."""
import pytest
import torch


def _weight(w, n, k):
    return w.view(-1).float()[: n * k].reshape(n, k) / 128 - 1


@pytest.mark.parametrize("train", [False, True])
def test_out_features_may_be_symbolic(train):
    """One graph serves every out_features of a weight whose size is marked dynamic."""
    import torch_ggml_ops_b200 as tgo

    own, base = torch.library.Library("torch_ggml_ops_b200", "IMPL"), torch.library.Library("torch_ggml_ops", "IMPL")
    own.impl("mmq_multi", lambda x, ws, qt, n: [(x.float() @ _weight(w, n, x.shape[-1]).t()).to(x.dtype) for w in ws], "CPU")
    base.impl("mmq_grad_input", lambda d, w, qt, k: (d.float() @ _weight(w, d.shape[-1], k)).to(d.dtype), "CPU")
    try:
        torch._dynamo.reset()
        step = lambda x, w: torch.cat(tgo.mmq_multi(x, [w, w], 12, w.shape[0]), -1)   # noqa: E731
        compiled = torch.compile(step, backend="aot_eager", fullgraph=True)
        for n in (24, 32, 40):
            w, x = torch.randint(0, 256, (n, 16), dtype=torch.uint8), torch.randn(5, 16).bfloat16().requires_grad_(train)
            torch._dynamo.mark_dynamic(w, 0)
            y = compiled(x, w)
            assert torch.equal(y, step(x, w))
            if train:
                assert torch.equal(*(torch.autograd.grad(v.float().sum(), x)[0] for v in (y, step(x, w))))
    finally:
        own._destroy()
        base._destroy()
