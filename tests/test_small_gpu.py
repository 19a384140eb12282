"""Few tokens per weight row (dense calls of at most 24 rows whose fragments fit in shared memory, sparsely
hit experts) take a kernel of their own: the edges of its row, token and reduction tiles, its grouped work list and its multi-weight
launch, against the fp32 oracle."""
import numpy as np
import pytest
import torch

from oracle import blocks, ref
from helpers import ALL_TYPES, dense_case, expert_case, routing_from_sizes, to_dev

pytestmark = pytest.mark.gpu

# The result is rounded to bf16 once (8 significant bits: half a unit is at most 2^-8 of a value), the
# weights not at all; IQ2_S rounds magnitude * scale to bf16 as well, an independent error of the same
# size per product.
TOL = {qt: 2.0 ** -8 * (2.0 ** 0.5 if qt == ref.IQ2_S else 1.0) for _, qt in ALL_TYPES}


@pytest.mark.parametrize("name,qt", ALL_TYPES)
@pytest.mark.parametrize("M,N,K", [(1, 1, 256), (7, 17, 512), (8, 128, 256), (9, 1000, 2304), (16, 40, 768), (17, 4100, 512),
                                   (24, 16, 2048), (3, 72, 5120), (2, 60000, 256)])
def test_dense(cuda, name, qt, M, N, K):
    import torch_ggml_ops_b200 as tgo

    w, W, _ = dense_case(qt, N, K, 3 + qt)
    x = blocks.gaussian_bf16((M, K), M)
    y = tgo.mmq(to_dev(x), to_dev(w), qt, N)
    assert ref.rel_frobenius(y.float().cpu(), ref.mmq_forward(x, W)) < TOL[qt]


@pytest.mark.parametrize("name,qt", ALL_TYPES)
def test_no_less_exact_than_rounded_weights(cuda, name, qt):
    """Against 64 bits: at most the error of the exact product with weights rounded to bf16, as the GEMM has
    them, rounded to bf16 (98304 results: either error is known to a quarter of a percent)."""
    import torch_ggml_ops_b200 as tgo

    M, N, K = 24, 4096, 1024
    w, W, Wb = dense_case(qt, N, K, 30 + qt)
    x = blocks.gaussian_bf16((M, K), M)
    want = x.double() @ torch.from_numpy(W).double().t()
    rounded = (x.double() @ Wb.double().t()).to(torch.bfloat16).double()
    y = tgo.mmq(to_dev(x), to_dev(w), qt, N).double().cpu()
    assert float((y - want).norm()) < float((rounded - want).norm())


@pytest.mark.parametrize("name,qt", ALL_TYPES)
@pytest.mark.parametrize("N,K", [(72, 2048), (40, 512)])
@pytest.mark.parametrize("sizes", [[1, 0, 8, 9, 3, 40, 2, 1], [28, 1, 10, 17, 7, 9]])
def test_grouped_pair_and_invalid_groups(cuda, name, qt, N, K, sizes):
    from torch_ggml_ops_b200 import native

    E = len(sizes) + 2
    ids = list(range(E - 1, 1, -1))
    w0, W0 = expert_case(qt, E, N, K, 1)
    w1, W1 = expert_case(qt, E, N, K, 2)
    ei, eo = routing_from_sizes(sizes, ids)
    ei[2] = E   # its rows must stay as they are
    R = sum(sizes)
    x = blocks.gaussian_bf16((R, K), 3)
    y0, y1 = (torch.full((R, N), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ws = torch.empty(native.grouped_workspace_bytes(R, len(sizes)), dtype=torch.uint8, device="cuda")
    native.grouped_fwd(to_dev(x), to_dev(w0), to_dev(w1), y0, y1, to_dev(ei), to_dev(eo), E, R, N, K, qt, ws)
    skip = np.zeros(R, dtype=bool)
    skip[int(eo[1]):int(eo[2])] = True
    live = torch.from_numpy(~skip)
    for y, W in ((y0, W0), (y1, W1)):
        got, want = y.float().cpu(), ref.grouped_forward(x, W, ei.tolist(), eo.tolist())
        assert bool((got[~live] == 7.0).all())
        assert ref.rel_frobenius(got[live], want[live]) < TOL[qt]


def test_several_weights_in_one_launch(cuda):
    import torch_ggml_ops_b200 as tgo

    qt, M, N, K = ref.Q5_K, 5, 200, 512
    ws = [to_dev(blocks.dense_weight(qt, N, K, s)) for s in range(4)]
    x = to_dev(blocks.gaussian_bf16((M, K), 9))
    for y, w in zip(tgo.mmq_multi(x, ws, qt, N), ws):
        assert torch.equal(y, tgo.mmq(x, w, qt, N))


@pytest.mark.parametrize("name,qt", ALL_TYPES)
@pytest.mark.parametrize("M,N,K", [(3, 17, 512), (17, 72, 2304), (24, 200, 512)])
def test_infinite_and_huge_values(cuda, name, qt, M, N, K):
    """An infinite activation gives the infinities of the weights' signs (NaN where two meet or the weight is
    zero), a huge one the finite product, an infinite block scale likewise; other tokens and rows keep their bits."""
    import torch_ggml_ops_b200 as tgo

    w, W, Wb = dense_case(qt, N, K, 3 + qt)
    x = blocks.gaussian_bf16((M, K), M)
    plain = tgo.mmq(to_dev(x), to_dev(w), qt, N).cpu()
    odd = x.clone()
    odd[0, K - 1] = float("inf")
    odd[1, 5], odd[1, 300] = float("-inf"), float("inf")
    odd[2] *= 2.0 ** 118
    bad = np.asarray(w).reshape(N, K // 256, -1).copy()
    d_at = {ref.Q3_K: 108, ref.Q6_K: 208}.get(qt, 0)
    bad[5, 1, d_at:d_at + 2] = np.array([np.inf], dtype=np.float16).view(np.uint8)
    Wd = Wb.double()
    y = tgo.mmq(to_dev(odd), to_dev(w), qt, N).cpu()
    want = (odd.double()[:3, None, :] * Wd[None]).sum(-1)
    assert torch.equal(torch.isnan(y[:2]), torch.isnan(want[:2]))
    live = ~torch.isnan(want[:2])
    assert torch.equal(y[:2].double()[live], want[:2][live]) and bool(torch.isinf(want[:2][live]).all())
    assert bool(torch.isfinite(y[2]).all()) and ref.rel_frobenius(y[2].double() * 2.0 ** -118, want[2] * 2.0 ** -118) < 2.0 ** -7
    assert torch.equal(y[3:], plain[3:])
    # one infinite scale: that row alone, infinite or NaN as the decoded weights make it
    z = tgo.mmq(to_dev(x), to_dev(bad), qt, N).cpu()
    wide = tgo.mmq(to_dev(torch.cat([x, x.new_zeros(64, K)])), to_dev(bad), qt, N).cpu()[:M]   # enough rows for the tile GEMM
    assert bool((~torch.isfinite(z[:, 5])).all())
    assert torch.equal(torch.isnan(z[:, 5]), torch.isnan(wide[:, 5])) and torch.equal(torch.nan_to_num(z[:, 5]), torch.nan_to_num(wide[:, 5]))
    keep = torch.arange(N) != 5
    assert torch.equal(z[:, keep], plain[:, keep])


@pytest.mark.parametrize("name,qt", ALL_TYPES)
@pytest.mark.parametrize("M,K,few", [(8, 4096, True), (9, 4096, True), (16, 4096, True), (25, 4096, False), (16, 7168, False),
                                     (8, 8192, True), (1, 16384, False)])
def test_shared_memory_limits(cuda, name, qt, M, K, few):
    """Rows x in_features whose fragments leave room for the slices only if there are fewer of them, or for none:
    the few-token kernel (which does not round the weights to bf16: a smaller error) or the tile GEMM."""
    import torch_ggml_ops_b200 as tgo

    N = 40
    w, W, Wb = dense_case(qt, N, K, 3 + qt)
    x = blocks.gaussian_bf16((M, K), M)
    ws = [to_dev(w), to_dev(dense_case(qt, N, K, 4 + qt)[0])]
    y = tgo.mmq(to_dev(x), ws[0], qt, N)
    assert ref.rel_frobenius(y.float().cpu(), ref.mmq_forward(x, W)) < 2 * TOL[qt]
    # rounded weights, exact product: the GEMM's result up to its own rounding to bf16, the other kernel's not
    rounded = (x.double() @ Wb.double().t()).to(torch.bfloat16)
    same = float((y.cpu() == rounded).float().mean())
    assert (same < 0.95) == few, same
    assert torch.equal(tgo.mmq_multi(to_dev(x), ws, qt, N)[0], y)


@pytest.mark.parametrize("name,qt", ALL_TYPES)
def test_infinite_values_in_groups(cuda, name, qt):
    from torch_ggml_ops_b200 import native

    sizes, ids, E, N, K = [3, 9, 1, 12], [4, 1, 3, 0], 5, 40, 512
    w0, w1 = (blocks.expert_weights(qt, E, N, K, s) for s in (1, 2))
    ei, eo = routing_from_sizes(sizes, ids)
    R = sum(sizes)
    x = blocks.gaussian_bf16((R, K), 3)
    x[4, 17], x[20, 511] = float("inf"), float("-inf")
    y0, y1 = (torch.empty((R, N), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ws = torch.empty(native.grouped_workspace_bytes(R, len(sizes)), dtype=torch.uint8, device="cuda")
    native.grouped_fwd(to_dev(x), to_dev(w0), to_dev(w1), y0, y1, to_dev(ei), to_dev(eo), E, R, N, K, qt, ws)
    for y, w in ((y0, w0), (y1, w1)):
        got = y.double().cpu()
        W = torch.from_numpy(ref.expert_weights_fp32(w, qt, N, K)).to(torch.bfloat16).double()
        for r, e in ((4, 1), (20, 0)):
            want = (x[r].double() * W[e]).sum(-1)
            assert torch.equal(torch.isnan(got[r]), torch.isnan(want))
            assert torch.equal(got[r][~torch.isnan(want)], want[~torch.isnan(want)])
        rest = torch.ones(R, dtype=torch.bool)
        rest[[4, 20]] = False
        assert bool(torch.isfinite(got[rest]).all())
