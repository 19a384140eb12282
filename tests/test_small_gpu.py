"""Few tokens per weight row (dense calls of at most 24 rows, sparsely hit experts) take a kernel of
their own: the edges of its row, token and reduction tiles, its grouped work list and its multi-weight
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
