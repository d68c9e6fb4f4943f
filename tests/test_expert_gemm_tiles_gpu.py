"""Edges of the tiles of the grouped expert GEMM: loads around the 256 rows of a tile and the box
sizes its rows are fetched in, feature counts with and without CTA pairs, padded and packed
buffers.  Bound per element: one rounding to bf16 (2^-8 of the value) plus K fp32 additions
(K * 2^-24 of the sum of the products' magnitudes)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

EDGES = [1, 15, 16, 17, 31, 33, 64, 65, 127, 128, 129, 192, 193, 255, 256]
LONG = [257, 0, 288, 511, 512, 513, 769, 4097]


@pytest.mark.parametrize("K,N", [(64, 128), (128, 256), (192, 384), (320, 512)])
@pytest.mark.parametrize("loads,cap,relu", [(EDGES, 0, True), (LONG, 0, False), (EDGES, 257, False),
                                            ([0, 0, 3], 0, False), ([300] * 5, 300, True)])
def test_tile_edges(K, N, loads, cap, relu):
    from brainstorm_b200._C import expert

    E = len(loads)
    rows_total = cap * E if cap else sum(loads)
    g = torch.Generator(device="cuda").manual_seed(K + N + rows_total)
    rows = torch.randn(rows_total, K, device="cuda", generator=g).bfloat16()
    weights = torch.randn(E, N, K, device="cuda", generator=g).bfloat16()
    out = torch.full((rows_total, N), -7.0, device="cuda", dtype=torch.bfloat16)
    expert.grouped_expert_linear(rows, weights, torch.tensor(loads, dtype=torch.int32,
                                                             device="cuda"), bool(cap), cap, relu,
                                 out=out)
    expert.check_status()
    start = 0
    for e, load in enumerate(loads):
        begin = e * cap if cap else start
        a, w = rows[begin:begin + load].double(), weights[e].double()
        want = a @ w.T
        bound = 2.0 ** -8 * want.abs() + K * 2.0 ** -24 * (a.abs() @ w.abs().T)
        want = want.relu() if relu else want
        assert bool(((out[begin:begin + load].double() - want).abs() <= bound).all()), (e, load)
        if cap:  # rows of the slot beyond the load stay as they were
            assert bool((out[begin + load:begin + cap] == -7.0).all())
        start += load
