"""Index tensors that a program edits after the scan, in ways that a version counter does not see: the
operators go by what the tensor holds when they run.  Against the same call on a copy of the edited
tensor, which carries nothing of where it came from; whole bytes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CELLS, PATHS = 1 << 17, 32  # 2^22 elements: 16 MB of indices


def through_data(t, rows, values):
    t.data[rows] = values


def through_dlpack(t, rows, values):
    torch.utils.dlpack.from_dlpack(torch.utils.dlpack.to_dlpack(t))[rows] = values


def in_place(t, rows, values):
    t[rows] = values


@pytest.mark.parametrize("edit", [through_data, through_dlpack, in_place])
@pytest.mark.parametrize("from_scores", [False, True])
def test_edits_between_the_operators_are_seen(edit, from_scores):
    from brainstorm_b200._C import router as R

    g = torch.Generator(device="cuda").manual_seed(3)
    score = torch.rand((CELLS, PATHS), generator=g, device="cuda")
    if from_scores:
        indices, loads = R.route_scores(score, "topk", 2, output="seat_indices")
    else:
        indices, loads = R.generate_indices_and_loads((score > 0.93).to(torch.int32))
    x = torch.randn((CELLS, 64), generator=g, device="cuda").bfloat16()
    slot = int(loads.max())
    # two cells change places: the columns still hold every seat once
    pair = torch.tensor([5, CELLS - 9], device="cuda")
    edit(indices, pair, indices[pair.flip(0)])
    (rows,) = R.dispatch_with_indices_and_loads(x, indices, loads, None, False, None, True, slot)
    (want,) = R.dispatch_with_indices_and_loads(x, indices.clone(), loads, None, False, None, True,
                                                slot)
    assert torch.equal(rows, want)
    # a cell's routes are dropped between dispatch and combine
    edit(indices, pair[:1], torch.zeros((1, PATHS), dtype=torch.int32, device="cuda"))
    for gates in (None, score):
        (out,) = R.combine_with_indices_and_loads(rows, indices, loads, gates, None, True)
        (want,) = R.combine_with_indices_and_loads(rows, indices.clone(), loads, gates, None, True)
        assert torch.equal(out, want)
        assert not out[5].any()


def test_a_graph_reads_the_indices_of_each_replay():
    from brainstorm_b200._C import router as R

    def scan(seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        return R.generate_indices_and_loads(
            (torch.rand((CELLS, PATHS), generator=g, device="cuda") < 0.05).to(torch.int32))

    indices, loads = scan(11)
    later, later_loads = scan(12)
    slot = 2 * int(later_loads.max())
    rows = torch.randn((slot * PATHS, 8), device="cuda")

    def run(at, n):
        return R.combine_with_indices_and_loads(rows, at, n, None, None, True)[0]

    run(indices, loads)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run(indices, loads)
    indices.copy_(later)
    loads.copy_(later_loads)
    graph.replay()
    assert torch.equal(out, run(later, later_loads))
