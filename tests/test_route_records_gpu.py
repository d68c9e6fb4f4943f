"""Dispatch and combine through the route records that the index scan leaves beside its
indices, against the same calls without them (and those against the checker elsewhere): records
that are full, overfull and empty, loads that cut routes off, odd path counts, all row types.
Bit for bit: the order and the rounding of the sums do not depend on where the routes come from."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def make(R, cells, paths, density, seed, cap):
    g = torch.Generator(device="cuda").manual_seed(seed)
    odds = torch.tensor(density, device="cuda")[
        torch.randint(0, len(density), (cells, 1), generator=g, device="cuda")]
    mask = (torch.rand((cells, paths), generator=g, device="cuda") < odds).to(torch.int32)
    caps = None if cap is None else torch.tensor([cap], dtype=torch.int32, device="cuda")
    return R.generate_indices_and_loads(mask, caps)


@pytest.mark.parametrize("cells,paths", [(131072, 17), (80000, 30), (65536, 32), (22001, 97),
                                         (8192, 256), (1 << 20, 20)])
@pytest.mark.parametrize("dtype,width", [(torch.float32, 4), (torch.bfloat16, 24),
                                         (torch.float16, 1032), (torch.bfloat16, 2056)])
@pytest.mark.parametrize("capped", [False, True])
def test_records_give_the_same_rows_and_sums(cells, paths, dtype, width, capped):
    from brainstorm_b200._C import router as R

    if cells * width > 1 << 26:
        width = 8
    # 0 to all routes per cell; four in the mean, so that most records are full or overfull
    density = [0.0, 1.0 / paths, 4.0 / paths, 8.0 / paths] + ([1.0] if cells <= 131072 else [])
    cap = cells // 20 if capped else None
    indices, loads = make(R, cells, paths, density, cells + paths, cap)
    assert getattr(indices, R._RECORDS, None) is not None
    plain = indices.clone()  # no notes: the general kernels
    assert getattr(plain, R._RECORDS, None) is None
    x = torch.randn((cells, width), device="cuda").to(dtype)
    gates = torch.rand((cells, paths), device="cuda")
    mpl = int(loads.max())
    if mpl * paths * width > 1 << 29:
        mpl = 0
    for weights in (None, gates.to(dtype)):
        (a,) = R.dispatch_with_indices_and_loads(x, indices, loads, weights, False, None, mpl > 0,
                                                 mpl)
        (b,) = R.dispatch_with_indices_and_loads(x, plain, loads, weights, False, None, mpl > 0,
                                                 mpl)
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    residual = torch.randn((cells, width), device="cuda").to(dtype)
    for weights in (None, gates, gates.to(dtype)):
        for keep in (None, residual):
            (c,) = R.combine_with_indices_and_loads(a, indices, loads, weights,
                                                    None if keep is None else keep.clone(),
                                                    mpl > 0)
            (d,) = R.combine_with_indices_and_loads(a, plain, loads, weights,
                                                    None if keep is None else keep.clone(),
                                                    mpl > 0)
            assert torch.equal(c.view(torch.uint8), d.view(torch.uint8))


def test_notes_of_edited_or_special_tensors_are_not_used():
    from brainstorm_b200._C import router as R

    indices, loads = make(R, 65536, 32, [0.05], 5, None)
    assert R._records_of(indices, 65536, 32) is not None
    assert R._records_of(indices, 65535, 32) is None
    x = torch.randn((65536, 8), device="cuda")
    indices[7] = 0  # in place: the cell goes nowhere now
    assert R._records_of(indices, 65536, 32) is None
    (rows,) = R.dispatch_with_indices_and_loads(x, indices, loads)
    (out,) = R.combine_with_indices_and_loads(rows, indices, loads)
    assert float(out[7].abs().sum()) == 0.0
    with torch.inference_mode():
        indices, loads = make(R, 65536, 32, [0.05], 5, None)
    assert getattr(indices, R._RECORDS, None) is None
    # values other than 0/1: the seats are no counts, every record sends its reader to the row
    mask = torch.zeros((65536, 32), dtype=torch.int32, device="cuda")
    mask[::2, 3] = 2
    indices, loads = R.generate_indices_and_loads(mask)
    records = getattr(indices, R._RECORDS)[0].view(65536, 8)
    assert bool(((records[:, 0] & 0x40000000) != 0).all())


def test_records_used_on_another_stream_outlive_their_tensor():
    from brainstorm_b200._C import router as R

    indices, loads = make(R, 65536, 32, [0.05], 9, None)
    x = torch.randn((65536, 64), device="cuda")
    total = int(loads.max())
    (want,) = R.dispatch_with_indices_and_loads(x, indices.clone(), loads, None, False, None, True,
                                                total)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)
        (got,) = R.dispatch_with_indices_and_loads(x, indices, loads, None, False, None, True, total)
    for t in (indices, loads, x):
        t.record_stream(side)
    counts = getattr(indices, R._DENSE)
    counts.record_stream(side)
    del indices, t
    junk = [torch.full((65536 * 8,), -1, dtype=torch.int32, device="cuda") for _ in range(8)]
    side.synchronize()
    assert torch.equal(got, want) and len(junk) == 8


def test_a_graph_does_not_keep_records_of_indices_made_before_it():
    from brainstorm_b200._C import router as R

    indices, loads = make(R, 65536, 32, [0.05], 11, None)
    later, later_loads = make(R, 65536, 32, [0.05], 12, None)
    assert R._records_of(indices, 65536, 32) is not None
    rows = torch.randn((int(later_loads.max()) * 2 * 32, 8), device="cuda")

    def run(at, n):
        return R.combine_with_indices_and_loads(rows, at, n, None, None, True)[0]

    run(indices, loads)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run(indices, loads)
        inside, _ = R.generate_indices_and_loads((indices > 0).to(torch.int32))
        assert R._records_of(inside, 65536, 32) is not None
    assert R._records_of(inside, 65536, 32) is None
    indices.copy_(later)
    loads.copy_(later_loads)
    graph.replay()
    assert torch.equal(out, run(later, later_loads))


def test_notes_do_not_follow_a_tensor_to_other_memory():
    from brainstorm_b200._C import router as R

    indices, loads = make(R, 65536, 32, [0.05], 13, None)
    later, _ = make(R, 65536, 32, [0.05], 14, None)
    indices.data = later.clone()
    assert R._records_of(indices, 65536, 32) is None
    rows = torch.randn((65536 * 4, 8), device="cuda")
    (a,) = R.combine_with_indices_and_loads(rows, indices, loads, None, None, True)
    (b,) = R.combine_with_indices_and_loads(rows, indices.clone(), loads, None, None, True)
    assert torch.equal(a, b)
