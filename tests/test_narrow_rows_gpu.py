"""Dispatch and combine of rows that are no multiple of 16 bytes, at row lengths around the
rounds and pieces they are moved in, against torch: whole rows for dispatch; for combine the
same products and sums in fp32, one path after the other, rounded once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1, 2, 3, 31, 33, 62, 64, 65, 127, 129, 255, 257, 510, 514, 1002,
                                   1023, 1026, 2049, 2050, 4098])
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("padded", [False, True])
def test_narrow_rows(width, dtype, padded):
    check(777, 5, width, dtype, padded)


@pytest.mark.parametrize("width,dtype", [(130, torch.bfloat16), (230, torch.float16),
                                         (301, torch.bfloat16), (500, torch.float16),
                                         (506, torch.bfloat16), (514, torch.float16),
                                         (65, torch.float32), (255, torch.float32)])
@pytest.mark.parametrize("padded", [False, True])
def test_narrow_rows_of_many_cells(width, dtype, padded):
    """More items than a resident wave of warps, between and around 256 and 1024 bytes a row."""
    check(9473, 7, width, dtype, padded)


def check(cells, paths, width, dtype, padded):
    from brainstorm_b200._C import router as R

    if dtype == torch.float16 and width % 2:
        pytest.skip("odd fp16 cells are refused")
    g = torch.Generator(device="cuda").manual_seed(width)
    mask = (torch.rand((cells, paths), generator=g, device="cuda") < 0.4).to(torch.int32)
    indices, loads = R.generate_indices_and_loads(mask)
    slot = int(loads.max()) + 3
    x = torch.randn((cells, width), generator=g, device="cuda").to(dtype)
    gates = torch.rand((cells, paths), generator=g, device="cuda")
    base = torch.arange(paths, device="cuda") * slot if padded else loads.cumsum(0) - loads
    cell, path = (indices > 0).nonzero(as_tuple=True)
    at = base[path] + indices[cell, path] - 1
    total = slot * paths if padded else int(loads.sum())
    for weights in (None, gates.to(dtype)):
        want = torch.zeros((total, width), dtype=dtype, device="cuda")
        moved = x[cell]
        if weights is not None:
            moved = (moved.float() * weights[cell, path].float()[:, None]).to(dtype)
        want[at] = moved
        (rows,) = R.dispatch_with_indices_and_loads(x, indices, loads, weights, False, None, padded,
                                                    slot if padded else 0)
        assert torch.equal(rows, want)
    residual = torch.randn((cells, width), generator=g, device="cuda").to(dtype)
    for weights in (None, gates, gates.to(dtype)):
        acc = torch.zeros((cells, width), device="cuda")
        for e in range(paths):
            mine = indices[:, e] > 0
            row = rows[base[e] + indices[mine, e] - 1].float()
            if weights is not None:
                row = row * weights[mine, e].float()[:, None]
            acc[mine] = acc[mine] + row
        for keep in (None, residual):
            want = acc.to(dtype)
            if keep is not None:
                none = (indices > 0).sum(dim=1) == 0
                want[none] = keep[none]
            (out,) = R.combine_with_indices_and_loads(rows, indices, loads, weights,
                                                      None if keep is None else keep.clone(),
                                                      padded)
            assert torch.equal(out, want)
