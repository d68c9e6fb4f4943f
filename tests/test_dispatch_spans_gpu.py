"""The pipelined dispatch at the edges of the items a CTA owns: cell counts around a CTA's span and
around one resident wave, rows of one and of several pieces, slots and capacities that leave rows to
zero, up to more paths than a CTA has threads.  Rows, tags and zeros against torch, for the indices
as the scan returned them and for a copy of them, whose empty rows a second launch zeroes; whole
bytes (a weighted row is one product, rounded once)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [2, 7, 8, 9, 15, 17, 31, 33, 4737, 18943, 18945, 40000])
@pytest.mark.parametrize("paths,width", [(4, 8), (30, 1032), (32, 2056), (257, 16), (1000, 8)])
@pytest.mark.parametrize("layout", ["packed", "capacity", "slots", "wide slots"])
def test_spans(cells, paths, width, layout):
    from brainstorm_b200._C import router as R

    if cells * max(width, paths) > 1 << 25:
        cells = (1 << 25) // max(width, paths)
    g = torch.Generator(device="cuda").manual_seed(cells + paths)
    mask = (torch.rand((cells, paths), generator=g, device="cuda") < 2.0 / paths).to(torch.int32)
    caps = None
    if layout == "capacity":  # loads rounded up: packed slots with rows to zero at their end
        caps = torch.tensor([3, 50, 4000, 50000], dtype=torch.int32, device="cuda")
    indices, loads = R.generate_indices_and_loads(mask, caps, caps is not None)
    slot = int(loads.max()) + (40 if layout == "wide slots" else 0)
    padded = "slots" in layout
    x = torch.randn((cells, width), generator=g, device="cuda").bfloat16()
    gates = torch.rand((cells, paths), generator=g, device="cuda").bfloat16()
    base = torch.arange(paths, device="cuda") * slot if padded else loads.cumsum(0) - loads
    total = slot * paths if padded else int(loads.sum())
    cell, path = mask.nonzero(as_tuple=True)
    at = base[path] + mask.cumsum(dim=0)[cell, path] - 1
    want_tags = torch.zeros(total, dtype=torch.int32, device="cuda")
    want_tags[at] = (cell + 1).to(torch.int32)
    for weights in (None, gates):
        want = torch.zeros((total, width), dtype=torch.bfloat16, device="cuda")
        want[at] = x[cell] if weights is None else \
            (x[cell].float() * weights[cell, path].float()[:, None]).bfloat16()
        for idx in (indices, indices.clone()):
            for tags in (False, True):
                got = R.dispatch_with_indices_and_loads(x, idx, loads, weights, tags, None, padded,
                                                        slot if padded else 0)
                assert got[0].shape == want.shape
                assert torch.equal(got[0].view(torch.int16), want.view(torch.int16))
                if tags:
                    assert torch.equal(got[1], want_tags)
