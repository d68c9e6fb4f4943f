"""The pipelined dispatch at the edges of the items a CTA owns: cell counts around a CTA's span and
around one resident wave, rows of one and of several pieces, slots and capacities that leave rows to
zero, up to more paths than a CTA has threads.  Against the same call on a copy of the indices,
which takes the general kernels; whole bytes."""
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
    for weights in (None, gates):
        for tags in (False, True):
            got = R.dispatch_with_indices_and_loads(x, indices, loads, weights, tags, None, padded,
                                                    slot if padded else 0)
            want = R.dispatch_with_indices_and_loads(x, indices.clone(), loads, weights, tags,
                                                     None, padded, slot if padded else 0)
            for a, b in zip(got, want):
                assert a.shape == b.shape
                assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
