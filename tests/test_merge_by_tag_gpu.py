"""Merging paths by tag without fusing their cells, against the two operators it stands for (which
are compared with the checker elsewhere): row counts around the one-CTA sort, one to many
paths, empty paths, padding tags, negative tags, rows with and without 16-byte alignment.  Bit
for bit: both add a tag's rows in ascending order."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def pieces(total, paths, span, width, dtype, seed, lowest):
    g = torch.Generator().manual_seed(seed)
    cuts = sorted(torch.randint(0, total + 1, (paths - 1,), generator=g).tolist())
    sizes = [b - a for a, b in zip([0] + cuts, cuts + [total])]
    tags = torch.randint(lowest, lowest + span, (total,), generator=g, dtype=torch.int32).cuda()
    cells = torch.randn((total,) + width, generator=g).to(dtype).cuda()
    datas = [c.clone() if i % 2 else c for i, c in enumerate(cells.split(sizes))]
    return datas, list(tags.split(sizes))


@pytest.mark.parametrize("total,paths,span", [(2, 1, 1), (3, 2, 5), (31, 128, 9), (1000, 8, 300),
                                              (1024, 3, 1), (4095, 16, 4000), (4096, 16, 7),
                                              (4097, 16, 2000), (30000, 128, 12000)])
@pytest.mark.parametrize("width,dtype", [((4,), torch.float32), ((3,), torch.float32),
                                         ((2, 12), torch.bfloat16), ((7,), torch.float16),
                                         ((), torch.float32)])
@pytest.mark.parametrize("lowest", [0, 1, -3])
def test_merge_equals_fuse_and_combine(total, paths, span, width, dtype, lowest):
    from brainstorm_b200._C import router as R

    datas, tags = pieces(total, paths, span, width, dtype, total + paths, lowest)
    for padded in (False, True):
        got = R._merge_paths_by_tag(datas, tags, padded)
        fused, fused_tags, inverse = R.fuse_split_cells_from_paths(datas, is_tag_fuse=True,
                                                                   loads=None, tags=tags)
        want = R.combine_with_indices_and_loads(fused, inverse, None, None, None,
                                                ever_padded=padded, is_tag_index=True,
                                                tags=fused_tags)
        for a, b in zip(got, want):
            assert a.dtype == b.dtype and torch.equal(a, b)


def test_what_the_merge_leaves_to_the_two_operators():
    from brainstorm_b200._C import router as R

    datas, tags = pieces(20, 3, 9, (4,), torch.float32, 1, 1)
    assert R._merge_paths_by_tag([d.double() for d in datas], tags, False) is None
    assert R._merge_paths_by_tag(datas, [t.long() for t in tags], False) is None
    assert R._merge_paths_by_tag(datas[:1] + [d[:, :2] for d in datas[1:]], tags, False) is None
    assert R._merge_paths_by_tag([datas[0][:1]], [tags[0][:1]], False) is None
    assert R._merge_paths_by_tag([d.cpu() for d in datas], tags, False) is None
