"""The single-launch index scan and gate at the edges of their tiles: cell counts around 32, a
tile, a CTA's run and the one-CTA limit, path counts with and without 16-byte rows, masks that
are written whole and masks that are zeroed and scattered into.  Whole values, compared bit for
bit with the checker."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu

CELLS = [1, 31, 33, 256, 257, 513, 1025, 9001, 40961]
PATHS = [1, 3, 5, 16, 30, 33, 36, 97, 129, 250, 256, 260]


def mask_of(rng, cells, paths, kind):
    if kind == "top1":
        mask = np.zeros((cells, paths), dtype=np.int32)
        mask[np.arange(cells), rng.integers(0, paths, cells)] = 1
        return mask
    if kind == "mixed":  # dense and sparse tiles in one mask
        odds = np.repeat(rng.choice([0.01, 0.12, 0.13, 0.9], (cells + 63) // 64), 64)[:cells, None]
        return (rng.random((cells, paths)) < odds).astype(np.int32)
    if kind == "ones":
        return np.ones((cells, paths), dtype=np.int32)
    # integer semantics; not below zero: the reference leaves a path at the first 1024 cells
    # whose sum passes its threshold, which a falling sum would tell from a cell by cell rule
    return rng.integers(0, 4, (cells, paths)).astype(np.int32)


@pytest.mark.parametrize("kind", ["top1", "mixed", "ones", "integers"])
@pytest.mark.parametrize("paths", PATHS)
@pytest.mark.parametrize("cells", CELLS)
def test_scan_edges(cells, paths, kind):
    from brainstorm_b200._C import router as R

    rng = np.random.default_rng(cells * 1000 + paths)
    mask = mask_of(rng, cells, paths, kind)
    dev = torch.from_numpy(mask).cuda()
    caps = [max(1, cells // 3)]
    caps_dev = torch.tensor(caps, dtype=torch.int32, device="cuda")
    for tag in (False, True):
        if kind == "integers" and tag:
            continue  # several cells may name one tag row; which of them stays is not defined
        got = R.generate_indices_and_loads(dev, caps_dev, False, False, tag)
        want = oracle.generate_indices_and_loads(mask, caps, False, False, tag)
        assert np.array_equal(got[0].cpu().numpy(), want[0]), tag
        assert np.array_equal(got[1].cpu().numpy(), want[1]), tag
    limit = rng.integers(0, cells + 2, paths).astype(np.int32)
    start = rng.integers(0, 3, paths).astype(np.int32)
    prefix = torch.from_numpy(start.copy()).cuda()
    got, _ = R.throttle_hotmask(dev, prefix, torch.from_numpy(limit).cuda())
    start_np = start.copy()
    want, _ = oracle.throttle_hotmask(mask, start_np, limit)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(prefix.cpu().numpy(), start_np)
    if kind != "integers":
        prefix = torch.from_numpy(start.copy()).cuda()
        idx, loads, _, throttled = R.throttle_and_generate_indices(
            dev, prefix, torch.from_numpy(limit).cuda(), caps_dev, with_mask=True)
        want_idx, want_loads = oracle.generate_indices_and_loads(want, caps)
        assert np.array_equal(throttled.cpu().numpy(), want)
        assert np.array_equal(idx.cpu().numpy(), want_idx)
        assert np.array_equal(loads.cpu().numpy(), want_loads)
        assert np.array_equal(prefix.cpu().numpy(), start_np)


@pytest.mark.parametrize("paths", [5, 30, 32, 256, 260])
@pytest.mark.parametrize("first", [-50, -9001, -46340])
def test_tags_after_a_run_with_a_negative_sum(paths, first):
    """A first run that sums to less than zero starts the 0/1 runs after it below seat 1: a cell
    whose seat is not a row of the output goes nowhere."""
    from brainstorm_b200._C import router as R

    cells = 9001
    rng = np.random.default_rng(paths)
    mask = (rng.random((cells, paths)) < 0.1).astype(np.int32)
    mask[0] = 0
    mask[0, ::2] = first  # index first * first, past the rows that the later seats name
    seat = np.cumsum(mask, axis=0, dtype=np.int64) * mask
    assert first * first > seat[1:].max() and seat.min() < 0
    want = np.zeros_like(mask)
    cell, path = np.nonzero((seat >= 1) & (seat <= cells))
    want[seat[cell, path] - 1, path] = cell + 1
    dev = torch.from_numpy(mask).cuda()
    got, loads = R.generate_indices_and_loads(dev, None, False, False, True)
    assert np.array_equal(got.cpu().numpy(), want)
    assert np.array_equal(loads.cpu().numpy(), mask.sum(axis=0))


def test_scan_of_an_array_that_is_only_4_byte_aligned():
    from brainstorm_b200._C import router as R

    rng = np.random.default_rng(3)
    mask = mask_of(rng, 3000, 32, "mixed")
    room = torch.zeros(3000 * 32 + 1, dtype=torch.int32, device="cuda")
    view = room[1:].view(3000, 32)
    view.copy_(torch.from_numpy(mask))
    idx, loads = R.generate_indices_and_loads(view)
    want = oracle.generate_indices_and_loads(mask)
    assert np.array_equal(idx.cpu().numpy(), want[0])
    assert np.array_equal(loads.cpu().numpy(), want[1])


def picks_by_key(score, k):
    """The k first of every row in descending order of the bits (NaN above everything), lower
    paths first among equals."""
    bits = score.view(np.uint32).astype(np.int64)
    key = np.where(bits & 0x80000000, 0xffffffff - bits, bits + 0x80000000)
    order = np.argsort(-key, axis=1, kind="stable")[:, :k]
    mask = np.zeros(score.shape, dtype=np.int32)
    np.put_along_axis(mask, order, 1, axis=1)
    return mask


@pytest.mark.parametrize("paths", [4, 8, 12, 20, 32, 36, 64, 68, 100, 128, 132, 200, 256])
@pytest.mark.parametrize("cells", [1, 33, 300, 5003, 40000])
def test_gate_edges(cells, paths):
    from brainstorm_b200._C import router as R

    rng = np.random.default_rng(cells + paths)
    score = rng.choice(np.array([0.0, -0.0, 0.25, 1.0, -3.0, np.inf, -np.inf,
                                 np.finfo(np.float32).min, 1e-40], dtype=np.float32),
                       (cells, paths))
    score[::2] = rng.standard_normal((score[::2].shape)).astype(np.float32)
    score[rng.random(score.shape) < 0.01] = np.nan
    dev = torch.from_numpy(score).cuda()
    for k in sorted({1, 2, min(5, paths), paths}):
        want = picks_by_key(score, k)
        idx, loads, mask = R.route_scores(dev, "topk", k, output="seat_indices", with_mask=True)
        assert np.array_equal(mask.cpu().numpy(), want), k
        want_idx, want_loads = oracle.generate_indices_and_loads(want)
        assert np.array_equal(idx.cpu().numpy(), want_idx), k
        assert np.array_equal(loads.cpu().numpy(), want_loads), k
    for residual in (-1, 0, paths - 1):
        with np.errstate(invalid="ignore"):
            want = oracle.threshold_hot_mask(score, 0.5, residual)
        got = R.route_scores(dev, "threshold", threshold=0.5, residual_path=residual)[0]
        assert np.array_equal(got.cpu().numpy(), want), residual


@pytest.mark.parametrize("paths", [4, 8, 12, 20, 32, 36, 64, 68, 100, 128, 132, 200, 256])
@pytest.mark.parametrize("cells", [1, 33, 300, 5003, 40000])
def test_gate_values(cells, paths):
    """The renormalised gates of every row shape and of partial last tiles: the same sums in the same
    order and one division; 1e-6 leaves either side a rounding of each."""
    from brainstorm_b200._C import router as R

    score = np.random.default_rng(7 * cells + paths).random((cells, paths)).astype(np.float32)
    dev = torch.from_numpy(score).cuda()
    for k in sorted({1, 2, min(5, paths), paths}):
        idx, _, gates, mask = R.route_scores(dev, "topk", k, output="seat_indices", with_gates=True,
                                             with_mask=True)
        want = oracle.renormalised_topk_score(score, k)
        np.testing.assert_allclose(gates.cpu().numpy(), want, rtol=1e-6, atol=0)
        picked = picks_by_key(score, k)
        assert np.array_equal(mask.cpu().numpy(), picked), k
        assert np.array_equal(idx.cpu().numpy(), np.cumsum(picked, axis=0) * picked), k


def test_gates_go_to_an_array_of_any_float_alignment():
    """Through the C entry point: torch's own allocations are always aligned further."""
    from brainstorm_b200 import _lib

    cells, paths, k = 1000, 20, 3
    score = torch.from_numpy(np.random.default_rng(1).standard_normal(
        (cells, paths)).astype(np.float32)).cuda()
    nbytes = _lib.query("brt_index_scratch_bytes", cells, paths)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    found = []
    for shift in range(4):
        room = torch.full((cells * paths + 8,), -7.0, device="cuda")
        out = torch.empty((cells, paths), dtype=torch.int32, device="cuda")
        loads = torch.empty(paths, dtype=torch.int32, device="cuda")
        _lib.call("brt_route_scores", score.data_ptr(), cells, paths, 0, k, 0.0, -1, 2,
                  out.data_ptr(), loads.data_ptr(), None, None, 0, 0, 0, None, None,
                  room.data_ptr() + 4 * shift, None, scratch.data_ptr(), nbytes,
                  _lib.raw_stream(score.device))
        room = room.cpu()
        end = shift + cells * paths
        assert torch.all(room[:shift] == -7) and torch.all(room[end:] == -7)
        found.append(room[shift:end].reshape(cells, paths).numpy())
    want = oracle.renormalised_topk_score(score.cpu().numpy(), k)
    for got in found:
        assert np.array_equal(got, found[0])
    assert np.abs(found[0] - want).max() <= 1e-6


def test_seats_of_an_array_that_is_only_4_byte_aligned_are_refused():
    from brainstorm_b200 import _lib

    score = torch.rand((64, 8), device="cuda")
    nbytes = _lib.query("brt_index_scratch_bytes", 64, 8)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    out = torch.zeros(64 * 8 + 4, dtype=torch.int32, device="cuda")
    loads = torch.empty(8, dtype=torch.int32, device="cuda")

    def call(scores, to, mask_to):
        return _lib.query("brt_route_scores", scores, 64, 8, 0, 1, 0.0, -1, 2, to,
                          loads.data_ptr(), None, None, 0, 0, 0, None, None, None, mask_to,
                          scratch.data_ptr(), nbytes, _lib.raw_stream(score.device))

    good, bad = out.data_ptr(), out.data_ptr() + 4
    for args in ((score.data_ptr() + 4, good, None), (score.data_ptr(), bad, None),
                 (score.data_ptr(), good, bad)):
        assert call(*args) == 4  # BRT_ERR_UNSUPPORTED, nothing is launched
    assert not out.cpu().any()


@pytest.mark.parametrize("cells,paths", [(600, 8), (1024, 8), (4096, 4), (16384, 4), (2048, 9),
                                         (4900, 256)])
def test_a_captured_scan_clears_its_words_for_every_replay(cells, paths):
    """Small masks: a graph's memset covers more than the words, within the scratch."""
    from brainstorm_b200 import _lib

    rng = np.random.default_rng(cells)
    mask = torch.zeros((cells, paths), dtype=torch.int32, device="cuda")
    out = torch.empty_like(mask)
    loads = torch.empty(paths, dtype=torch.int32, device="cuda")
    nbytes = _lib.query("brt_index_scratch_bytes", cells, paths)
    room = torch.full((nbytes + 256,), 7, dtype=torch.uint8, device="cuda")

    def scan():
        _lib.call("brt_generate_indices_and_loads", mask.data_ptr(), out.data_ptr(),
                  loads.data_ptr(), None, cells, paths, None, 0, 0, 0, 0, room.data_ptr(), nbytes,
                  _lib.raw_stream(mask.device))

    scan()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        scan()
    for density in (0.02, 0.5, 0.02):
        new = (rng.random((cells, paths)) < density).astype(np.int32)
        mask.copy_(torch.from_numpy(new))
        graph.replay()
        want = oracle.generate_indices_and_loads(new)
        assert np.array_equal(out.cpu().numpy(), want[0])
        assert np.array_equal(loads.cpu().numpy(), want[1])
    assert bool((room[nbytes:] == 7).all())


# The largest masks of these path counts whose bit words fit a CTA's shared memory on 148 SMs when
# the base seats of a few tiles at a time are all that is kept beside them.
@pytest.mark.parametrize("cells,paths", [(56756224, 4), (10381312, 16), (719872, 192),
                                         (184704, 260)])
def test_the_largest_masks_of_one_launch(cells, paths):
    from brainstorm_b200 import _lib
    from brainstorm_b200._C import router as R

    g = torch.Generator(device="cuda").manual_seed(paths)
    score = torch.rand((cells, paths), generator=g, device="cuda")
    score[cells // 3:cells // 2] = score[cells // 3:cells // 2].bernoulli_()  # dense tiles below
    best = score == score.max(dim=1, keepdim=True).values
    first = (best.cumsum(dim=1, dtype=torch.int32) == 1) & best
    del best

    def seats_of(mask):
        seats = mask.t().contiguous().cumsum(dim=1, dtype=torch.int32)
        loads = seats[:, -1].contiguous()
        return seats.t().contiguous().mul_(mask), loads

    if paths <= 256:
        want, loads = seats_of(first.to(torch.int32))
        got, got_loads = R.route_scores(score, "topk", 1, output="seat_indices")
        assert torch.equal(got, want) and torch.equal(got_loads, loads)
        del got, want
    mask = (first | (score >= 0.95)).to(torch.int32)
    del first, score
    want, loads = seats_of(mask)
    before = _lib.query("brt_kernel_launch_count")
    got, got_loads = R.generate_indices_and_loads(mask)
    assert _lib.query("brt_kernel_launch_count") == before + 1
    assert torch.equal(got, want) and torch.equal(got_loads, loads)
    del got
    limit = torch.full((paths,), cells // paths, dtype=torch.int32, device="cuda")
    prefix = torch.zeros_like(limit)
    got = R.throttle_hotmask(mask, prefix, limit)[0]
    assert torch.equal(got, ((want > 0) & (want <= limit)).to(torch.int32))
    assert torch.equal(prefix, torch.minimum(loads, limit))
