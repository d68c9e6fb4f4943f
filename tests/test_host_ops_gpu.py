"""The native host side of the router operators against the Python operators alone, over the forms
of calls that programs make: plain ones (which it takes), and other orders, strides, types,
devices and kinds of tensors (which it has to decline), errors included."""
import pytest
import torch

pytestmark = pytest.mark.gpu


class Declines:
    def __getattr__(self, name):
        return lambda *args: None


@pytest.fixture
def both(monkeypatch):
    """Run a function natively and without the native side; results and errors must agree."""
    from brainstorm_b200 import _lib

    native = _lib.host_ops()

    def outcome(make):
        try:
            return flat(make()), None
        except Exception as exc:  # noqa: BLE001 - whatever an operator raises
            return None, (type(exc), str(exc))

    def flat(value):
        if isinstance(value, torch.Tensor):
            return [value]
        return [t for v in value for t in flat(v)]

    def run(make):
        monkeypatch.setattr(_lib, "host_ops", lambda: native)
        got, error = outcome(make)
        monkeypatch.setattr(_lib, "host_ops", lambda: Declines())
        want, expected = outcome(make)
        monkeypatch.setattr(_lib, "host_ops", lambda: native)
        assert error == expected
        if want is not None:
            assert len(got) == len(want)
            for a, b in zip(got, want):
                assert a.dtype == b.dtype and a.shape == b.shape and a.device == b.device
                assert a.stride() == b.stride() and type(a) is type(b)
                assert torch.equal(a, b)
        return got, error

    return run


def masks(cells, paths):
    g = torch.Generator(device="cuda").manual_seed(cells + paths)
    m = (torch.rand((cells, paths), generator=g, device="cuda") < 0.2).to(torch.int32)
    wide = torch.zeros((cells, paths + 4), dtype=torch.int32, device="cuda")
    wide[:, :paths] = m
    return {"plain": m, "transposed": m.t().contiguous().t(), "slice": wide[:, :paths],
            "int64": m.long(), "cpu": m.cpu(), "empty": m[:0]}


@pytest.mark.parametrize("form", ["plain", "transposed", "slice", "int64", "cpu", "empty"])
@pytest.mark.parametrize("cells,paths", [(64, 32), (1000, 30), (65536, 32)])
def test_scans(both, cells, paths, form):
    from brainstorm_b200._C import router as R

    mask = masks(cells, paths)[form]
    caps = torch.tensor([3, 9], dtype=torch.int32, device="cuda")
    each = torch.full((paths,), 7, dtype=torch.int32, device="cuda")
    for args in [(mask,), (mask, caps), (mask, caps, True), (mask, each, True, True),
                 (mask, None, True), (mask, caps.long()), (mask, each[:2], True, True),
                 (mask, caps, False, False, True)]:
        both(lambda: R.generate_indices_and_loads(*args))
    limit = torch.full((paths,), 5, dtype=torch.int32, device="cuda")
    for with_mask in (False, True):
        for thr in (limit, limit.long(), limit[:-1], limit.cpu()):
            both(lambda: R.throttle_and_generate_indices(
                mask, torch.ones(paths, dtype=torch.int32, device="cuda"), thr, caps,
                with_mask=with_mask))


@pytest.mark.parametrize("cells,paths", [(64, 32), (1000, 30), (65536, 32), (5, 260)])
def test_gates(both, cells, paths):
    from brainstorm_b200._C import router as R

    score = torch.rand((cells, paths), device="cuda",
                       generator=torch.Generator(device="cuda").manual_seed(cells))
    limit = torch.full((paths,), 5, dtype=torch.int32, device="cuda")
    for s in (score, score.double(), score.t().contiguous().t(), score.cpu(), score[:0]):
        for output in ("mask", "throttled_mask", "seat_indices", "throttled_seat_indices", "none"):
            for k in (1, 2, 0, paths + 1):
                for extras in (False, True):
                    both(lambda: R.route_scores(
                        s, "topk", k, output=output, supported_capacities=limit,
                        prefix=torch.zeros(paths, dtype=torch.int32, device="cuda"),
                        throttle_capacity=limit, with_gates=extras, with_mask=extras))
        both(lambda: R.route_scores(s, "threshold", threshold=0.5, residual_path=0))
        both(lambda: R.route_scores(s, "threshold", threshold=1, residual_path=paths))
        both(lambda: R.route_scores(s, "topk", 1, output="throttled_mask"))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16, torch.float64])
@pytest.mark.parametrize("width", [(16,), (3,), (2, 5, 4)])
@pytest.mark.parametrize("cells,paths", [(64, 32), (1, 4), (65536, 33)])
def test_moves(both, cells, paths, dtype, width):
    from brainstorm_b200 import Annotator
    from brainstorm_b200._C import router as R

    mask = masks(cells, paths)["plain"]
    mask[0, 0] = 1
    x = torch.randn((cells,) + width, device="cuda").to(dtype)
    gates = torch.rand((cells, paths), device="cuda")
    indices, loads = R.generate_indices_and_loads(mask)
    slot = int(loads.max())
    strided = torch.zeros((cells, 2) + width, device="cuda", dtype=dtype)[:, 0]
    strided.copy_(x)
    for data in (x, strided, Annotator([0])(x.clone()), x.cpu(), x[:0]):
        for idx in (indices, indices.clone()):
            for lo in (loads, loads.cpu(), loads.long()):
                for gate in (None, gates.to(dtype), gates.half()):
                    for padded, mpl in ((True, slot), (True, 0), (False, 0), (True, -1)):
                        if data.is_cuda and data.size(0) and mpl < 0:
                            continue  # a slot of no rows is not defined
                        both(lambda: R.dispatch_with_indices_and_loads(
                            data, idx, lo, gate, False, None, padded, mpl))
    if dtype == torch.float64 or (dtype == torch.float16 and width == (3,)):
        return  # refused above, natively and not
    (rows,) = R.dispatch_with_indices_and_loads(x, indices, loads, None, False, None, True, slot)
    base = torch.randn((cells,) + width, device="cuda").to(dtype)
    for data in (rows, rows.cpu(), torch.cat([rows, rows])[::2] * 0 + rows):
        for lo in (loads, loads.cpu(), loads.long(), None):
            for gate in (None, gates, gates.to(dtype), gates.double(), gates.t().contiguous().t()):
                for out in (False, True):
                    both(lambda: R.combine_with_indices_and_loads(
                        data, indices, lo, gate, base.clone() if out else None, True))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        both(lambda: R.combine_with_indices_and_loads(rows, indices, loads, gates, None, True))
        both(lambda: R.dispatch_with_indices_and_loads(x, indices, loads, None, False, None, True,
                                                       slot))
    side.synchronize()
    with torch.inference_mode():
        both(lambda: R.generate_indices_and_loads(mask))
        idx, lo = R.generate_indices_and_loads(mask)
        both(lambda: R.dispatch_with_indices_and_loads(x, idx, lo, None, False, None, True, slot))
        both(lambda: R.combine_with_indices_and_loads(rows, idx, lo, gates, None, True))


def test_residual_is_returned_itself_and_the_note_travels():
    from brainstorm_b200._C import router as R

    indices, loads = R.generate_indices_and_loads(masks(65536, 32)["plain"])
    assert getattr(indices, R._DENSE).data_ptr() == loads.data_ptr() + 4 * 32
    rows = torch.randn((int(loads.sum()), 8), device="cuda")
    base = torch.randn((65536, 8), device="cuda")
    (out,) = R.combine_with_indices_and_loads(rows, indices, loads, None, base)
    assert out is base


@pytest.mark.parametrize("paths", [1, 30])
def test_packed_dispatch_takes_loads_of_any_shape(paths):
    from brainstorm_b200._C import router as R

    indices, loads = R.generate_indices_and_loads(masks(500, paths)["plain"])
    x = torch.randn((500, 64), device="cuda")
    (want,) = R.dispatch_with_indices_and_loads(x, indices, loads)
    shapes = [(1, paths), (paths, 1)] + ([()] if paths == 1 else [])
    for shape in shapes:
        (got,) = R.dispatch_with_indices_and_loads(x, indices, loads.reshape(shape))
        assert torch.equal(got, want)


def test_other_threads_run_while_a_launch_waits():
    """With the stream busy and its queue full an operator waits; the process must not."""
    import threading
    import time

    from brainstorm_b200._C import router as R

    mask = masks(64, 32)["plain"]
    indices, loads = R.generate_indices_and_loads(mask)
    x = torch.randn((64, 16), device="cuda")
    slot = int(loads.max())

    def step():
        R.generate_indices_and_loads(mask)
        (rows,) = R.dispatch_with_indices_and_loads(x, indices, loads, None, False, None, True,
                                                    slot)
        R.combine_with_indices_and_loads(rows, indices, loads, None, None, True)
        R.route_scores(x, "topk", 1, output="seat_indices")

    step()
    torch.cuda.synchronize()
    ticks, stop = [], threading.Event()

    def tick():
        while not stop.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.001)

    thread = threading.Thread(target=tick)
    thread.start()
    longest = 0.0
    try:
        torch.cuda._sleep(2_000_000_000)  # about a second
        begin = time.perf_counter()
        while time.perf_counter() - begin < 2.0:  # more launches than any queue holds
            at = time.perf_counter()
            step()
            longest = max(longest, time.perf_counter() - at)
            if longest > 0.3:
                break
    finally:
        stop.set()
        thread.join()
    torch.cuda.synchronize()
    assert longest > 0.3, "no launch had to wait"
    gaps = [b - a for a, b in zip(ticks, ticks[1:])]
    assert max(gaps) < 0.5 * longest


def test_running_out_of_memory_keeps_its_kind():
    """What a program catches to free something and try again."""
    from brainstorm_b200._C import router as R

    cells = torch.arange(1 << 18, device="cuda")
    mask = torch.zeros((1 << 18, 64), dtype=torch.int32, device="cuda")
    mask[cells, cells % 64] = 1  # 4096 cells for every path
    score = torch.rand((1 << 18, 64), device="cuda")
    limit = torch.full((64,), 5, dtype=torch.int32, device="cuda")
    indices, loads = R.generate_indices_and_loads(mask)
    x = torch.randn((1 << 18, 64), device="cuda")
    slot = 1 << 18
    rows = torch.randn((64 * 4096, 64), device="cuda")
    calls = [
        lambda: R.generate_indices_and_loads(mask),
        lambda: R.throttle_and_generate_indices(mask, torch.zeros_like(limit), limit),
        lambda: R.route_scores(score, "topk", 1, output="seat_indices", with_gates=True),
        lambda: R.dispatch_with_indices_and_loads(x, indices, loads, None, False, None, True, slot),
        lambda: R.combine_with_indices_and_loads(rows, indices, loads, None, None, True),
    ]
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    try:  # nothing beyond what is allocated now
        torch.cuda.set_per_process_memory_fraction(
            torch.cuda.memory_reserved() / torch.cuda.mem_get_info()[1])
        for call in calls:
            with pytest.raises(torch.OutOfMemoryError):
                held = []
                for _ in range(8):  # what the reserved blocks still have room for
                    held.append(call())
            held = None
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    for call in calls[:3]:
        call()
    torch.cuda.synchronize()
