"""The work that users of this framework have it do, as measurable cases.

A case is a dict of plain values; its ``op`` names the kind of program it stands for:

``gate``     gate scores -> seat indices, loads (and gates, mask), ``route_scores``
``step``     route mask -> indices -> dispatch -> identity expert -> combine, through the
             ``_C.router`` operators, as a layer with experts of its own drives them
``samples``  ``ScatterRouter("threshold", "dispatch")`` -> ``GatherRouter("combine")`` over whole
             samples: branches of a dynamic-routing network, merged by tag
``experts``  one grouped expert linear layer over a dispatched buffer
``layer``    a whole mixture-of-experts feed-forward layer: ``ScatterRouter`` with its gate,
             two grouped expert layers, weighted ``GatherRouter``

Sizes are those of the benchmark workloads and of the tests, or generic ones around them.
"""
import math

import numpy as np
import torch

from brainstorm_b200 import Annotator
from brainstorm_b200._C import expert, router
from brainstorm_b200.router import GatherRouter, ScatterRouter
from brainstorm_b200.runtime.grid_tensor import init_grid_tensor, to_torch_tensor

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


def _size(case):
    return 4 if case["dtype"] == "f32" else 2


# ------------------------------------------------------------------------------------- cases
def listed():
    return [
        # decode: a few dozen tokens, where latency and the number of launches are the cost
        dict(name="step_decode_bf16", op="step", cells=64, width=1024, paths=32, k=2,
             dtype="bf16", bias="normal", cap=1.0, padded=True, weigh="combine", residual=False),
        # the small top-1 routing step of the benchmark: fp32, capacity 1.25, weighted combine
        # into the residual stream
        dict(name="step_switch8_f32", op="step", cells=4096, width=768, paths=8, k=1,
             dtype="f32", bias="none", cap=1.25, padded=True, weigh="combine", residual=True),
        # the benchmark's headline step: 8 x 4096 tokens, 32 experts, top-2, capacity 1.0
        dict(name="step_top2_bf16", op="step", cells=32768, width=1024, paths=32, k=2,
             dtype="bf16", bias="normal", cap=1.0, padded=True, weigh="combine", residual=False),
        # 128 experts with strongly skewed loads: most of the padded output stays empty
        dict(name="step_switch128_bf16", op="step", cells=262144, width=768, paths=128, k=1,
             dtype="bf16", bias="zipf", cap=2.0, padded=True, weigh="combine", residual=False),
        # one rank's share of the expert-parallel workload: no capacity, packed rows whose
        # number the host reads
        dict(name="step_packed_bf16", op="step", cells=65536, width=2048, paths=64, k=2,
             dtype="bf16", bias="normal", cap=0.0, padded=False, weigh="combine",
             residual=False),
        # ragged everything: odd number of cells, rows that are no multiple of 16 bytes, a
        # number of paths that is no multiple of 4, gates applied at dispatch
        dict(name="step_ragged_f16", op="step", cells=9001, width=1002, paths=30, k=2,
             dtype="f16", bias="normal", cap=0.0, padded=False, weigh="dispatch",
             residual=False),
        # scores of a top-2 layer to indices, renormalised gates and hot mask in one call
        dict(name="gate_top2_32", op="gate", cells=32768, paths=32, k=2, bias="normal", cap=0.0,
             extras=True),
        # the largest gate: scores over 128 experts to throttled seat indices
        dict(name="gate_switch128", op="gate", cells=262144, paths=128, k=1, bias="zipf",
             cap=2.0, extras=False),
        # convolutional samples to any subset of 8 branches (the first for those that no gate
        # opens for) and back, through the routers
        dict(name="samples_threshold_f32", op="samples", cells=64, width=256 * 56 * 56, paths=8,
             dtype="f32", threshold=0.5),
        # expert layer over many experts of very different loads (partial tiles everywhere)
        dict(name="experts_skewed_bf16", op="experts", rows=36343, paths=128, inner=768,
             outer=3072, relu=True, bias="zipf", dtype="bf16"),
        # a decode batch through the whole layer: reading the experts' weights is the cost
        dict(name="layer_decode_bf16", op="layer", cells=64, width=1024, hidden=4096, paths=32,
             k=2, bias="normal", cap=4.0, dtype="bf16"),
        # a prefill batch through the whole layer: the tensor cores are the cost
        dict(name="layer_prefill_bf16", op="layer", cells=16384, width=1024, hidden=4096,
             paths=32, k=2, bias="normal", cap=1.5, dtype="bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_any(rng):
    op = rng.choice(["step", "step", "step", "gate", "samples", "experts", "layer"])
    bias = rng.choice(["none", "normal", "zipf"])
    if op == "gate":
        paths = 4 * _log_int(rng, 1, 64)
        k = rng.choice([1, 1, 2, min(4, paths)])
        return dict(op=op, cells=_log_int(rng, 16, 262144), paths=paths, k=k, bias=bias,
                    cap=rng.choice([0.0, 1.0, 2.0]), extras=rng.random() < 0.5)
    if op == "step":
        paths = rng.choice([4 * _log_int(rng, 1, 32), _log_int(rng, 3, 64)])
        dtype = rng.choice(["bf16", "bf16", "f16", "f32"])
        width = rng.choice([64 * _log_int(rng, 1, 32), 2 * _log_int(rng, 16, 1024)])
        padded = rng.random() < 0.5
        return dict(op=op, cells=_log_int(rng, 16, 262144), width=width, paths=paths,
                    k=rng.choice([1, 2, 2, min(4, paths)]), dtype=dtype, bias=bias,
                    cap=rng.choice([1.0, 1.25, 2.0]) if padded else 0.0, padded=padded,
                    weigh=rng.choice(["combine", "combine", "dispatch"]),
                    residual=rng.random() < 0.25)
    if op == "samples":
        return dict(op=op, cells=_log_int(rng, 8, 96),
                    width=rng.choice([64, 128, 256]) * rng.choice([7, 14, 28, 56]) ** 2,
                    paths=rng.choice([2, 4, 6, 8, 16]), dtype="f32",
                    threshold=rng.choice([0.4, 0.5, 0.7]))
    if op == "experts":
        return dict(op=op, rows=_log_int(rng, 32, 65536), paths=_log_int(rng, 2, 128),
                    inner=64 * _log_int(rng, 2, 32), outer=128 * _log_int(rng, 2, 32),
                    relu=rng.random() < 0.5, bias=bias, dtype="bf16")
    width = 128 * _log_int(rng, 2, 12)
    return dict(op=op, cells=_log_int(rng, 16, 16384), width=width,
                hidden=width * rng.choice([2, 4]), paths=4 * _log_int(rng, 1, 16),
                k=rng.choice([1, 2]), bias=bias, cap=rng.choice([1.0, 1.5, 4.0]), dtype="bf16")


def draw(rng):
    """One more case of the ranges above, none dearer than the largest listed one of its op."""
    limits = {}
    for case in listed():
        w = work(case)
        old = limits.get(case["op"], {"bytes": 0, "flops": 0})
        limits[case["op"]] = {key: max(old[key], w[key]) for key in w}
    while True:
        case = _draw_any(rng)
        w, limit = work(case), limits[case["op"]]
        if w["bytes"] <= limit["bytes"] and w["flops"] <= limit["flops"]:
            return case


# ------------------------------------------------------------------------------------ inputs
def _capacity(case):
    """Rows a path may hold: ``k * ceil(factor * cells / paths)``; 0 without a capacity."""
    if not case["cap"]:
        return 0
    return max(1, case["k"] * math.ceil(case["cap"] * case["cells"] / case["paths"]))


def _path_bias(kind, paths, normal, ranks):
    if kind == "normal":
        return 0.5 * normal
    if kind == "zipf":
        share = (ranks + 1.0) ** -1.1
        return 4.0 * share / share.max()
    return 0.0 * normal


def _expected_kept(case):
    """Routes that the capacity keeps, and cells with at least one of them, for typical loads
    of this bias."""
    rng = np.random.default_rng(0)
    paths, k, cells = case["paths"], case["k"], case["cells"]
    bias = _path_bias(case["bias"], paths, rng.standard_normal(paths), rng.permutation(paths))
    logits = rng.standard_normal((4096, paths)) + bias
    picks = np.argsort(-logits, axis=1)[:, :k]
    loads = np.bincount(picks.reshape(-1), minlength=paths) * (cells / 4096.0)
    cap = _capacity(case)
    keep = np.minimum(1.0, cap / np.maximum(loads, 1e-9)) if cap else np.ones(paths)
    kept = float((loads * keep).sum())
    routed = float((1.0 - np.prod(1.0 - keep[picks], axis=1)).mean() * cells)
    return kept, routed


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _scores(case, g):
    cells, paths = case["cells"], case["paths"]
    normal = torch.randn(paths, generator=g, device="cuda")
    ranks = torch.randperm(paths, generator=g, device="cuda").float()
    logits = torch.randn((cells, paths), generator=g, device="cuda")
    logits += _path_bias(case["bias"], paths, normal, ranks)
    return torch.softmax(logits, dim=1)


def _picks(score, k):
    """The k best paths of every cell; equal scores go to the lower path."""
    return torch.sort(score, dim=1, descending=True, stable=True).indices[:, :k]


def _mask(score, k):
    mask = torch.zeros(score.shape, dtype=torch.int32, device="cuda")
    return mask.scatter_(1, _picks(score, k), 1)


def _renormalised(score, mask):
    kept = score * mask
    return kept / kept.sum(dim=1, keepdim=True).clamp_min(torch.finfo(torch.float32).eps)


def _loads(case, g):
    """Rows per expert that add up to ``rows``, as the bias of the gate spreads them."""
    paths = case["paths"]
    normal = torch.randn(paths, generator=g, device="cuda")
    ranks = torch.randperm(paths, generator=g, device="cuda").float()
    share = torch.softmax(_path_bias(case["bias"], paths, 2.0 * normal, ranks).double(), dim=0)
    loads = (share * case["rows"]).to(torch.int32)
    loads[int(torch.argmax(loads))] += case["rows"] - int(loads.sum())
    return loads


def prepare(case, seed):
    g = _generator(seed)
    op = case["op"]
    state = {"case": case}
    if op == "gate":
        state["score"] = _scores(case, g)
        if case["cap"]:
            state["limit"] = torch.full((case["paths"],), _capacity(case), dtype=torch.int32,
                                        device="cuda")
    elif op == "step":
        dtype = DTYPES[case["dtype"]]
        score = _scores(case, g)
        state["mask"] = _mask(score, case["k"])
        gates = score if case["k"] == 1 else _renormalised(score, state["mask"])
        state["gates"] = gates.to(dtype) if case["weigh"] == "dispatch" else gates
        state["x"] = torch.randn((case["cells"], case["width"]), generator=g,
                                 device="cuda").to(dtype)
        if case["cap"]:
            state["limit"] = torch.full((case["paths"],), _capacity(case), dtype=torch.int32,
                                        device="cuda")
        if case["residual"]:
            state["residual"] = torch.randn((case["cells"], case["width"]), generator=g,
                                            device="cuda").to(dtype)
    elif op == "samples":
        state["x"] = torch.randn((case["cells"], case["width"]), generator=g, device="cuda")
        state["score"] = torch.sigmoid(torch.randn((case["cells"], case["paths"]), generator=g,
                                                   device="cuda"))
        state["annotate"] = Annotator([0])
        state["scatter"] = ScatterRouter(protocol_type="threshold", fabric_type="dispatch",
                                         protocol_kwargs={"threshold": case["threshold"],
                                                          "residual_path": 0})
        state["gather"] = GatherRouter(fabric_type="combine")
    elif op == "experts":
        state["loads"] = _loads(case, g)
        state["rows"] = (0.5 * torch.randn((case["rows"], case["inner"]), generator=g,
                                           device="cuda")).bfloat16()
        state["weights"] = (torch.randn((case["paths"], case["outer"], case["inner"]),
                                        generator=g, device="cuda")
                            / case["inner"] ** 0.5).bfloat16()
    else:
        cap = _capacity(case)
        state["x"] = torch.randn((case["cells"], case["width"]), generator=g,
                                 device="cuda").bfloat16()
        state["score"] = _scores(case, g)
        state["gates"] = _renormalised(state["score"], _mask(state["score"], case["k"]))
        for name, outer, inner in (("w1", case["hidden"], case["width"]),
                                   ("w2", case["width"], case["hidden"])):
            state[name] = (torch.randn((case["paths"], outer, inner), generator=g, device="cuda")
                           / inner ** 0.5).bfloat16()
        state["cap"] = cap
        state["scatter"] = ScatterRouter(
            protocol_type="topk", fabric_type="fused_dispatch",
            protocol_kwargs={"top_k": case["k"]},
            fabric_kwargs={"supported_capacities": [cap], "max_path_padding": True,
                           "max_path_load": cap}).cuda()
        state["gather"] = GatherRouter(
            fabric_type="fused_combine",
            fabric_kwargs={"transform": True, "max_path_padding": True})
    return state


# -------------------------------------------------------------------------------------- runs
def run(state):
    return _RUN[state["case"]["op"]](state)


def _run_gate(state):
    case, score = state["case"], state["score"]
    if case["cap"]:
        prefix = torch.zeros(case["paths"], dtype=torch.int32, device=score.device)
        return router.route_scores(
            score, "topk", case["k"], output="throttled_seat_indices", prefix=prefix,
            throttle_capacity=state["limit"], supported_capacities=state["limit"],
            with_gates=case["extras"], with_mask=case["extras"])
    return router.route_scores(score, "topk", case["k"], output="seat_indices",
                               with_gates=case["extras"], with_mask=case["extras"])


def _run_step(state):
    case, mask = state["case"], state["mask"]
    padded, cap = case["padded"], _capacity(case)
    if cap:
        prefix = torch.zeros(case["paths"], dtype=torch.int32, device=mask.device)
        indices, loads, _ = router.throttle_and_generate_indices(mask, prefix, state["limit"],
                                                                 state["limit"])
    else:
        indices, loads = router.generate_indices_and_loads(mask)
    at_dispatch = case["weigh"] == "dispatch"
    (rows,) = router.dispatch_with_indices_and_loads(
        state["x"], indices, loads, state["gates"] if at_dispatch else None, False, None, padded,
        cap)
    (out,) = router.combine_with_indices_and_loads(
        rows, indices, loads, None if at_dispatch else state["gates"], state.get("residual"),
        padded)
    return indices, loads, rows, out


def _run_samples(state):
    flows = state["scatter"](state["annotate"](state["x"]), state["score"])
    merged = state["gather"](flows)
    return to_torch_tensor(merged), merged.tag


def _run_experts(state):
    return expert.grouped_expert_linear(state["rows"], state["weights"], state["loads"],
                                        relu=state["case"]["relu"])


def _run_layer(state):
    cap = state["cap"]
    rows, tags, loads, extra = to_torch_tensor(state["scatter"](state["x"], state["score"]),
                                               retrieve_attr=True)
    hidden = expert.grouped_expert_linear(rows, state["w1"], loads[-1], True, cap, relu=True)
    outs = expert.grouped_expert_linear(hidden, state["w2"], loads[-1], True, cap)
    out = state["gather"](init_grid_tensor(outs, tags, loads, extra), score=state["gates"])
    return to_torch_tensor(out)


_RUN = {"gate": _run_gate, "step": _run_step, "samples": _run_samples, "experts": _run_experts,
        "layer": _run_layer}


# -------------------------------------------------------------------------------------- work
def work(case):
    """Bytes (every input read once, every output written once, nothing in between two calls
    that a layer could not keep) and operations of one pass."""
    op = case["op"]
    if op == "gate":
        arrays = 2 + (2 if case["extras"] else 0)
        return {"bytes": 4 * case["cells"] * case["paths"] * arrays, "flops": 0}
    if op == "step":
        row = case["width"] * _size(case)
        scan = 4 * case["cells"] * case["paths"]
        kept, routed = _expected_kept(case)
        total = case["paths"] * _capacity(case) if case["padded"] else kept
        # scan: mask in, indices out; dispatch: cells and indices in, rows out; combine: kept
        # rows, indices and gates in, cells out
        gates = scan if case["weigh"] == "combine" else scan * _size(case) // 4
        bytes_ = 4 * scan + gates + int((routed + total + kept + case["cells"]) * row)
        return {"bytes": bytes_, "flops": 2 * int(kept) * case["width"]}
    if op == "samples":
        share = 0.5 * math.erfc(math.log(case["threshold"] / (1 - case["threshold"]))
                                / math.sqrt(2.0))
        cells, paths = case["cells"], case["paths"]
        kept = cells * (paths * share + (1.0 - share) ** paths)
        return {"bytes": int((2 * cells + 2 * kept) * case["width"] * 4),
                "flops": int(kept * case["width"])}
    if op == "experts":
        rows, inner, outer = case["rows"], case["inner"], case["outer"]
        return {"bytes": 2 * (rows * (inner + outer) + case["paths"] * inner * outer),
                "flops": 2 * rows * inner * outer}
    kept, _ = _expected_kept(case)
    width, hidden, paths = case["width"], case["hidden"], case["paths"]
    weights = 2 * 2 * min(paths, case["cells"] * case["k"]) * width * hidden
    return {"bytes": int(weights + 2 * 2 * case["cells"] * width + 8 * case["cells"] * paths),
            "flops": int(4 * kept * width * hidden)}


def tolerance(case):
    """Whole values are exact everywhere.  fp32: sums of a few terms in any order.  16 bits: fp32
    sums in another order, whose rounding to the type falls to the other side now and then."""
    op = case["op"]
    if op == "layer":
        return {"rel": 2e-3}
    if op == "experts":
        return {"rel": 2.5e-4}
    if op == "step" and case["dtype"] != "f32":
        return {"rel": 1e-4}
    return {"rel": 5e-7}


# ------------------------------------------------------------------------------------- exact
def _seats(mask):
    return mask.long().cumsum(dim=0) * mask.long()


def _throttle(mask, cap):
    seats = _seats(mask)
    return seats * (seats <= cap) if cap else seats


def exact(case, seed):
    state = prepare(case, seed)
    return _EXACT[case["op"]](case, state)


def _exact_gate(case, state):
    score, cap = state["score"], _capacity(case)
    mask = _mask(score, case["k"])
    seats = _throttle(mask, cap)
    loads = (seats > 0).sum(dim=0)
    out = (seats, loads)
    if cap:
        out += (torch.clamp_max(mask.long().sum(dim=0), cap),)
    if case["extras"]:
        kept = score.double() * mask
        denom = kept.sum(dim=1, keepdim=True).clamp_min(torch.finfo(torch.float32).eps)
        out += (kept / denom, (seats > 0).long())
    return out


def _row_bases(loads, case, cap):
    if case.get("padded", True):
        return torch.arange(case["paths"], device="cuda") * cap
    return loads.cumsum(dim=0) - loads


def _exact_step(case, state):
    cap = _capacity(case)
    seats = _throttle(state["mask"], cap)
    loads = (seats > 0).sum(dim=0)
    cell, path = (seats > 0).nonzero(as_tuple=True)
    slot = _row_bases(loads, case, cap)[path] + seats[cell, path] - 1
    total = case["paths"] * cap if case["padded"] else int(loads.sum())
    moved = state["x"][cell].double()
    weight = state["gates"][cell, path].double()[:, None]
    rows = torch.zeros((total, case["width"]), dtype=torch.float64, device="cuda")
    rows[slot] = moved * weight if case["weigh"] == "dispatch" else moved
    moved *= weight
    if case["residual"]:
        out = state["residual"].double()
        out[cell] = 0.0
    else:
        out = torch.zeros((case["cells"], case["width"]), dtype=torch.float64, device="cuda")
    out.index_add_(0, cell, moved)
    return seats, loads, rows, out


def _exact_samples(case, state):
    times = (state["score"] > case["threshold"]).sum(dim=1).clamp_min(1)
    tags = torch.arange(1, case["cells"] + 1, device="cuda")
    return state["x"].double() * times.double()[:, None], tags


def _exact_experts(case, state):
    out = torch.empty((case["rows"], case["outer"]), dtype=torch.float64, device="cuda")
    start = 0
    for e, load in enumerate(state["loads"].tolist()):
        part = out[start:start + load]
        torch.mm(state["rows"][start:start + load].double(), state["weights"][e].double().T,
                 out=part)
        start += load
    return out.relu_() if case["relu"] else out


def _exact_layer(case, state):
    seats = _throttle(_mask(state["score"], case["k"]), state["cap"])
    out = torch.zeros((case["cells"], case["width"]), dtype=torch.float64, device="cuda")
    for e in range(case["paths"]):
        cells = seats[:, e].nonzero()[:, 0]
        if cells.numel():
            hidden = (state["x"][cells].double() @ state["w1"][e].double().T).relu_()
            rows = hidden @ state["w2"][e].double().T
            out.index_add_(0, cells, rows * state["gates"][cells, e].double()[:, None])
    return out


_EXACT = {"gate": _exact_gate, "step": _exact_step, "samples": _exact_samples,
          "experts": _exact_experts, "layer": _exact_layer}
