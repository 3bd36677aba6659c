"""Performance cases of nanoep_b200: what a program that serves or trains a mixture-of-experts model has it do.

Three kinds of case, all on one GPU:

``exchange``  one process of one GPU: ``CudaBuffer.dispatch`` followed by ``CudaBuffer.combine`` (identity experts).
``group``     a whole expert-parallel group as logical peers of one GPU (``EmulatedGroup``): the kernels that a group of
              several GPUs runs, with every cross-rank step in them.
``layer``     ``ExpertParallelMoE.forward``: dispatch, SwiGLU experts on the tensor cores, combine.

``fresh`` means that routing is new in every pass (forward); a cached exchange reuses the routing handle of an earlier
dispatch, as the backward pass and repeated exchanges do.  Expert-major receive rows have no fixed order inside one
expert's range, so expert-major cases return what has one: the combined rows, the gate weights and the counts.  A compact
exchange returns the received rows and their metadata as well (in a group their number depends on the routing).
"""

from __future__ import annotations

import math
from datetime import timedelta

import torch
import torch.distributed as dist

from nanoep_b200 import CudaBuffer, EmulatedGroup, EPConfig
from nanoep_b200.models.moe_layer import ExpertParallelMoE

# ----------------------------------------------------------------------------------------------- cases


def _exchange(name, tokens, capacity, hidden, experts, topk, *, expand, alignment=1, zero_padding=False, routing="balanced", cached=False,
              return_weights=False, bias=False, reduce_per_rank=False, async_op=False):
    return dict(name=name, kind="exchange", tokens=tokens, capacity=capacity, hidden=hidden, experts=experts, topk=topk, expand=expand,
                alignment=alignment, zero_padding=zero_padding, routing=routing, cached=cached, return_weights=return_weights, bias=bias,
                reduce_per_rank=reduce_per_rank, async_op=async_op)


def _group(name, ranks, tokens, capacity, hidden, experts, topk, *, expand, alignment=1, zero_padding=False, routing="balanced", cached=False,
           return_weights=False, bias=False, reduce_per_rank=False):
    return dict(name=name, kind="group", ranks=ranks, tokens=tokens, capacity=capacity, hidden=hidden, experts=experts, topk=topk, expand=expand,
                alignment=alignment, zero_padding=zero_padding, routing=routing, cached=cached, return_weights=return_weights, bias=bias,
                reduce_per_rank=reduce_per_rank)


def _layer(name, tokens, capacity, hidden, inner, experts, topk, *, routing="balanced", fuse_combine=True, bias=False):
    return dict(name=name, kind="layer", tokens=tokens, capacity=capacity, hidden=hidden, inner=inner, experts=experts, topk=topk, routing=routing,
                fuse_combine=fuse_combine, bias=bias)


def listed():
    return [
        # One token of one sequence: the latency of a single decode step's exchange.
        _exchange("decode-1", 1, 128, 7168, 256, 8, expand=True, routing="uniform"),
        # A decode batch in a buffer that is sized for prefill, as a server keeps one buffer for both.
        _exchange("decode-32", 32, 4096, 7168, 256, 8, expand=True, routing="uniform"),
        # The reference's published figure (256 tokens, hidden 4096, top-8), in the compact layout, with a shared expert's
        # output as the bias and the gate weights on the way back.
        _exchange("small-compact-256", 256, 256, 4096, 256, 8, expand=False, routing="uniform", return_weights=True, bias=True),
        # Training or prefill at the DeepSeek-V3 shape: fresh routing in every step, layout ready for a grouped GEMM.
        _exchange("prefill-4096", 4096, 4096, 7168, 256, 8, expand=True, alignment=128, zero_padding=True),
        # Backward of the same layer on a ragged batch: gradients take the forward's routing, gate gradients come back.
        _exchange("backward-3001", 3001, 4096, 7168, 256, 8, expand=True, alignment=128, zero_padding=True, cached=True, return_weights=True),
        # Skewed routing with masked choices, compact layout, one cached handle for many asynchronous exchanges.
        _exchange("skewed-8192", 8192, 8192, 4096, 64, 6, expand=False, routing="zipf", cached=True, async_op=True),
        # A decode batch across a group of eight: all cross-rank steps at a size where their latency is the cost.
        _group("group-decode-16", 8, 16, 128, 7168, 256, 8, expand=True, routing="uniform"),
        # A prefill chunk across a group of eight, rows padded for a grouped GEMM.
        _group("group-prefill-512", 8, 512, 512, 7168, 256, 8, expand=True, alignment=128, zero_padding=True),
        # A compact exchange across a group of four with skewed routing, the forward and its gate weights.
        _group("group-skewed-1000", 4, 1000, 1024, 4096, 64, 6, expand=False, routing="zipf", return_weights=True),
        # One GPU's share of an expert layer (32 of 256 experts at the DeepSeek-V3 shape) in a decode step: weight traffic.
        _layer("layer-decode-64", 64, 128, 7168, 2048, 32, 8),
        # A mid-sized batch with uneven experts, through the separate combine, with a shared expert's output as the bias.
        _layer("layer-skewed-777", 777, 1024, 4096, 1536, 32, 6, routing="zipf", fuse_combine=False, bias=True),
        # The full layer in prefill or training: tensor-core bound.
        _layer("layer-prefill-4096", 4096, 4096, 7168, 2048, 32, 8),
    ]


def _log_int(rng, low, high):
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    """One more case of the same ranges; never more work than the largest listed case of its kind."""
    kind = rng.choice(["exchange", "exchange", "group", "layer"])
    routing = rng.choice(["balanced", "uniform", "zipf"])
    if kind == "layer":
        hidden, inner = 256 * rng.randint(4, 28), 128 * rng.randint(4, 16)
        experts, topk = rng.choice([8, 16, 24, 32]), rng.randint(2, 8)
        tokens = _log_int(rng, 1, 4096)
        case = _layer("", tokens, max(tokens, rng.choice([1, 128, 1024])), hidden, inner, experts, topk, routing=routing,
                      fuse_combine=rng.random() < 0.7, bias=rng.random() < 0.3)
        del case["name"]
        return case
    expand = rng.random() < 0.6
    options = dict(expand=expand, routing=routing, cached=rng.random() < 0.4, return_weights=rng.random() < 0.5, bias=rng.random() < 0.3,
                   reduce_per_rank=rng.random() < 0.3)
    if expand:
        options["alignment"] = rng.choice([1, 8, 16, 128])
        options["zero_padding"] = rng.random() < 0.5
    if kind == "exchange":
        hidden, topk = 256 * rng.randint(2, 28), rng.randint(1, 8)
        experts = rng.choice([8, 32, 60, 64, 128, 160, 256])
        tokens = _log_int(rng, 1, min(8192, 4096 * 8 * 7168 // (hidden * topk)))
        case = _exchange("", tokens, max(tokens, rng.choice([1, 256, 4096])), hidden, experts, topk, async_op=rng.random() < 0.3, **options)
    else:
        ranks, topk = rng.choice([2, 4, 8]), rng.randint(1, 8)
        hidden = 256 * rng.randint(2, 28)
        experts = ranks * rng.choice([2, 8, 16, 20, 32])
        topk = min(topk, experts)
        tokens = _log_int(rng, 1, min(1024, 512 * 8 * 8 * 7168 // (hidden * topk * ranks)))
        case = _group("", ranks, tokens, max(tokens, rng.choice([1, 128, 512])), hidden, experts, topk, **options)
    del case["name"]
    return case


# ----------------------------------------------------------------------------------------------- inputs
# A program opens one buffer per configuration and keeps it; two are kept here, so that a run over many
# configurations does not fill the card.
_open: dict[tuple, object] = {}


def _buffer(case):
    key = (case["kind"] == "group", case.get("ranks", 1), case["capacity"], case["hidden"], case["experts"], case["topk"],
           case.get("reduce_per_rank", False))
    if key in _open:
        _open[key] = _open.pop(key)
        return _open[key]
    while len(_open) >= 2:
        _open.pop(next(iter(_open))).close()
    config = EPConfig(num_experts=case["experts"], num_topk=case["topk"], hidden=case["hidden"], num_max_tokens_per_rank=case["capacity"])
    if case["kind"] == "group":
        buf = EmulatedGroup(case["ranks"], config, allow_multiple_reduction=case["reduce_per_rank"])
    else:
        if not dist.is_initialized():
            dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1, timeout=timedelta(seconds=60))
        buf = CudaBuffer(dist.group.WORLD, config, allow_multiple_reduction=case.get("reduce_per_rank", False))
    _open[key] = buf
    return buf


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _routing(case, gen):
    """Distinct experts per token and gate weights that sum to one: a router's softmax top-k (balanced), uniformly random
    experts, or experts of Zipf(1.2) popularity with a tenth of the choices after the first masked."""
    tokens, experts, topk = case["tokens"], case["experts"], case["topk"]
    if case["routing"] == "balanced":
        w, idx = torch.softmax(torch.randn(tokens, experts, generator=gen, device="cuda"), dim=-1).topk(topk, dim=-1)
        return idx, w / w.sum(-1, keepdim=True)
    if case["routing"] == "uniform":
        idx = torch.rand(tokens, experts, generator=gen, device="cuda").topk(topk, dim=-1).indices
        return idx, torch.full((tokens, topk), 1.0 / topk, device="cuda")
    popularity = torch.arange(1, experts + 1, device="cuda").float().pow(-1.2)[torch.randperm(experts, generator=gen, device="cuda")]
    noise = torch.rand(tokens, experts, generator=gen, device="cuda").clamp_(1e-12, 1 - 1e-7).log().neg().log().neg()
    idx = (popularity.log() + noise).topk(topk, dim=-1).indices
    w = torch.rand(tokens, topk, generator=gen, device="cuda") + 0.1
    drop = torch.rand(tokens, topk, generator=gen, device="cuda") < 0.1
    drop[:, 0] = False
    idx = idx.masked_fill(drop, -1)
    return idx, w / w.sum(-1, keepdim=True)


def _normal(gen, *shape, scale=1.0):
    return (torch.randn(*shape, generator=gen, device="cuda") * scale).to(torch.bfloat16)


def _weights(gen, *shape, scale):
    """Like ``_normal``, one expert at a time: the fp32 values of all experts would not fit beside three states."""
    out = torch.empty(shape, dtype=torch.bfloat16, device="cuda")
    for e in range(shape[0]):
        out[e] = torch.randn(*shape[1:], generator=gen, device="cuda") * scale
    return out


def prepare(case, seed):
    gen = _generator(seed)
    buf = _buffer(case)
    state = {"case": case, "buffer": buf}
    ranks = case.get("ranks", 1)
    xs, idxs, ws, biases = [], [], [], []
    for _ in range(ranks):
        idx, w = _routing(case, gen)
        xs.append(_normal(gen, case["tokens"], case["hidden"]))
        idxs.append(idx)
        ws.append(w)
        biases.append(_normal(gen, case["tokens"], case["hidden"]) if case["bias"] else None)
    if case["kind"] == "layer":
        hidden, inner, experts = case["hidden"], case["inner"], case["experts"]
        state["layer"] = ExpertParallelMoE(buf, _weights(gen, experts, 2 * inner, hidden, scale=0.02),
                                           _weights(gen, experts, hidden, inner, scale=0.02), fuse_combine=case["fuse_combine"])
    elif case["cached"]:
        layout = dict(do_expand=case["expand"], alignment=case["alignment"])
        if case["kind"] == "group":
            state["handles"] = [got.handle for got in buf.dispatch(xs, topk_idx=idxs, weights=ws, **layout)]
        else:
            state["handles"] = [buf.dispatch(xs[0], topk_idx=idxs[0], weights=ws[0], **layout).handle]
    state.update(xs=xs, idxs=idxs, ws=ws, biases=biases if case["bias"] else None)
    return state


# ----------------------------------------------------------------------------------------------- one pass


def _outputs(case, got, back):
    out = {"x": back.x}
    if case["return_weights"]:
        out["topk_weights"] = back.topk_weights
    compact = case["kind"] == "exchange" and not case["expand"]
    if compact:
        out.update(recv_x=got.x, recv_topk_idx=got.topk_idx, recv_topk_weights=got.topk_weights)
    if not case["cached"]:
        layout = got.handle.layout
        out.update(expert_counts=layout.expert_counts, expert_offsets=layout.expert_offsets)
        if compact:
            out["recv_metadata"] = layout.recv_metadata
    return out


def _run_exchange(case, state):
    buf, x, idx, w = state["buffer"], state["xs"][0], state["idxs"][0], state["ws"][0]
    asynchronous = case["async_op"]
    if case["cached"]:
        got = buf.dispatch(x, weights=w, handle=state["handles"][0], zero_padding=case["zero_padding"], async_op=asynchronous)
    else:
        got = buf.dispatch(x, topk_idx=idx, weights=w, do_expand=case["expand"], alignment=case["alignment"],
                           zero_padding=case["zero_padding"], async_op=asynchronous)
    if asynchronous:
        got.event.current_stream_wait()
    back = buf.combine(got.x, got.handle, weights=got.topk_weights if case["return_weights"] else None,
                       bias=state["biases"][0] if case["bias"] else None, async_op=asynchronous)
    if asynchronous:
        back.event.current_stream_wait()
    return _outputs(case, got, back)


def _run_group(case, state):
    group = state["buffer"]
    if case["cached"]:
        got = group.dispatch(state["xs"], weights=state["ws"], handles=state["handles"], zero_padding=case["zero_padding"])
    else:
        got = group.dispatch(state["xs"], topk_idx=state["idxs"], weights=state["ws"], do_expand=case["expand"], alignment=case["alignment"],
                             zero_padding=case["zero_padding"])
    back = group.combine([g.x for g in got], [g.handle for g in got], weights=[g.topk_weights for g in got] if case["return_weights"] else None,
                         bias=state["biases"])
    return [_outputs(case, g, b) for g, b in zip(got, back)]


def run(state):
    case = state["case"]
    if case["kind"] == "exchange":
        return _run_exchange(case, state)
    if case["kind"] == "group":
        return _run_group(case, state)
    bias = state["biases"][0] if case["bias"] else None
    return state["layer"](state["xs"][0], state["idxs"][0], state["ws"][0], bias=bias)


# ----------------------------------------------------------------------------------------------- what a pass cannot do without


def work(case):
    tokens, hidden, experts, topk = case["tokens"], case["hidden"], case["experts"], case["topk"]
    ranks = case.get("ranks", 1)
    kept = 1 - 0.1 * (topk - 1) / topk if case["routing"] == "zipf" else 1.0  # a tenth of the choices after the first is masked
    source = ranks * tokens
    assigned = source * topk * kept
    row = 2 * hidden
    inputs = source * (row + 4 * topk) + (source * row if case["bias"] else 0)
    if case["kind"] == "layer":
        inner = case["inner"]
        touched = experts * (1 - (1 - min(1.0, topk / experts)) ** (tokens * kept))  # experts that hold a token
        return {"bytes": inputs + source * row + source * topk * 8 + touched * 3 * inner * hidden * 2, "flops": 6.0 * assigned * hidden * inner}
    if case["expand"]:
        received = assigned
        if case["zero_padding"]:
            # an expert's rows are padded up to the alignment: half of it on average, all but the rows of a small count
            per_expert = assigned / experts
            received += experts * (case["alignment"] - 1) * (0.5 if per_expert > 1 else 0.5 * per_expert)
    else:
        per_rank = 1 - (1 - 1 / ranks) ** (topk * kept) if ranks > 1 else 1.0  # ranks that a token goes to
        received = source * ranks * per_rank
    weights = received * 4 * (1 if case["expand"] else topk)
    dispatch = inputs + received * row + weights + (0 if case["cached"] else source * topk * 8 + received * (topk + 2) * 4 / (topk if case["expand"] else 1))
    combine = (assigned if case["expand"] else received) * row + source * row
    if case["return_weights"]:
        combine += weights + source * topk * 4
    return {"bytes": dispatch + combine, "flops": (assigned if case["expand"] else received) * hidden}


def tolerance(case):
    # An exchange moves bits; a combine adds in FP32 in ascending choice and rounds once: one right answer.
    if case["kind"] != "layer":
        return "exact"
    # Against the same layer in 64 bits (bf16 activations between the GEMMs, one bf16 round per returned row and one of the
    # result are the differences): relative error 2.9e-3, largest difference 1.8e-2 of the result's scale; four times that.
    return {"rel": 1.2e-2, "max": 7e-2}
