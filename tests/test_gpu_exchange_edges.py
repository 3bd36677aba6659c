"""Dispatch and combine on one GPU at the sizes where a kernel's split changes: edges of waves, tiles and launch shapes.

Everything is compared with the CPU oracle bit for bit."""

import pytest
import torch

from nanoep_b200 import EmulatedGroup, EPConfig
from nanoep_b200.testing.cases import make_case
from nanoep_b200.testing.checks import assert_dispatch_matches

pytestmark = pytest.mark.gpu


def _cuda(ts):
    return [t.cuda() for t in ts]


@pytest.mark.parametrize("world", [1, 2])
@pytest.mark.parametrize("experts_per_rank", [31, 33, 257])
@pytest.mark.parametrize("alignment", [1, 3, 128])
def test_padding_rows_of_many_experts(world, experts_per_rank, alignment):
    """Gap rows are numbered 32 experts at a time, eight such waves per pass; rows longer than the zero source."""
    case = make_case(world, kind="mixed", seed=experts_per_rank, hidden=8192, tokens=19, experts_per_rank=experts_per_rank, topk=4)
    cfg = EPConfig(case.num_experts, case.num_topk, case.hidden, case.capacity)
    with EmulatedGroup(world, cfg) as group:
        first = group.dispatch(_cuda(case.xs), topk_idx=_cuda(case.indices), weights=_cuda(case.weights), do_expand=True, alignment=alignment,
                               zero_padding=True)
        again = group.dispatch(_cuda(case.xs), handles=[f.handle for f in first], weights=_cuda(case.weights), zero_padding=True)
        torch.cuda.synchronize()
        group.check_status()
        for got in (first, again):
            for r in range(world):
                assert_dispatch_matches(got[r], case.xs, case.indices, case.weights, case.num_experts, r, expand=True, alignment=alignment,
                                        zero_padding=True)


def _values(case, seed=3):
    gen = torch.Generator().manual_seed(seed)
    return [torch.randn(idx.shape[0], case.num_topk, case.hidden, generator=gen).to(torch.bfloat16) for idx in case.indices]


def _expert_rows(values, meta, capacity):
    y = torch.full((capacity, values.shape[-1]), float("nan"), dtype=torch.bfloat16)  # padding must not be read
    slots, tok = meta[:, 2:], meta[:, 1]
    row, k = (slots >= 0).nonzero(as_tuple=True)
    y[slots[row, k]] = values[tok[row], k]
    return y


@pytest.mark.parametrize("tokens,topk,hidden", [(1, 8, 256), (2, 1, 768), (5, 9, 7168), (37, 17, 1280), (700, 4, 512)])
@pytest.mark.parametrize("multiple", [False, True])
def test_single_rank_combine_shapes(tokens, topk, hidden, multiple):
    """Row sums of a single-rank group: rows shorter and longer than a work item, one to three batches of eight rows per
    token, masked choices, tokens without a row, both rounding modes, both layouts."""
    case = make_case(1, kind="random", seed=tokens, hidden=hidden, tokens=tokens, experts_per_rank=max(4, topk), topk=topk)
    if tokens > 2:
        case.indices[0][tokens // 2] = -1
    cfg = EPConfig(case.num_experts, case.num_topk, case.hidden, case.capacity)
    values = _values(case)
    bias = torch.randn(tokens, hidden).to(torch.bfloat16)
    with EmulatedGroup(1, cfg, allow_multiple_reduction=multiple) as group:
        for expand in (True, False):
            got = group.dispatch(_cuda(case.xs), topk_idx=_cuda(case.indices), weights=_cuda(case.weights), do_expand=expand, alignment=4 if expand else 1)[0]
            meta = got.handle.layout.recv_metadata.cpu().long()
            y = _expert_rows(values[0], meta, got.handle.layout.expanded_capacity) if expand else values[0][meta[:, 1], 0]
            back = group.combine([y.cuda()], [got.handle], weights=[got.topk_weights], bias=[bias.cuda()])[0]
            torch.cuda.synchronize()
            group.check_status()
            valid = case.indices[0] >= 0
            want = torch.zeros(tokens, hidden)
            if expand:
                for k in range(topk):  # FP32 in ascending choice
                    want = torch.where(valid[:, k, None], want + values[0][:, k].float(), want)
                if multiple:
                    want = want.to(torch.bfloat16).float()
            else:
                want = torch.where(valid.any(1)[:, None], want + values[0][:, 0].float(), want)
            want = (want + bias.float()).to(torch.bfloat16)
            assert torch.equal(back.x.cpu().view(torch.int16), want.view(torch.int16)), expand
            torch.testing.assert_close(back.topk_weights.cpu(), case.weights[0].masked_fill(~valid, 0), rtol=0, atol=0)


@pytest.mark.parametrize("tokens,experts,topk,kind", [
    (1, 1, 1, "random"), (31, 7, 3, "mixed"), (33, 40, 32, "random"), (64, 5, 2, "masked"), (512, 64, 2, "mixed"), (513, 9, 3, "random"),
    (1025, 300, 2, "mixed"), (4200, 16, 2, "random"), (8300, 3, 1, "random"),
])
def test_single_rank_plan(tokens, experts, topk, kind):
    """The one-launch plan of a single-rank group: one to eight CTAs, one or several chunks per warp, ragged last chunk."""
    case = make_case(1, kind=kind, seed=tokens, hidden=256, tokens=tokens, experts_per_rank=experts, topk=topk)
    case.indices[0][::7] = -1  # tokens without a row
    cfg = EPConfig(case.num_experts, case.num_topk, case.hidden, case.capacity)
    with EmulatedGroup(1, cfg) as group:
        for expand, alignment in ((True, 1), (True, 24), (False, 1)):
            got = group.dispatch(_cuda(case.xs), topk_idx=_cuda(case.indices), weights=_cuda(case.weights), do_expand=expand, alignment=alignment,
                                 zero_padding=True)
            torch.cuda.synchronize()
            group.check_status()
            assert_dispatch_matches(got[0], case.xs, case.indices, case.weights, case.num_experts, 0, expand=expand, alignment=alignment,
                                    zero_padding=True)


@pytest.mark.parametrize("world", [8, 16])  # parameter blocks by value, and from device memory
def test_many_logical_ranks(world):
    case = make_case(world, kind="mixed", seed=world, hidden=512, tokens=9, experts_per_rank=3, topk=4)
    cfg = EPConfig(case.num_experts, case.num_topk, case.hidden, case.capacity)
    with EmulatedGroup(world, cfg) as group:
        first = group.dispatch(_cuda(case.xs), topk_idx=_cuda(case.indices), weights=_cuda(case.weights), do_expand=True, alignment=8, zero_padding=True)
        again = group.dispatch(_cuda(case.xs), handles=[f.handle for f in first], weights=_cuda(case.weights), zero_padding=True)
        back = [group.combine([g.x for g in got], [g.handle for g in got], weights=[g.topk_weights for g in got]) for got in (first, again)]
        torch.cuda.synchronize()
        group.check_status()
        for got in (first, again):
            for r in range(world):
                assert_dispatch_matches(got[r], case.xs, case.indices, case.weights, case.num_experts, r, expand=True, alignment=8, zero_padding=True)
        for r in range(world):
            idx, x = case.indices[r], case.xs[r].float()
            # the sum of up to four equal bf16 values is exact in FP32 and rounded once
            want = (x * (idx >= 0).sum(-1, keepdim=True)).to(torch.bfloat16)
            for b in back:
                assert torch.equal(b[r].x.cpu(), want)
                assert torch.equal(b[r].topk_weights.cpu(), torch.where(idx >= 0, case.weights[r], 0.0))


@pytest.mark.parametrize("setting", [-3000, -40001, -200001])  # stages * 1000 + chunk / 128: three whole-row stages, 40 and 200 of 128 bytes
def test_reduction_with_many_stages(setting):
    """Every stage of the reduce ring has its own row count; token counts of neighbouring stages differ here."""
    from nanoep_b200.utils.build import load_extension

    world = 2
    case = make_case(world, kind="mixed", seed=5, hidden=256, tokens=300, experts_per_rank=4, topk=4)
    cfg = EPConfig(case.num_experts, case.num_topk, case.hidden, case.capacity)
    ext = load_extension()
    ext.set_combine_trace(False, 0, setting)
    try:
        with EmulatedGroup(world, cfg) as group:
            got = group.dispatch(_cuda(case.xs), topk_idx=_cuda(case.indices), weights=_cuda(case.weights), do_expand=True, alignment=1)
            # two CTAs per rank: 150 tokens of one to four chunks each go round the ring
            back = group.combine([g.x for g in got], [g.handle for g in got], weights=[g.topk_weights for g in got], num_sms=2)
            torch.cuda.synchronize()
            group.check_status()
            for r in range(world):
                idx, x = case.indices[r], case.xs[r].float()
                want = (x * (idx >= 0).sum(-1, keepdim=True)).to(torch.bfloat16)  # up to four equal bf16 values: exact in FP32
                assert torch.equal(back[r].x.cpu(), want)
    finally:
        ext.set_combine_trace(False, 0, 0)


def _own_rows_round_trip(tokens, own_shares, setting, num_sms, seed, run=1):
    """Two ranks with `tokens` tokens each (one number per rank) of which a share of the choices names an expert of the token's own
    rank (drawn for `run` tokens at a time); every choice comes back with values of its own."""
    from nanoep_b200.utils.build import load_extension

    world, hidden, local, topk = 2, 256, 6, 4
    gen = torch.Generator().manual_seed(seed)
    cfg = EPConfig(world * local, topk, hidden, max(tokens))
    xs = [torch.randn(n, hidden, generator=gen).to(torch.bfloat16) for n in tokens]
    ws = [torch.rand(n, topk, generator=gen) for n in tokens]
    idxs = []
    for r, n in enumerate(tokens):
        if run == 1:
            own = torch.rand(n, topk, generator=gen) < own_shares[r]
        else:
            own = (torch.rand((n + run - 1) // run, 1, generator=gen) < own_shares[r]).repeat_interleave(run, 0)[:n].expand(n, topk)
        within = torch.rand(n, local, generator=gen).topk(topk, dim=-1).indices
        idx = torch.where(own, within + r * local, within + (1 - r) * local)
        idxs.append(idx.masked_fill(torch.rand(n, topk, generator=gen) < 0.15, -1))
    # what a choice's expert returns; ranks may have different numbers of tokens
    values = [torch.randn(n, topk, hidden, generator=gen).to(torch.bfloat16) for n in tokens]
    padded = torch.zeros(world, max(tokens), topk, hidden, dtype=torch.bfloat16)
    for r, v in enumerate(values):
        padded[r, : v.shape[0]] = v
    ext = load_extension()
    ext.set_combine_trace(False, 0, setting)
    try:
        with EmulatedGroup(world, cfg) as group:
            for expand in (True, False, True):
                got = group.dispatch(_cuda(xs), topk_idx=_cuda(idxs), weights=_cuda(ws), do_expand=expand, alignment=8 if expand else 1)
                ys = []
                for r in range(world):
                    meta = got[r].handle.layout.recv_metadata.cpu().long()
                    src, tok, v = meta[:, 0], meta[:, 1], meta[:, 2:]
                    row, k = (v >= 0).nonzero(as_tuple=True)
                    if expand:
                        y = torch.full((got[r].handle.layout.expanded_capacity, hidden), float("nan"), dtype=torch.bfloat16)
                        y[v[row, k]] = padded[src[row], tok[row], k]
                    else:
                        y = padded[src, tok, (v >= 0).int().argmax(-1)]  # the rank's first choice names the row
                    ys.append(y.cuda())
                back = group.combine(ys, [g.handle for g in got], weights=[g.topk_weights for g in got], num_sms=num_sms)
                torch.cuda.synchronize()
                group.check_status()
                for r, n in enumerate(tokens):
                    want = torch.zeros(n, hidden)
                    for k in range(topk):  # FP32 in ascending choice
                        e = idxs[r][:, k]
                        counts = e >= 0
                        if not expand:  # one row per rank, with its first choice
                            earlier = (idxs[r][:, :k] >= 0) & (idxs[r][:, :k] // local == (e // local)[:, None])
                            counts = counts & ~earlier.any(-1)
                        want = torch.where(counts[:, None], want + values[r][:, k].float(), want)
                    assert torch.equal(back[r].x.cpu().view(torch.int16), want.to(torch.bfloat16).view(torch.int16)), (expand, r)
                    assert torch.equal(back[r].topk_weights.cpu(), ws[r].masked_fill(idxs[r] < 0, 0))
    finally:
        ext.set_combine_trace(False, 0, 0)


@pytest.mark.parametrize("own_share", [0.0, 0.6, 1.0])  # of the choices that name an expert of the token's own rank
@pytest.mark.parametrize("setting", [0, 2])  # reduction through its ring (own rows are read in place) and in registers (they are returned like others)
@pytest.mark.parametrize("num_sms", [1, 3, None])  # one CTA: every row of a rank in one sequence, far more than a transfer warp's board of flags
def test_rows_of_own_tokens(own_share, setting, num_sms):
    _own_rows_round_trip([230, 230], [own_share] * 2, setting, num_sms, int(own_share * 10))


@pytest.mark.parametrize("tokens,own_shares,run", [([700, 5], [0.98, 0.5], 1), ([613, 40], [0.9, 0.0], 37), ([64, 1000], [1.0, 0.95], 50), ([0, 333], [0.0, 1.0], 1)])
@pytest.mark.parametrize("num_sms", [1, 2])
def test_runs_of_own_tokens_between_few_others(tokens, own_shares, run, num_sms):
    """Flags of rows that stay where they are come in runs longer than a transfer warp's board, with few stored rows between."""
    _own_rows_round_trip(tokens, own_shares, 0, num_sms, sum(tokens) + run, run)


@pytest.mark.parametrize("masked", ["none", "choices", "tokens", "all"])
@pytest.mark.parametrize("expand,alignment", [(False, 1), (True, 1), (True, 16)])
@pytest.mark.parametrize("weighted", [False, True])
def test_outputs_own_exactly_what_they_show(masked, expand, alignment, weighted):
    """Whatever a single rank allocates before it knows its receive counts, the outputs keep no more memory than they show."""
    case = make_case(1, kind="random", seed=3, hidden=256, tokens=40, experts_per_rank=12, topk=4)
    idx = torch.stack([torch.randperm(case.num_experts)[: case.num_topk] for _ in range(40)])
    if masked == "choices":
        idx[::3, 1:] = -1
    elif masked == "tokens":
        idx[5:] = -1
    elif masked == "all":
        idx[:] = -1
    case.indices[0] = idx
    cfg = EPConfig(case.num_experts, case.num_topk, case.hidden, case.capacity)
    with EmulatedGroup(1, cfg) as group:
        got = group.dispatch(_cuda(case.xs), topk_idx=_cuda(case.indices), weights=_cuda(case.weights) if weighted else None, do_expand=expand,
                             alignment=alignment, zero_padding=True)[0]
        torch.cuda.synchronize()
        group.check_status()
        assert_dispatch_matches(got, case.xs, case.indices, case.weights, case.num_experts, 0, expand=expand, alignment=alignment,
                                zero_padding=True, weighted=weighted)
        for out in (got.x, got.topk_idx, got.topk_weights):
            if out is not None:
                assert out.untyped_storage().nbytes() == out.numel() * out.element_size() and out.storage_offset() == 0


def _one_rank_dispatch(idx, experts, hidden, **layout):
    gen = torch.Generator().manual_seed(idx.shape[0])
    x = torch.randn(idx.shape[0], hidden, generator=gen).to(torch.bfloat16)
    w = torch.rand(idx.shape, generator=gen)
    with EmulatedGroup(1, EPConfig(experts, idx.shape[1], hidden, idx.shape[0])) as group:
        got = group.dispatch([x.cuda()], topk_idx=[idx.cuda()], weights=[w.cuda()], zero_padding=True, **layout)[0]
        torch.cuda.synchronize()
        group.check_status()
    assert_dispatch_matches(got, [x], [idx], [w], experts, 0, expand=layout["do_expand"], alignment=layout["alignment"], zero_padding=True)
    lay = got.handle.layout
    kept = {t.untyped_storage().data_ptr(): t.untyped_storage().nbytes() for t in (lay.recv_metadata, got.handle.slot_map)}
    used = sum(t.numel() * t.element_size() for t in (lay.recv_metadata, got.handle.slot_map))
    assert sum(kept.values()) <= max(2 * used, 1 << 20)


@pytest.mark.parametrize("tokens,experts,topk", [(40, 511, 2), (40, 512, 2), (600, 513, 3), (1500, 1025, 4), (300, 2048, 9)])
def test_single_rank_plan_of_many_experts(tokens, experts, topk):
    """The plan scans 512 experts at a time; counts, offsets and alignment gaps go on across that line."""
    idx = torch.rand(tokens, experts, generator=torch.Generator().manual_seed(experts)).topk(topk, dim=-1).indices
    idx[::5, 0] = -1
    for layout in (dict(do_expand=True, alignment=1), dict(do_expand=True, alignment=12), dict(do_expand=False, alignment=1)):
        _one_rank_dispatch(idx, experts, 256, **layout)


@pytest.mark.parametrize("tokens", [32768, 32769])  # the one-launch plan's largest call, and one for the stage and plan kernels
@pytest.mark.parametrize("expand", [False, True])
def test_single_rank_plan_limit(tokens, expand):
    idx = torch.arange(tokens)[:, None] % 4
    _one_rank_dispatch(idx, 4, 256, do_expand=expand, alignment=8 if expand else 1)


@pytest.mark.parametrize("expand", [False, True])
def test_single_rank_handle_keeps_what_it_uses(expand):
    """20000 tokens, nearly all masked: the plan's bound is 1.4 MB (expert-major), the handle uses less than 1 KB."""
    idx = torch.full((20000, 8), -1)
    idx[::4000] = torch.arange(8)
    _one_rank_dispatch(idx, 16, 256, do_expand=expand, alignment=1)


def test_single_rank_alignment_far_above_the_counts():
    """16 choices could fill 16 experts of 2^19 rows; they go to one, so the handle needs a sixteenth of the bound."""
    idx = torch.full((4, 4), -1)
    idx[:, 2] = 3
    _one_rank_dispatch(idx, 16, 256, do_expand=True, alignment=1 << 19)


@pytest.mark.parametrize("world", [1, 2])
@pytest.mark.parametrize("tokens", [1, 700, 5000, 33000])  # one to eight CTAs, and no longer in one launch; the bad id is in the last token
def test_invalid_expert_id_stops_the_next_call(world, tokens):
    cfg = EPConfig(8, 2, 256, tokens)
    with EmulatedGroup(world, cfg) as group:
        x = [torch.zeros(tokens, 256, dtype=torch.bfloat16, device="cuda") for _ in range(world)]
        idx = [torch.zeros(tokens, 2, dtype=torch.int64, device="cuda") for _ in range(world)]
        for i in idx:
            i[:, 1] = 1
        idx[-1][-1, 1] = 8
        torch.cuda.synchronize()
        for _ in range(5):
            group.dispatch(x, topk_idx=idx, do_expand=True, alignment=1)
            with pytest.raises(RuntimeError, match="expert id"):  # no synchronisation in between
                group.check_status()
            torch.cuda.synchronize()
            for w in group.windows:
                w.clear_status(group.comm_stream.cuda_stream)
            torch.cuda.synchronize()
