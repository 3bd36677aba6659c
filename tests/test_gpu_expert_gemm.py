"""The grouped GEMM with weights as the M operand: experts of any number of rows, token tiles of every size."""

from datetime import timedelta

import pytest
import torch
import torch.distributed as dist

from nanoep_b200 import CudaBuffer, EPConfig
from nanoep_b200.models.moe_layer import ExpertParallelMoE, dense_reference
from nanoep_b200.ops import grouped_gemm as gg
from nanoep_b200.parallel.cuda_buffer import handle_metadata

pytestmark = pytest.mark.gpu


def _problem(counts, K, N):
    blocks = [(c + 127) // 128 for c in counts]
    offsets = torch.tensor([0] + blocks, dtype=torch.int64).cumsum(0) * 128
    a = torch.full((int(offsets[-1]), K), float("nan"), dtype=torch.bfloat16)
    real = torch.zeros(int(offsets[-1]), dtype=torch.bool)
    for e, c in enumerate(counts):
        lo = int(offsets[e])
        a[lo : lo + c] = (torch.randn(c, K) * 0.5).to(torch.bfloat16)
        real[lo : lo + c] = True
    w = (torch.randn(len(counts), N, K) * 0.1).to(torch.bfloat16)
    return a.cuda(), w.cuda(), offsets.cuda(), torch.tensor(counts, dtype=torch.int64, device="cuda"), real.cuda()


@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("largest", [0, 64, 128, 300])  # token tile 256, 64 and 128 (300: where the experts are small); larger experts are split
@pytest.mark.parametrize("counts,K,N", [([1], 64, 256), ([31, 32, 0, 33, 64], 512, 512), ([0, 129, 255, 256, 257, 0], 256, 768), ([1000, 5, 2304], 1024, 256)])
def test_rows_that_exist(counts, K, N, largest, swiglu):
    """Padding rows hold NaN and must not reach a real row; rows of experts end anywhere inside a tile."""
    torch.manual_seed(7)
    a, w, offsets, n, real = _problem(counts, K, N)
    scale = None if swiglu else torch.rand(a.shape[0], device="cuda") + 0.5
    out = gg.grouped_gemm(a, w, offsets, swiglu=swiglu, row_scale=scale, expert_counts=n, max_expert_rows=largest)
    few = gg.grouped_gemm(a, w, offsets, swiglu=swiglu, row_scale=scale, expert_counts=n, max_expert_rows=largest, max_ctas=4)
    torch.cuda.synchronize()
    gg.check_status()
    ref = gg.grouped_gemm_reference(a, w, offsets, swiglu=swiglu)
    if scale is not None:
        ref = ref * scale[:, None]
    # one bf16 round of an fp32-accumulated product
    torch.testing.assert_close(out[real].float(), ref[real], rtol=1e-2, atol=1e-2)
    assert torch.equal(out[real], few[real]), "the result does not depend on the number of CTAs"


@pytest.mark.parametrize("largest", [0, 64, 128])  # token tiles of 256, 64 and 128
@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize(
    "counts,ranges,K,N",
    [
        ([3, 0, 40], [1024, 512, 2048], 128, 512),  # the offsets allow far more units than the counts give
        ([0, 0], [128, 256], 64, 256),              # no unit at all
        ([1], [128], 64, 512),                      # fewer units than clusters
        ([2304, 1000, 129, 0, 777, 256, 1, 511], None, 64, 2048),  # short units, several per cluster
        ([640, 385, 130], None, 2048, 1280),
        ([700, 0, 3, 0, 130, 4000], [4096] * 6, 64, 5120),  # largest = 64 is far from true here: 1024 places for 1560 units
    ],
)
def test_units_taken_over_by_running_clusters(counts, ranges, K, N, swiglu, largest):
    """Without a cap on the CTAs the units are handed out as clusters get free; with one every cluster has a fixed share.
    Each unit is computed the same way wherever it runs."""
    torch.manual_seed(11)
    a, w, offsets, n, real = _problem(counts if ranges is None else ranges, K, N)
    a = torch.nan_to_num(a, nan=0.25)
    if ranges is not None:
        real.zero_()
        for e, c in enumerate(counts):
            real[int(offsets[e]) : int(offsets[e]) + c] = True
        n = torch.tensor(counts, dtype=torch.int64, device="cuda")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    shape = (a.shape[0], N // 2 if swiglu else N)
    runs = [gg.grouped_gemm(a, w, offsets, swiglu=swiglu, expert_counts=n, max_expert_rows=largest, max_ctas=cap,
                            out=torch.full(shape, 3.0, dtype=torch.bfloat16, device="cuda")) for cap in (0, sms, 2, 0)]
    torch.cuda.synchronize()
    gg.check_status()
    ref = gg.grouped_gemm_reference(a, w, offsets, swiglu=swiglu)
    torch.testing.assert_close(runs[0][real].float(), ref[real], rtol=1e-2, atol=1e-2)  # one bf16 round of an fp32-accumulated product
    for other in runs[1:]:
        assert torch.equal(runs[0][real], other[real])


def test_limits_start_when_the_kernel_in_front_has_ended():
    """A GEMM that starts early sits on its SMs while the kernel in front of it runs (a pull may wait for its peers): that time
    does not count towards its own limits, and what that kernel writes is what it reads."""
    torch.manual_seed(12)
    a, w, offsets, n, _ = _problem([4096] * 2, 4096, 4096)
    a *= 0.1
    w2 = (torch.randn(2, 512, 4096) * 0.02).to(torch.bfloat16).cuda()
    h, late, early = (torch.empty(a.shape[0], cols, dtype=torch.bfloat16, device="cuda") for cols in (4096, 512, 512))
    ext, status = gg._ext(), gg.status_tensor(a.device)

    def run(out, front_ctas, is_early, limit_s):
        gg.grouped_gemm(a, w, offsets, expert_counts=n, max_ctas=front_ctas, out=h)
        ext.grouped_gemm(h, w2, offsets, out, status, gg.PLAIN, None, None, 0, limit_s, None, 4, False, n, 0, is_early)

    run(late, 0, False, 5.0)
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    h.zero_()
    start.record()
    run(early, 2, True, 2e-3)  # one pair of CTAs in front, the others are free
    end.record()
    torch.cuda.synchronize()
    gg.check_status()
    assert start.elapsed_time(end) > 6, "the kernel in front ran far longer than the limit"
    assert torch.equal(early, late)


@pytest.mark.parametrize("pair", [False, True])
def test_matches_the_gated_kernels(pair):
    """The kernels with tokens as M (row blocks gated by counters) add the same products: at most one bf16 step apart."""
    torch.manual_seed(8)
    a, w, offsets, n, _ = _problem([128, 256, 384], 512, 512)
    full = torch.full((a.shape[0] // 128,), 128, dtype=torch.int32, device="cuda")
    for swiglu in (False, True):
        got = gg.grouped_gemm(a, w, offsets, swiglu=swiglu, expert_counts=n)
        gated = gg.grouped_gemm(a, w, offsets, swiglu=swiglu, tile_ready=full, tile_expected=full, pair=pair)
        torch.testing.assert_close(got.float(), gated.float(), rtol=8e-3, atol=1e-3)


def test_bad_offsets_are_reported():
    a = torch.zeros(256, 128, dtype=torch.bfloat16, device="cuda")
    w = torch.zeros(2, 256, 128, dtype=torch.bfloat16, device="cuda")
    n = torch.tensor([100, 100], dtype=torch.int64, device="cuda")
    for bad in ([0, 100, 256], [0, 128, 128]):
        gg.grouped_gemm(a, w, torch.tensor(bad, dtype=torch.int64, device="cuda"), expert_counts=n)
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError, match="expert_offsets"):
            gg.check_status()


@pytest.fixture(scope="module")
def one_rank():
    own = not dist.is_initialized()
    if own:
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1, timeout=timedelta(seconds=60))
    yield dist.group.WORLD
    if own:
        dist.destroy_process_group()


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("tokens", [1, 64, 65, 129, 700])
def test_layer_on_one_rank(one_rank, tokens, fused):
    """Uneven experts, masked choices and a bias; routing changes between two passes and padding rows hold whatever was there."""
    H, inner, E, K = 512, 384, 5, 3
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    w13 = (torch.randn(E, 2 * inner, H, device="cuda", generator=gen) * 0.06).to(torch.bfloat16)
    w2 = (torch.randn(E, H, inner, device="cuda", generator=gen) * 0.06).to(torch.bfloat16)
    with CudaBuffer(one_rank, EPConfig(E, K, H, 700)) as buf:
        layer = ExpertParallelMoE(buf, w13, w2, fuse_combine=fused)
        for _ in range(2):
            x = (torch.randn(tokens, H, device="cuda", generator=gen) * 0.5).to(torch.bfloat16)
            bias = torch.randn(tokens, H, device="cuda", generator=gen).to(torch.bfloat16)
            skew = torch.rand(tokens, E, device="cuda", generator=gen) * torch.arange(1, E + 1, device="cuda")
            gate, idx = skew.topk(K, dim=-1)
            idx = torch.where(torch.rand(tokens, K, device="cuda", generator=gen) < 0.2, -1, idx)
            gate = (gate / gate.sum(-1, keepdim=True)).float()
            poison = torch.full((8 << 20,), float("nan"), dtype=torch.bfloat16, device="cuda")
            del poison
            out = layer(x, idx, gate, bias=bias)
            torch.cuda.synchronize()
            buf.check_status()
            gg.check_status()
            want = dense_reference(x, idx, gate, w13, w2).float() + bias.float()
            torch.testing.assert_close(out.float(), want, rtol=3e-2, atol=3e-2)


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("hidden,tokens,masked", [(512, 0, 0.0), (512, 1, 0.0), (512, 200, 0.2), (512, 200, 0.97), (512, 40, 1.0), (16384, 4000, 0.0)])
def test_layer_queued_in_front_of_its_counts(one_rank, hidden, tokens, masked, fused):
    """One native call, on tensors of their bound where the call is small, against the layer step by step: the same bits and
    the same handle, also without a single choice, with tokens that have none, and beyond the limit on the bound."""
    inner, E, K = 256, 4, 2
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    w13 = (torch.randn(E, 2 * inner, hidden, device="cuda", generator=gen) * 0.03).to(torch.bfloat16)
    w2 = (torch.randn(E, hidden, inner, device="cuda", generator=gen) * 0.06).to(torch.bfloat16)
    with CudaBuffer(one_rank, EPConfig(E, K, hidden, max(tokens, 8))) as buf:
        layer = ExpertParallelMoE(buf, w13, w2, fuse_combine=fused)
        x = (torch.randn(tokens, hidden, device="cuda", generator=gen) * 0.5).to(torch.bfloat16)
        bias = torch.randn(tokens, hidden, device="cuda", generator=gen).to(torch.bfloat16)
        gate, idx = torch.rand(tokens, E, device="cuda", generator=gen).topk(K, dim=-1)
        idx = torch.where(torch.rand(tokens, K, device="cuda", generator=gen) < masked, -1, idx)
        for weights in (gate, None):
            steps = layer._forward_in_steps(x, idx, weights, None, bias)
            old = layer.last_handle
            poison = torch.full((64 << 20,), float("nan"), dtype=torch.bfloat16, device="cuda")
            del poison
            whole = layer(x, idx, weights, bias=bias)
            new = layer.last_handle
            again = layer(x, None, weights, handle=new, bias=bias)
            torch.cuda.synchronize()
            buf.check_status()
            gg.check_status()
            assert torch.equal(whole, steps) and torch.equal(again, steps)
            assert (new.layout.recv_count, new.layout.expanded_capacity) == (old.layout.recv_count, old.layout.expanded_capacity)
            for a, b in zip(handle_metadata(new), handle_metadata(old)):
                assert a.shape == b.shape and a.dtype == b.dtype
            assert torch.equal(new.layout.expert_counts, old.layout.expert_counts) and torch.equal(new.topk_idx, old.topk_idx)


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("tokens", [1, 300, 20000])  # queued in front of the counts, and beyond the limit on the bound
def test_layer_refuses_an_invalid_expert_id(one_rank, tokens, fused):
    """The pass that got the bad id raises, however early its kernels were queued; the next pass is not affected."""
    E, K, hidden, inner = 8, 2, 4096, 128
    w13 = torch.zeros(E, 2 * inner, hidden, dtype=torch.bfloat16, device="cuda")
    w2 = torch.zeros(E, hidden, inner, dtype=torch.bfloat16, device="cuda")
    with CudaBuffer(one_rank, EPConfig(E, K, hidden, tokens)) as buf:
        layer = ExpertParallelMoE(buf, w13, w2, fuse_combine=fused)
        x = torch.zeros(tokens, hidden, dtype=torch.bfloat16, device="cuda")
        good = torch.tensor([0, 1], device="cuda").expand(tokens, K).contiguous()
        bad = good.clone()
        bad[-1, 1] = E
        gate = torch.ones(tokens, K, device="cuda")
        for _ in range(3):
            with pytest.raises(RuntimeError, match="expert id"):
                layer(x, bad, gate)
            buf.clear_status()
            assert not layer(x, good, gate).any()
            torch.cuda.synchronize()
            buf.check_status()
            gg.check_status()


@pytest.mark.parametrize(
    "hidden,inner,tokens,fused,ahead",
    [
        (512, 256, 0, True, True), (512, 256, 1, False, True), (512, 256, 200, True, True), (512, 256, 200, False, True),
        (16384, 256, 4000, True, False), (16384, 256, 4000, False, False),  # 266 MB of rows
        (4096, 128, 7900, True, True), (4096, 128, 7900, False, True), (4096, 128, 8000, True, False),  # 127 and 129 MB
        (256, 4096, 20000, True, True), (256, 4096, 24000, True, False), (256, 8192, 24000, False, False),  # 20-24 MB, but 336, 403 and 805 MB with activations
    ],
)
def test_when_a_layer_is_queued_in_front_of_its_counts(one_rank, hidden, inner, tokens, fused, ahead):
    """Its tensors have the size of their bound then: only so many bytes of rows, and of what the GEMMs make of them."""
    E, K = 4, 2
    ext = gg._ext()
    w13 = torch.zeros(E, 2 * inner, hidden, dtype=torch.bfloat16, device="cuda")
    w2 = torch.zeros(E, hidden, inner, dtype=torch.bfloat16, device="cuda")
    with CudaBuffer(one_rank, EPConfig(E, K, hidden, max(tokens, 8))) as buf:
        layer = ExpertParallelMoE(buf, w13, w2, fuse_combine=fused)
        x = torch.zeros(tokens, hidden, dtype=torch.bfloat16, device="cuda")
        gate, idx = torch.rand(tokens, E, device="cuda").topk(K, dim=-1)
        before = ext.queued_ahead_count()
        layer(x, idx, gate)
        assert ext.queued_ahead_count() - before == ahead
        layer(x, None, gate, handle=layer.last_handle)  # the counts are known
        assert ext.queued_ahead_count() - before == ahead
        torch.cuda.synchronize()


@pytest.mark.parametrize("max_ctas", [1, 2, 6])
def test_scatter_on_a_small_grid(one_rank, max_ctas):
    """The down-projection with the scatter epilogue takes any cap on its grid and gives the same bits."""
    T, H, inner, E, K = 150, 256, 128, 3, 2
    gen = torch.Generator(device="cuda").manual_seed(4)
    x = (torch.randn(T, inner, device="cuda", generator=gen) * 0.5).to(torch.bfloat16)
    w2 = (torch.randn(E, H, inner, device="cuda", generator=gen) * 0.1).to(torch.bfloat16)
    idx = torch.rand(T, E, device="cuda", generator=gen).topk(K, dim=-1).indices
    gate = torch.rand(T, K, device="cuda", generator=gen)
    with CudaBuffer(one_rank, EPConfig(E, K, H, T)) as buf:
        got = buf.dispatch(torch.zeros(T, H, dtype=torch.bfloat16, device="cuda"), topk_idx=idx, weights=gate, do_expand=True, alignment=128)
        lay = got.handle.layout
        h = torch.zeros(lay.expanded_capacity, inner, dtype=torch.bfloat16, device="cuda")
        slots = lay.recv_metadata[:, 2:].long()
        h[slots] = x[lay.recv_metadata[:, 1].long()][:, None].expand(-1, K, -1)
        outs = []
        for cap in (0, max_ctas):
            gg._ext().grouped_gemm_scatter(buf.window, h, w2, lay.expert_offsets, got.handle.slot_map, lay.recv_metadata, got.topk_weights,
                                           gg.status_tensor(h.device), cap, 5.0, lay.expert_counts, lay.recv_count)
            outs.append(gg._ext().combine_finish([buf.window], [handle_metadata(got.handle)], [None])[0])
        torch.cuda.synchronize()
        buf.check_status()
        gg.check_status()
        assert torch.equal(outs[0], outs[1])
        want = sum((x.float()[:, None] @ w2[idx[:, k]].float().transpose(1, 2))[:, 0] * gate[:, k, None] for k in range(K))
        torch.testing.assert_close(outs[0].float(), want, rtol=1e-2, atol=2e-2)  # bf16 round per row and of the sum


@pytest.mark.parametrize("hidden", [512, 4096])  # 4096: the pull's rings fill their limit, and the gated GEMM has to fit beside them
@pytest.mark.parametrize("pairs", [None, False, True])
def test_overlapped_layer_on_one_rank(one_rank, hidden, pairs):
    """The gated up-projection beside the dispatch that fills its row blocks: same result as one after the other, no wait runs out."""
    T, inner, E, K = 1500, 256, 6, 3
    gen = torch.Generator(device="cuda").manual_seed(hidden)
    w13 = (torch.randn(E, 2 * inner, hidden, device="cuda", generator=gen) * 0.03).to(torch.bfloat16)
    w2 = (torch.randn(E, hidden, inner, device="cuda", generator=gen) * 0.06).to(torch.bfloat16)
    with CudaBuffer(one_rank, EPConfig(E, K, hidden, T)) as buf:
        overlapped = ExpertParallelMoE(buf, w13, w2, overlap_dispatch=True, cta_pairs=pairs)
        plain = ExpertParallelMoE(buf, w13, w2)
        for _ in range(3):
            x = (torch.randn(T, hidden, device="cuda", generator=gen) * 0.5).to(torch.bfloat16)
            gate, idx = torch.rand(T, E, device="cuda", generator=gen).topk(K, dim=-1)
            idx = torch.where(torch.rand(T, K, device="cuda", generator=gen) < 0.1, -1, idx)
            for handle in (None, True):
                routing = dict(handle=overlapped.last_handle) if handle else {}
                got = overlapped(x, None if handle else idx, gate, **routing)
                torch.cuda.synchronize()
                buf.check_status()
                gg.check_status()
                want = plain(x, idx, gate)
                torch.cuda.synchronize()
                # the same products, added in another order by the two GEMM kernels: bf16 rounds of h, of a row and of the sum
                torch.testing.assert_close(got.float(), want.float(), rtol=3e-2, atol=3e-2)
