// Python bindings of the tcgen05 grouped GEMM and helpers (tensor-map construction lives here).
#include "gemm_api.hpp"

#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>

#include "grouped_gemm_sm100.hpp"
#include "peer_window.hpp"
#include "pipeline.hpp"
#include "unit_queue.hpp"

namespace nep {
namespace {

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                              const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
    static EncodeFn fn = [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult result;
        cudaError_t e = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &result);
        TORCH_CHECK(e == cudaSuccess && result == cudaDriverEntryPointSuccess && ptr != nullptr, "cuTensorMapEncodeTiled is not available");
        return reinterpret_cast<EncodeFn>(ptr);
    }();
    return fn;
}

// Row-major bf16 [outer, rows, cols]; box = 64 columns (128 bytes, one swizzle row) x `box_rows` rows x `box_outer`.
CUtensorMap make_map(const void* base, int64_t rows, int64_t cols, int box_rows = 128, int64_t outer = 1, int box_outer = 0) {
    TORCH_CHECK(reinterpret_cast<uintptr_t>(base) % 16 == 0 && (cols * 2) % 16 == 0, "TMA operand must be 16-byte aligned with 16-byte row pitch");
    CUtensorMap map;
    const cuuint64_t dims[3] = {cuuint64_t(cols), cuuint64_t(rows), cuuint64_t(outer)};
    const cuuint64_t strides[2] = {cuuint64_t(cols) * 2, cuuint64_t(rows) * cuuint64_t(cols) * 2};
    const cuuint32_t box[3] = {64, cuuint32_t(box_rows), cuuint32_t(box_outer)};
    const cuuint32_t elem[3] = {1, 1, 1};
    CUresult r = encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, box_outer > 0 ? 3 : 2, const_cast<void*>(base), dims, strides, box, elem,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TORCH_CHECK(r == CUDA_SUCCESS, "cuTensorMapEncodeTiled failed");
    return map;
}

void check_bf16(const at::Tensor& t, int dims, const char* name) {
    TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16 && t.is_contiguous() && t.dim() == dims, name,
                " must be a contiguous CUDA bfloat16 tensor of the expected rank");
}

struct GemmCommon {
    gemm::Args args{};
    int grid = 0;
};

GemmCommon prepare(const at::Tensor& a, const at::Tensor& w, const at::Tensor& expert_offsets, const at::Tensor& status, int mode,
                   double timeout_s) {
    check_bf16(a, 2, "activations");
    check_bf16(w, 3, "weights");
    TORCH_CHECK(expert_offsets.is_cuda() && expert_offsets.scalar_type() == at::kLong && expert_offsets.is_contiguous() &&
                    expert_offsets.dim() == 1 && expert_offsets.size(0) == w.size(0) + 1,
                "expert_offsets must be a CUDA int64 tensor of num_experts + 1 entries");
    TORCH_CHECK(status.is_cuda() && status.scalar_type() == at::kInt && status.numel() >= 2, "status must be a CUDA int32 tensor");
    const int64_t rows = a.size(0), K = a.size(1), E = w.size(0), NW = w.size(1);
    TORCH_CHECK(w.size(2) == K, "weights must be [experts, N, K] with the activations' K");
    TORCH_CHECK(rows % 128 == 0, "row count must be a multiple of 128 (dispatch with alignment=128)");
    TORCH_CHECK(K % 64 == 0 && K >= 64, "K must be a multiple of 64");
    TORCH_CHECK(E >= 1 && E <= 1024, "1..1024 experts per rank");
    GemmCommon g;
    g.args.expert_offsets = expert_offsets.data_ptr<int64_t>();
    g.args.num_experts = int(E);
    g.args.rows = rows;
    g.args.m_blocks = int(rows / 128);
    g.args.k_blocks = int(K / 64);
    g.args.b_rows_per_expert = int(NW);
    if (mode == gemm::kSwiGLU) {
        TORCH_CHECK(NW % 256 == 0, "SwiGLU weight must be [experts, 2*I, K] with I a multiple of 128");
        g.args.swiglu_up_row_offset = int(NW / 2);
        g.args.n_tiles = int(NW / 2 / 128);
    } else {
        TORCH_CHECK(NW % 256 == 0, "N must be a multiple of 256");
        g.args.n_tiles = int(NW / 256);
    }
    g.args.status = reinterpret_cast<uint32_t*>(status.data_ptr<int>());
    g.args.timeout_ns = uint64_t(timeout_s * 1e9);
    // what a tensor map asks for, also where a call turns out to have nothing to do
    TORCH_CHECK((rows == 0 || reinterpret_cast<uintptr_t>(a.data_ptr()) % 16 == 0) && reinterpret_cast<uintptr_t>(w.data_ptr()) % 16 == 0,
                "TMA operand must be 16-byte aligned with 16-byte row pitch");
    const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
    g.grid = std::max(1, std::min(sms, g.args.m_blocks * g.args.n_tiles));
    return g;
}

cudaError_t launch_expert(GemmCommon& g, const at::Tensor& a, const at::Tensor& w, const c10::optional<at::Tensor>& counts, int mode,
                          int64_t max_expert_rows, int64_t max_ctas, bool early, int64_t assigned) {
    if (counts.has_value()) {
        TORCH_CHECK(counts->is_cuda() && counts->device() == a.device() && counts->scalar_type() == at::kLong && counts->is_contiguous() &&
                        counts->dim() == 1 && counts->size(0) == w.size(0),
                    "expert_counts must be an int64 tensor of num_experts entries on the activations' device");
        g.args.expert_counts = counts->data_ptr<int64_t>();
    }
    const int64_t rows = a.size(0), K = a.size(1), E = w.size(0), NW = w.size(1);
    gemm::ExpertMaps maps{};
    maps.weights = mode == gemm::kSwiGLU ? make_map(w.data_ptr(), NW / 2, K, 16, 2 * E, 2) : make_map(w.data_ptr(), E * NW, K);
    // A smaller token tile deepens the operand pipeline, which weights streamed from memory need; more rows than a tile holds
    // read the weights again, from L2.  Experts of 7168 x 2048, 32 of them, up-projection with tiles of 64, 128 and 256: 64
    // tokens 283, 287 and 302 us; 256 tokens (at most 78 rows an expert) 324, 293 and 310-329 us; 512 tokens (at most 158) 526,
    // 374 and 319 us.  So: the smallest tile that no expert can outgrow, and 128 also where every expert has at most one
    // block of 128 rows on average and none can hold more than four.
    // Where `rows` is a bound, the number of choices stands for it.  Up- and down-projection of 32 experts, tiles of 128 against 256: with a
    // router's even counts 0.96-0.98 of the time from 24 to 112 rows on average and 1.15-1.35 at 128; under Zipf(1.2) 0.97-1.02 up to
    // 48, 0.99-1.03 at 64, 1.06 at 72 to 80, 1.06-1.10 at 96, 1.13-1.20 at 128.  80 lies between the two lines.
    const bool one_block = max_expert_rows <= 512 && (assigned >= 0 ? assigned <= 80 * E : rows <= 128 * E);
    const int tile = max_expert_rows <= 0 ? 256 : max_expert_rows <= 64 ? 64 : max_expert_rows <= 128 || one_block ? 128 : 256;
    for (int b = 0; b < 4; ++b)
        if ((128 >> b) <= tile / 2) maps.tokens[b] = make_map(a.data_ptr(), rows, K, 128 >> b);
    const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
    // Units that the offsets allow: an expert of n rows has a range of whole blocks of 128, and tiles of 256 split an odd number of
    // them into one more.  Without a cap on the CTAs clusters take over one another's places.
    const int64_t blocks = rows / 128, tiles = tile <= 128 ? blocks * 128 / tile : (blocks + std::min(E, blocks)) / 2;
    g.args.dynamic = max_ctas <= 0;
    g.args.rows_bound = assigned >= 0;
    const int grid = max_ctas > 0 ? std::min<int>(sms, int(max_ctas)) : int(2 * gemm::unit_places(tiles * g.args.n_tiles, E, max_expert_rows, tile, g.args.n_tiles));
    return gemm::launch_expert(maps, g.args, mode, tile, grid, early, c10::cuda::getCurrentCUDAStream().stream());
}

// Which kernel a grouped_gemm call runs.  The one with tokens as N is the faster one (expert_gemm_sm100.cu has both sides), but it
// takes all of an SM's shared memory and works in pairs of CTAs: row blocks gated by counters (which share the SMs with the
// dispatch that fills them), a caller who asks for CTA pairs or for the three-stage pipeline (smaller, to run beside another
// kernel), and a call that may use a single CTA get the kernels with tokens as M.
// So do two kinds of call that the single-CTA kernel serves better, where every row of every range exists (with counts the other
// kernel leaves rows out).  Nearly no K: the accumulator's way out is the whole kernel, and it is longer for the transposed
// one (K = 64, N = 256 to 4096, 1 to 128 experts of 1 to 9 blocks: 12-444 us against 12-485, 1.11x on average; at K = 256 1.03x,
// from 768 on the other way).  And calls whose 128-row tiles fit the GPU once while the pairs' tiles need a second wave
// (one expert of 1152 rows, N = 4096: 32 against 50 us at K = 2048, 52 against 71 with SwiGLU at K = 4096).
enum Kernel { kExpertKernel, kPairKernel, kSingleKernel };
struct Choice {
    bool gated, pair;
    int64_t stages, max_ctas;
    bool swiglu, counts;
    int64_t m_blocks, n_tiles, K, sms;
};
Kernel choose_kernel(const Choice& c) {
    if (c.pair) return kPairKernel;
    if (c.gated || c.stages == 3 || c.max_ctas == 1) return kSingleKernel;
    if (c.counts) return kExpertKernel;
    const int64_t ctas = c.max_ctas > 0 ? std::min(c.max_ctas, c.sms) : c.sms;
    const bool one_wave_of_singles = c.m_blocks * c.n_tiles <= ctas && (c.m_blocks + 1) / 2 * c.n_tiles > ctas / 2;
    return (!c.swiglu && c.K <= 128) || one_wave_of_singles ? kSingleKernel : kExpertKernel;
}

// out = A @ W[e]^T per 128-row block (mode 0) or silu(gate) * up with W = [E, 2I, K] (mode 1).  `early` as in launch_expert.
// `assigned` >= 0: the rows of `a` are an upper bound (the offsets say where they end), and so many of them at most are real.
void grouped_gemm(const at::Tensor& a, const at::Tensor& w, const at::Tensor& expert_offsets, at::Tensor& out, at::Tensor& status, int64_t mode,
                  c10::optional<at::Tensor> tile_ready, c10::optional<at::Tensor> tile_expected, int64_t max_ctas, double timeout_s,
                  c10::optional<at::Tensor> row_scale, int64_t stages, bool pair, c10::optional<at::Tensor> expert_counts, int64_t max_expert_rows, bool early, int64_t assigned) {
    c10::cuda::CUDAGuard guard(a.device());
    TORCH_CHECK(mode == gemm::kPlain || mode == gemm::kSwiGLU, "mode must be 0 (plain) or 1 (SwiGLU)");
    auto g = prepare(a, w, expert_offsets, status, int(mode), timeout_s);
    check_bf16(out, 2, "out");
    const int64_t n_out = mode == gemm::kSwiGLU ? w.size(1) / 2 : w.size(1);
    TORCH_CHECK(out.size(0) == a.size(0) && out.size(1) == n_out, "out has the wrong shape");
    g.args.out = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
    g.args.ldo = int(n_out);
    if (tile_ready.has_value()) {
        TORCH_CHECK(tile_expected.has_value() && tile_ready->scalar_type() == at::kInt && tile_expected->scalar_type() == at::kInt &&
                        tile_ready->numel() >= g.args.m_blocks && tile_expected->numel() >= g.args.m_blocks &&
                        tile_ready->is_cuda() && tile_expected->is_cuda() && tile_ready->device() == a.device() &&
                        tile_expected->device() == a.device() && tile_ready->is_contiguous() && tile_expected->is_contiguous(),
                    "tile_ready/tile_expected must be contiguous int32 tensors on the activations' device with one entry per 128-row block");
        g.args.tile_ready = tile_ready->data_ptr<int>();
        g.args.tile_expected = tile_expected->data_ptr<int>();
    }
    if (row_scale.has_value()) {
        TORCH_CHECK(mode == gemm::kPlain && row_scale->is_cuda() && row_scale->scalar_type() == at::kFloat &&
                        row_scale->is_contiguous() && row_scale->numel() == a.size(0),
                    "row_scale must be float32 [rows] (plain mode only)");
        g.args.row_scale = row_scale->data_ptr<float>();
    }
    TORCH_CHECK(stages == 3 || stages == 4, "stages must be 3 or 4 (single-CTA) or 4 for the gated CTA-pair kernel");
    if (a.size(0) == 0) return;
    const int grid = max_ctas > 0 ? std::min<int>(g.grid, int(max_ctas)) : g.grid;
    PeerWindow::launches += 1;
    const Kernel kernel = choose_kernel(Choice{tile_ready.has_value(), pair, stages, max_ctas, mode == gemm::kSwiGLU, expert_counts.has_value(),
                                               g.args.m_blocks, g.args.n_tiles, a.size(1),
                                               at::cuda::getCurrentDeviceProperties()->multiProcessorCount});
    if (kernel == kExpertKernel) {
        cudaError_t ee = launch_expert(g, a, w, expert_counts, int(mode), max_expert_rows, max_ctas, early, assigned);
        TORCH_CHECK(ee == cudaSuccess, "grouped GEMM (expert) launch failed: ", cudaGetErrorString(ee));
        return;
    }
    const CUtensorMap map_a = make_map(a.data_ptr(), a.size(0), a.size(1)), map_b = make_map(w.data_ptr(), w.size(0) * w.size(1), w.size(2));
    if (kernel == kPairKernel) {
        const int sms = at::cuda::getCurrentDeviceProperties()->multiProcessorCount;
        const int pair_grid = max_ctas > 0 ? std::min<int>(sms, int(max_ctas)) : sms;
        // gated by tile counters = meant to share the SMs with the pull kernel: shorter pipeline
        cudaError_t pe = gemm::launch_pair(map_a, map_b, g.args, int(mode), pair_grid, c10::cuda::getCurrentCUDAStream().stream(),
                                           tile_ready.has_value() ? 4 : 6);
        TORCH_CHECK(pe == cudaSuccess, "grouped GEMM (CTA pairs) launch failed: ", cudaGetErrorString(pe));
        return;
    }
    cudaError_t e = gemm::launch(map_a, map_b, g.args, int(mode), int(stages), grid, c10::cuda::getCurrentCUDAStream().stream());
    TORCH_CHECK(e == cudaSuccess, "grouped GEMM launch failed: ", cudaGetErrorString(e));
}

// Down projection fused with the combine push: row r of (A @ W[e]^T) * slot_weight[r] is stored
// (bf16) into the return partition of the row's source rank; padding rows are skipped.  The return area
// exists once: a dispatch (whose peer barrier every rank passes only after its previous reduction) must lie
// between two such calls, as it does in a layer's forward pass.
void grouped_gemm_scatter(PeerWindow& window, const at::Tensor& a, const at::Tensor& w, const at::Tensor& expert_offsets,
                          const at::Tensor& slot_map, const at::Tensor& recv_metadata, c10::optional<at::Tensor> slot_weights, at::Tensor& status,
                          int64_t max_ctas, double timeout_s, c10::optional<at::Tensor> expert_counts, int64_t max_expert_rows, bool early, int64_t assigned) {
    c10::cuda::CUDAGuard guard(a.device());
    auto g = prepare(a, w, expert_offsets, status, gemm::kScatter, timeout_s);
    const WindowLayout& L = window.layout();
    TORCH_CHECK(w.size(1) == L.hidden, "down-projection N must equal the buffer's hidden size");
    TORCH_CHECK(slot_map.is_cuda() && slot_map.scalar_type() == at::kInt && slot_map.numel() == a.size(0) && slot_map.is_contiguous(),
                "slot_map must be contiguous int32 [rows]");
    TORCH_CHECK(recv_metadata.is_cuda() && recv_metadata.scalar_type() == at::kInt && recv_metadata.dim() == 2 &&
                    recv_metadata.size(1) == L.topk + 2 && recv_metadata.is_contiguous(),
                "recv_metadata must be int32 [N, topk + 2]");
    g.args.slot_map = slot_map.data_ptr<int>();
    g.args.recv_metadata = recv_metadata.data_ptr<int>();
    if (slot_weights.has_value()) {
        TORCH_CHECK(slot_weights->is_cuda() && slot_weights->scalar_type() == at::kFloat && slot_weights->numel() == a.size(0),
                    "slot_weights must be float32 [rows]");
        g.args.slot_weights = slot_weights->data_ptr<float>();
    }
    const CommonParams c = window.common();
    for (int p = 0; p < kMaxRanks; ++p) g.args.peers[p] = c.peers[p];
    TORCH_CHECK(L.ret_parts == L.topk, "the fused combine epilogue needs one return partition per choice (allow_multiple_reduction=False)");
    g.args.ret_offset = L.ret_offset;
    g.args.max_tokens = L.max_tokens;
    g.args.topk = L.topk;
    g.args.ranks = L.ranks;
    g.args.recv_rows = int(recv_metadata.size(0));
    g.args.ldo = L.hidden;
    if (a.size(0) == 0) return;
    PeerWindow::launches += 1;
    // the kernel works in pairs of CTAs: a cap of one means one pair
    const cudaError_t e = launch_expert(g, a, w, expert_counts, gemm::kScatter, max_expert_rows, max_ctas == 1 ? 2 : max_ctas, early, assigned);
    TORCH_CHECK(e == cudaSuccess, "grouped GEMM (scatter) launch failed: ", cudaGetErrorString(e));
}

// A whole expert layer: dispatch (fresh with `topk`, cached with `cached` = the handle's tensors and capacity), up-projection with SwiGLU,
// down-projection, combine, all on the caller's stream.  In one call because the host would otherwise sit between the kernels: where
// the dispatch allows it everything is queued before the receive counts have reached the host.
// us before -> after, a layer of 64 tokens (32 experts of 7168 x 2048) 466 -> 447, of 777 tokens (4096 x 1536) 314 -> 306.
pybind11::tuple moe_forward(PeerWindow& window, const at::Tensor& x, const c10::optional<at::Tensor>& topk, const c10::optional<at::Tensor>& weights,
                            const std::vector<at::Tensor>& cached, int64_t cached_capacity, bool expand, int64_t alignment, const at::Tensor& w13,
                            const at::Tensor& w2, at::Tensor& status, const c10::optional<at::Tensor>& bias, bool fuse_combine,
                            bool allow_multiple_reduction, int64_t num_sms, int64_t comm_stream, double mailbox_timeout_s) {
    at::Tensor result;
    const auto behind = [&](DispatchOut& got, bool bound) {
        const auto& m = got.metadata[0];
        const at::Tensor &rows = got.outputs[0][0], &counts = m[1], &offsets = m[2];
        const auto gate = weights.has_value() ? c10::make_optional(got.outputs[0][2]) : c10::nullopt;
        const at::TensorOptions bf16 = rows.options();
        const int64_t tokens = x.size(0), most = std::max<int64_t>(1, bound ? tokens : got.counts[0].first);
        const int64_t assigned = bound ? tokens * window.layout().topk : -1;
        at::Tensor h = at::empty({rows.size(0), w13.size(1) / 2}, bf16);
        grouped_gemm(rows, w13, offsets, h, status, gemm::kSwiGLU, {}, {}, 0, 5.0, {}, 4, false, counts, most, got.early, assigned);
        if (fuse_combine) {
            grouped_gemm_scatter(window, h, w2, offsets, m[7], m[0], gate, status, 0, 5.0, counts, most, true, assigned);
            result = combine_finish({&window}, got.metadata, {bias})[0];
        } else {
            at::Tensor y = at::empty({rows.size(0), w2.size(1)}, bf16);
            grouped_gemm(h, w2, offsets, y, status, gemm::kPlain, {}, {}, 0, 5.0, gate, 4, false, counts, most, true, assigned);  // gate weight in FP32
            result = combine({&window}, {y}, got.metadata, {rows.size(0)}, {c10::nullopt}, {bias}, expand, allow_multiple_reduction, num_sms, comm_stream,
                             -1, false, bound).outputs[0][0];
        }
    };
    auto out = dispatch({&window}, {x}, {topk}, {weights}, {cached}, {cached_capacity}, alignment, expand, false, num_sms, comm_stream, -1, false,
                        mailbox_timeout_s, {c10::nullopt}, 0, behind, w13.size(1) / 2 * 2 + (fuse_combine ? 0 : w2.size(1) * 2));
    return pybind11::make_tuple(result, out.metadata[0], out.counts[0]);
}

}  // namespace

void bind_gemm(pybind11::module_& m) {
    m.def(
        "grouped_gemm", &grouped_gemm,
        pybind11::arg("a"), pybind11::arg("w"), pybind11::arg("expert_offsets"), pybind11::arg("out"), pybind11::arg("status"),
        pybind11::arg("mode"), pybind11::arg("tile_ready") = c10::nullopt, pybind11::arg("tile_expected") = c10::nullopt,
        pybind11::arg("max_ctas") = 0, pybind11::arg("timeout_s") = 5.0, pybind11::arg("row_scale") = c10::nullopt,
        pybind11::arg("stages") = 4, pybind11::arg("pair") = false, pybind11::arg("expert_counts") = c10::nullopt,
        pybind11::arg("max_expert_rows") = 0, pybind11::arg("early") = false, pybind11::arg("assigned") = -1);

    m.def(
        "grouped_gemm_scatter", &grouped_gemm_scatter,
        pybind11::arg("window"), pybind11::arg("a"), pybind11::arg("w"), pybind11::arg("expert_offsets"),
        pybind11::arg("slot_map"), pybind11::arg("recv_metadata"), pybind11::arg("slot_weights"), pybind11::arg("status"),
        pybind11::arg("max_ctas") = 0, pybind11::arg("timeout_s") = 5.0,
        pybind11::arg("expert_counts") = c10::nullopt, pybind11::arg("max_expert_rows") = 0, pybind11::arg("early") = false, pybind11::arg("assigned") = -1);

    m.def("moe_forward", &moe_forward);
    m.def(
        "grouped_gemm_choice",
        [](bool gated, bool pair, int64_t stages, int64_t max_ctas, bool swiglu, bool counts, int64_t rows, int64_t n, int64_t k, int64_t sms) -> std::string {
            const Kernel kernel = choose_kernel(Choice{gated, pair, stages, max_ctas, swiglu, counts, rows / 128, n / 256, k, sms});
            return kernel == kExpertKernel ? "expert" : kernel == kPairKernel ? "pair" : "single";
        },
        pybind11::arg("gated") = false, pybind11::arg("pair") = false, pybind11::arg("stages") = 4, pybind11::arg("max_ctas") = 0,
        pybind11::arg("swiglu") = false, pybind11::arg("counts") = false, pybind11::arg("rows") = 1 << 16, pybind11::arg("n") = 4096,
        pybind11::arg("k") = 4096, pybind11::arg("sms") = 148,
        "Kernel that a grouped_gemm call with these arguments runs");
    m.def("gemm_kernel_registers", [](int64_t mode) { return gemm::kernel_registers(int(mode)); });
    m.def("gemm_shared_bytes", [](int64_t stages) { return int64_t(gemm::shared_bytes(int(stages))); });
}

}  // namespace nep
