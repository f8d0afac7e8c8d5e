// Bindings of the one-rank paths.  They allocate their results and launch in one call, so that a call costs the host a few
// allocations and launches instead of a Python pipeline.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <pybind11/stl.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/custom_class.h>
#include <torch/extension.h>

#include <array>
#include <atomic>
#include <climits>
#include <memory>
#include <mutex>

#include "launch_count.h"
#include "local.h"
#include "local_layer.h"
#include "lowlat.h"

namespace {

#define TM_CHECK_CUDA(call)                                                                          \
    do {                                                                                             \
        tmoe::count_launch();                                                                        \
        cudaError_t _e = (call);                                                                     \
        TORCH_CHECK(_e == cudaSuccess, "teramoe_b200: ", #call, " failed: ", cudaGetErrorString(_e)); \
    } while (0)

cudaStream_t cur_stream() { return at::cuda::getCurrentCUDAStream().stream(); }

struct TopK {
    const void* ptr;
    int is64, T, K;
};
TopK topk_of(const torch::Tensor& idx) {
    TORCH_CHECK(idx.is_cuda() && idx.is_contiguous() && idx.dim() == 2, "topk_idx must be a contiguous [T,K] CUDA tensor");
    TORCH_CHECK(idx.scalar_type() == torch::kInt64 || idx.scalar_type() == torch::kInt32, "topk_idx must be int64 or int32");
    TORCH_CHECK(idx.size(1) <= 32, "top-k must be <= 32");
    return TopK{idx.data_ptr(), idx.scalar_type() == torch::kInt64 ? 1 : 0, (int)idx.size(0), (int)idx.size(1)};
}
torch::Tensor weights_of(const torch::Tensor& w) {
    auto f = w.scalar_type() == torch::kFloat32 ? w : w.to(torch::kFloat32);
    return f.contiguous();
}
bool aligned16(const torch::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
torch::TensorOptions on(const torch::Tensor& like, torch::ScalarType t) { return torch::TensorOptions().dtype(t).device(like.device()); }

// The plain form of a call runs on the caller's stream and the asynchronous one on the communication stream, so a call may use tables of a
// handle that another stream writes.  It waits for them there (for `mark`, or else for whatever that stream holds by then), and the
// allocator keeps their memory until it is done with them, whenever the handle goes.
unsigned long long capture_of(const c10::cuda::CUDAStream& s) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    const cudaError_t e = cudaStreamGetCaptureInfo(s.stream(), &status, &id);
    TORCH_CHECK(e == cudaSuccess, "teramoe_b200: ", cudaGetErrorString(e));
    return status == cudaStreamCaptureStatusNone ? 0 : id;
}
void use_tables(const c10::cuda::CUDAStream& writer, unsigned long long capture, at::cuda::CUDAEvent* mark, std::initializer_list<torch::Tensor> tables) {
    const auto stream = c10::cuda::getCurrentCUDAStream();
    if (stream == writer) return;
    for (const auto& t : tables) c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), stream);
    // a graph does not wait for what was enqueued outside it, nor the other way round
    if (capture_of(stream) != capture) return;
    if (mark != nullptr) return mark->block(stream);
    if (capture_of(writer) != capture) return;
    at::cuda::CUDAEvent now;
    now.record(writer);
    now.block(stream);
}

// A tensor of its own over part of another one's memory, from byte `at` on.  An allocation costs the host about a microsecond, this a tenth of it: the
// tables of one handle, and the counts of one layout, lie in one block.  It lives as long as any of them, is saved or shared with another process as a
// whole, and resizing one of them would take its neighbour's memory: what a program keeps, saves or changes by itself has an allocation of its own.
torch::Tensor piece(const torch::Tensor& block, int64_t at, at::IntArrayRef sizes, at::ScalarType type) {
    auto t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(block.storage()), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                      c10::scalarTypeToTypeMeta(type));
    t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
    t.unsafeGetTensorImpl()->set_storage_offset(at / (int64_t)c10::elementSize(type));
    return t;
}

// Memory that the kernels of this call write in full, past torch.empty's dispatcher (which adds to the host's time what the allocation itself takes)
torch::Tensor written(at::IntArrayRef sizes, const torch::Tensor& like, at::ScalarType type) {
    return torch::Tensor(at::detail::empty_cuda(sizes, type, like.device(), c10::nullopt));
}

// Where the next part of a block starts: on a boundary as an allocation has it.
int64_t behind(int64_t at, int64_t bytes) { return (at + bytes + 511) / 512 * 512; }

// ------------------------------------------------------------------------------------------------ low latency
// The statistics of waits are accepted as the window kernels accept them and left as they are: nothing is waited for here.
void check_wait_stats(const c10::optional<torch::Tensor>& t) {
    TORCH_CHECK(!t.has_value() || (t->is_cuda() && t->scalar_type() == torch::kInt64 && t->is_contiguous()),
                "wait_stats must be a contiguous int64 CUDA tensor");
}

tmoe::LowLatLayout local_layout(int64_t E, int64_t M, int64_t H, int wire, bool logfmt) {
    tmoe::LowLatLayout l{};
    l.num_ranks = 1; l.num_experts = (int)E; l.max_tokens = (int)M; l.hidden = (int)H;
    l.use_fp8 = wire > 0; l.round_scale = wire > 1; l.use_ue8m0 = wire > 2; l.use_logfmt = logfmt ? 1 : 0;
    l.d_msg_bytes = 16; l.c_row_bytes = 16;
    return l;
}

// wire: 0 bf16, 1 e4m3 + fp32 scales, 2 power-of-two scales, 3 scales packed as UE8M0 bytes
// -> (recv_x [E,M,H], scales (transposed view of [E,groups,M]) or None, count [E], src_info [E,M], layout_range [E,1], entry_row [T,K],
//     id of the stream that writes it)
std::tuple<torch::Tensor, c10::optional<torch::Tensor>, torch::Tensor, torch::Tensor, torch::Tensor, torch::Tensor, int64_t>
ll_local_dispatch(torch::Tensor x, torch::Tensor topk_idx, int64_t M, int64_t E, int64_t wire, c10::optional<torch::Tensor> expert_stats,
                  c10::optional<torch::Tensor> wait_stats) {
    c10::cuda::CUDAGuard guard(x.device());
    check_wait_stats(wait_stats);
    x = x.contiguous();
    topk_idx = topk_idx.contiguous();
    const TopK tk = topk_of(topk_idx);
    TORCH_CHECK(x.is_cuda() && x.scalar_type() == torch::kBFloat16 && x.dim() == 2 && x.size(0) == tk.T, "x must be a bf16 [T, hidden] CUDA tensor");
    TORCH_CHECK(aligned16(x), "x must start on a 16-byte boundary");          // (rows are read 16 bytes at a time)
    int* stats = nullptr;
    if (expert_stats.has_value()) {
        TORCH_CHECK(expert_stats->is_cuda() && expert_stats->scalar_type() == torch::kInt32 && expert_stats->is_contiguous() &&
                    expert_stats->numel() >= E, "expert_stats must be a contiguous int32 CUDA tensor of one word per expert");
        stats = expert_stats->data_ptr<int>();
    }
    const int64_t H = x.size(1), G = H / 128;
    auto recv = torch::empty({E, M, H}, on(x, wire > 0 ? torch::kFloat8_e4m3fn : torch::kBFloat16));
    c10::optional<torch::Tensor> scales;
    if (wire > 0) scales = wire == 3 ? torch::empty({E, G / 4, M}, on(x, torch::kInt32)) : torch::empty({E, G, M}, on(x, torch::kFloat32));
    const auto count = written({E}, x, torch::kInt32);          // (a program keeps it without the handle)
    const int64_t at_src = behind(0, 8 * E), at_entry = behind(at_src, 4 * E * M);
    const auto block = torch::empty({at_entry + 4 * (int64_t)tk.T * tk.K}, on(x, torch::kUInt8));      // (src_info is not written in full)
    const auto range = piece(block, 0, {E, 1}, torch::kInt64), src_info = piece(block, at_src, {E, M}, torch::kInt32);
    const auto entry = piece(block, at_entry, {tk.T, tk.K}, torch::kInt32);
    TM_CHECK_CUDA(tmoe::ll_local_dispatch(local_layout(E, M, H, (int)wire, false), x.data_ptr(), tk.ptr, tk.is64, tk.T, tk.K, recv.data_ptr(),
                                          scales.has_value() ? scales->data_ptr() : nullptr, src_info.data_ptr<int>(),
                                          reinterpret_cast<long long*>(range.data_ptr<int64_t>()), count.data_ptr<int>(), stats,
                                          entry.data_ptr<int>(), cur_stream()));
    if (scales.has_value()) {
        // [E, M, groups] over column-major memory
        const int64_t groups = scales->size(1), sizes[3] = {E, M, groups}, strides[3] = {groups * M, 1, M};
        scales->unsafeGetTensorImpl()->set_sizes_and_strides(sizes, strides);
    }
    return {recv, scales, count, src_info, range, entry, c10::cuda::getCurrentCUDAStream().id()};
}

torch::Tensor ll_local_combine(torch::Tensor x, torch::Tensor topk_idx, torch::Tensor topk_weights, torch::Tensor entry_row,
                               int64_t writer, int64_t M, int64_t E, int64_t H, bool logfmt, c10::optional<torch::Tensor> out,
                               c10::optional<torch::Tensor> wait_stats) {
    c10::cuda::CUDAGuard guard(x.device());
    check_wait_stats(wait_stats);
    const auto w_stream = c10::cuda::CUDAStream::unpack3(writer, x.device().index(), c10::DeviceType::CUDA);
    if (w_stream != c10::cuda::getCurrentCUDAStream()) use_tables(w_stream, capture_of(w_stream), nullptr, {entry_row});
    x = x.contiguous();
    topk_idx = topk_idx.contiguous();
    const TopK tk = topk_of(topk_idx);
    const auto w = weights_of(topk_weights);
    TORCH_CHECK(x.is_cuda() && x.scalar_type() == torch::kBFloat16 && x.numel() == E * M * H, "x must be bf16 [E_local, ranks*max_tokens, hidden]");
    TORCH_CHECK(w.is_cuda() && w.numel() == (int64_t)tk.T * tk.K, "topk_weights must have one weight per entry");
    if (!out.has_value()) out = torch::empty({tk.T, H}, on(x, torch::kBFloat16));
    TORCH_CHECK(out->is_cuda() && out->scalar_type() == torch::kBFloat16 && out->is_contiguous() && out->dim() == 2 && out->size(0) == tk.T &&
                out->size(1) == H, "out must be a contiguous bf16 [T, hidden] CUDA tensor");
    TORCH_CHECK(aligned16(x) && aligned16(*out), "x and out must start on a 16-byte boundary");
    TM_CHECK_CUDA(tmoe::ll_local_combine(local_layout(E, M, H, 0, logfmt), x.data_ptr(), tk.ptr, tk.is64, w.data_ptr<float>(),
                                         entry_row.data_ptr<int>(), tk.T, tk.K, (int)entry_row.size(0), (int)entry_row.size(1), out->data_ptr(),
                                         cur_stream()));
    return *out;
}

// ------------------------------------------------------------------------------------------------ un-fused exchange
struct Scratch {
    torch::Tensor all;                       // int32: totals [E + 2], row_local [T], chunk_base, and, with `rows`, [T] more
    int *totals, *row_local, *chunk_base;
    int64_t extra;                           // byte of the last part
};
Scratch route_scratch(const torch::Tensor& idx, const TopK& tk, int64_t E, bool rows) {
    const int64_t chunks = std::max<int64_t>(1, (tk.T + tmoe::kLocalChunk - 1) / tmoe::kLocalChunk);
    Scratch s;
    s.extra = behind(0, 4 * (E + 2 + tk.T + chunks));
    s.all = written({s.extra / 4 + (rows ? tk.T : 0)}, idx, torch::kInt32);
    s.totals = s.all.data_ptr<int>();
    s.row_local = s.totals + E + 2;
    s.chunk_base = s.row_local + tk.T;
    return s;
}

tmoe::LocalPart part(const torch::Tensor& src, const torch::Tensor& dst) {
    return tmoe::LocalPart{src.data_ptr(), dst.data_ptr(), (uint32_t)(src.size(1) * src.element_size())};
}

// -> (tokens [1], tokens per expert [E], is_token_in_rank [T,1])
std::tuple<torch::Tensor, torch::Tensor, torch::Tensor> local_counts(torch::Tensor topk_idx, int64_t E) {
    c10::cuda::CUDAGuard guard(topk_idx.device());
    topk_idx = topk_idx.contiguous();
    const TopK tk = topk_of(topk_idx);
    const auto s = route_scratch(topk_idx, tk, E, false);
    const auto in_rank = written({tk.T, 1}, topk_idx, torch::kBool);
    TM_CHECK_CUDA(tmoe::local_route(tk.ptr, tk.is64, tk.T, tk.K, (int)E, s.totals, s.row_local, s.chunk_base,
                                    reinterpret_cast<uint8_t*>(in_rank.data_ptr<bool>()), nullptr, 0, cur_stream()));
    return {piece(s.all, 4 * E, {1}, torch::kInt32), piece(s.all, 0, {E}, torch::kInt32), in_rank};
}

// Events of dropped layouts, for the next ones: creating and destroying one costs about as much as recording it.
struct Marks {
    static constexpr size_t kMost = 16;
    std::mutex mutex;
    std::vector<at::cuda::CUDAEvent> spare;
    at::cuda::CUDAEvent take() {
        std::lock_guard<std::mutex> lock(mutex);
        if (spare.empty()) return at::cuda::CUDAEvent();
        at::cuda::CUDAEvent e = std::move(spare.back());
        spare.pop_back();
        return e;
    }
    void give(at::cuda::CUDAEvent&& e) {
        std::lock_guard<std::mutex> lock(mutex);
        if (e.isCreated() && spare.size() < kMost) spare.push_back(std::move(e));
    }
};

// What a dispatch leaves for the calls on its handle: where the tokens' rows are, the totals, and the stream that writes both.
struct LocalLayout {
    LocalLayout() = default;
    LocalLayout(const LocalLayout&) = delete;
    ~LocalLayout() {
        if (marks != nullptr) marks->give(std::move(written));
    }

    torch::Tensor send_row, scratch;         // [T]; [E + 1] and more: entries per expert, rows
    int64_t E = 0;
    c10::cuda::CUDAStream writer = c10::cuda::getCurrentCUDAStream();
    unsigned long long capture = capture_of(writer);
    std::shared_ptr<Marks> marks;
    at::cuda::CUDAEvent written;             // recorded where `mark` was called

    // Not called in a graph, nor for a plain call of known size: that one is on the caller's stream, which those who go on with its handle on
    // another one usually wait for anyway.
    void mark(std::shared_ptr<Marks> m) {
        marks = std::move(m);
        written = marks->take();
        written.record(writer);
    }
    void use(std::initializer_list<torch::Tensor> tables) { use_tables(writer, capture, marks != nullptr ? &written : nullptr, tables); }
    // The number of rows, for whoever asks, from any stream and without waiting for what was enqueued since.  Of a dispatch inside a graph,
    // that of the last replay.
    int64_t rows() {
        c10::cuda::CUDAGuard guard(scratch.device());
        const torch::Tensor n = scratch.narrow(0, E, 1);
        if (marks == nullptr) return n.item<int>();
        const auto side = c10::cuda::getStreamFromPool();
        c10::cuda::CUDAStreamGuard on_side(side);
        written.block(side);
        return n.item<int>();
    }
};

// The one piece of host state: a pinned block that local_route writes the counts into, each with the number of the call.
class LocalExchange {
  public:
    // -> (received payloads, recv_idx, recv_w, counts per expert rounded up to `alignment` (empty with worst_rows), rows (-1: not read),
    //     layout)
    py::tuple dispatch(std::vector<torch::Tensor> parts, torch::Tensor topk_idx, torch::Tensor topk_weights, int64_t E, int64_t worst_rows,
                       int64_t alignment, bool mark) {
        std::vector<torch::Tensor> recv;
        torch::Tensor idx_out, w_out;
        std::shared_ptr<LocalLayout> layout;
        std::vector<int64_t> counts;
        int64_t rows = -1;
        {
            py::gil_scoped_release nogil;
            c10::cuda::CUDAGuard guard(topk_idx.device());
            std::lock_guard<std::mutex> lock(mutex_);
            const cudaStream_t stream = cur_stream();
            topk_idx = topk_idx.contiguous();
            const TopK tk = topk_of(topk_idx);
            const auto w = weights_of(topk_weights);
            TORCH_CHECK(w.is_cuda() && w.numel() == (int64_t)tk.T * tk.K, "topk_weights must have one weight per entry");
            TORCH_CHECK(!parts.empty() && parts.size() <= tmoe::kLocalMaxParts, "one or two payloads");
            const auto s = route_scratch(topk_idx, tk, E, true);
            const int64_t cap = worst_rows > 0 ? worst_rows : tk.T;
            std::vector<tmoe::LocalPart> lp;
            for (auto& p : parts) {
                p = p.contiguous();
                TORCH_CHECK(p.is_cuda() && p.dim() == 2 && p.size(0) == tk.T, "payloads must be [T, C] CUDA tensors");
                recv.push_back(torch::empty({cap, p.size(1)}, p.options()));
                lp.push_back(part(p, recv.back()));
            }
            idx_out = torch::empty({cap, tk.K}, topk_idx.options());
            w_out = torch::empty({cap, tk.K}, w.options());
            const auto send_row = piece(s.all, s.extra, {tk.T}, torch::kInt32);
            const bool wait = worst_rows <= 0;
            if (wait) host_block(E + 1);
            TM_CHECK_CUDA(tmoe::local_route(tk.ptr, tk.is64, tk.T, tk.K, (int)E, s.totals, s.row_local, s.chunk_base, nullptr,
                                            wait ? host_words() : nullptr, seq_, stream));
            TM_CHECK_CUDA(tmoe::local_dispatch(lp.data(), (int)lp.size(), tk.ptr, tk.is64, w.data_ptr<float>(), tk.T, tk.K, (int)E, s.totals,
                                               s.row_local, s.chunk_base, send_row.data_ptr<int>(), idx_out.data_ptr(), w_out.data_ptr<float>(),
                                               (int)std::max<int64_t>(worst_rows, 0), stream));
            layout = std::make_shared<LocalLayout>();
            layout->send_row = send_row;
            layout->scratch = s.all;
            layout->E = E;
            // the handle keeps the indices, which another stream may have made
            c10::cuda::CUDACachingAllocator::recordStream(topk_idx.storage().data_ptr(), layout->writer);
            if ((mark || !wait) && layout->capture == 0) layout->mark(marks_);
            if (wait) {
                // the rows are being copied while the host waits for the counts
                rows = await_count(0, stream);
                counts.resize(E);
                for (int64_t e2 = 0; e2 < E; ++e2) counts[e2] = (await_count(1 + e2, stream) + alignment - 1) / alignment * alignment;
                if (rows < cap) {
                    for (auto& r : recv) r = r.narrow(0, 0, rows);
                    idx_out = idx_out.narrow(0, 0, rows);
                    w_out = w_out.narrow(0, 0, rows);
                }
            }
        }
        return py::make_tuple(recv, idx_out, w_out, counts, rows, layout);
    }

  private:
    void host_block(int64_t n) {
        if (!host_.defined() || host_.numel() < n)
            host_ = torch::zeros({n}, torch::TensorOptions().dtype(torch::kInt64).pinned_memory(true));
        seq_ = seq_ == INT_MAX ? 1 : seq_ + 1;
    }
    unsigned long long* host_words() const { return reinterpret_cast<unsigned long long*>(host_.data_ptr<int64_t>()); }
    // A count, when the kernel has written it.  The stream is asked now and then, so that a failed launch raises and does not spin.
    int64_t await_count(int64_t i, cudaStream_t stream) const {
        const unsigned long long* word = host_words() + i;
        for (int spins = 1;; ++spins) {
            unsigned long long v = __atomic_load_n(word, __ATOMIC_ACQUIRE);
            if ((v >> 32) == (unsigned long long)seq_) return (int64_t)(v & 0xffffffffull);
            if (spins % 20000 != 0) continue;
            const cudaError_t e = cudaStreamQuery(stream);
            TORCH_CHECK(e == cudaSuccess || e == cudaErrorNotReady, "teramoe_b200: dispatch failed: ", cudaGetErrorString(e));
            v = __atomic_load_n(word, __ATOMIC_ACQUIRE);
            TORCH_CHECK(e == cudaErrorNotReady || (v >> 32) == (unsigned long long)seq_, "teramoe_b200: dispatch wrote no counts");
        }
    }
    std::mutex mutex_;
    std::shared_ptr<Marks> marks_ = std::make_shared<Marks>();
    torch::Tensor host_;
    int seq_ = 0;
};

// A dispatch whose layout is known: payload rows of the tokens that have a row.
std::vector<torch::Tensor> local_scatter(std::vector<torch::Tensor> parts, const std::shared_ptr<LocalLayout>& layout, int64_t rows) {
    const torch::Tensor& send_row = layout->send_row;
    c10::cuda::CUDAGuard guard(send_row.device());
    layout->use({send_row});
    std::vector<torch::Tensor> recv;
    std::vector<tmoe::LocalPart> lp;
    const int64_t T = send_row.numel();
    TORCH_CHECK(!parts.empty() && parts.size() <= tmoe::kLocalMaxParts, "one or two payloads");
    for (auto& p : parts) {
        p = p.contiguous();
        TORCH_CHECK(p.is_cuda() && p.dim() == 2 && p.size(0) == T, "payloads must be [T, C] CUDA tensors");
        recv.push_back(torch::empty({rows, p.size(1)}, p.options()));
        lp.push_back(part(p, recv.back()));
    }
    TM_CHECK_CUDA(tmoe::local_move(lp.data(), (int)lp.size(), send_row.data_ptr<int>(), (int)T, rows, 1, nullptr, 0, 0, 0, nullptr,
                                   nullptr, cur_stream()));
    return recv;
}

// out[t] = row send_row[t] of x (zeros for tokens that went nowhere) and, with weights [rows, K], the entries' weights [T, K].
// x and weights may have more rows, and weights more columns, than the dispatch sent.
std::tuple<torch::Tensor, c10::optional<torch::Tensor>> local_combine(torch::Tensor x, const std::shared_ptr<LocalLayout>& layout, int64_t rows,
                                                                      torch::Tensor topk_idx, int64_t E, c10::optional<torch::Tensor> weights) {
    const torch::Tensor& send_row = layout->send_row;
    c10::cuda::CUDAGuard guard(x.device());
    layout->use({send_row, topk_idx});
    x = x.contiguous();
    const TopK tk = topk_of(topk_idx);
    TORCH_CHECK(x.is_cuda() && x.scalar_type() == torch::kBFloat16 && x.dim() == 2 && x.size(0) >= rows, "x must be a bf16 [rows, H] CUDA tensor");
    TORCH_CHECK(send_row.numel() == tk.T, "the handle is one of another routing");
    auto out = torch::empty({tk.T, x.size(1)}, x.options());
    c10::optional<torch::Tensor> w_out;
    torch::Tensor w;
    if (weights.has_value()) {
        TORCH_CHECK(weights->device() == x.device() && weights->dim() == 2 && weights->size(0) >= rows && weights->size(1) >= tk.K,
                    "topk_weights must be a [rows, K] tensor on the device of x, as the dispatch returned it");
        w = weights_of(weights->size(1) == tk.K ? *weights : weights->narrow(1, 0, tk.K));
        w_out = torch::empty({tk.T, tk.K}, w.options());
    }
    const tmoe::LocalPart p = part(x, out);
    TM_CHECK_CUDA(tmoe::local_move(&p, 1, send_row.data_ptr<int>(), tk.T, rows, 0, tk.ptr, tk.is64, tk.K, (int)E,
                                   w.defined() ? w.data_ptr<float>() : nullptr, w_out.has_value() ? w_out->data_ptr<float>() : nullptr, cur_stream()));
    return {out, w_out};
}

// ------------------------------------------------------------------------------------------------ layer
int64_t layer_rows(const tmoe::LocalLayerPlan& plan) { return std::max(plan.slots_cap, 128); }

// bytes of the arena that a call with these sizes uses: expert outputs in slot order
int64_t local_layer_arena_bytes(int64_t T, int64_t K, int64_t E, int64_t H) {
    return layer_rows(tmoe::local_layer_plan((int)T, (int)K, (int)E, (int)H, 64, 0)) * H * 2;
}

// which kernels a call with these sizes runs, for tests that are about one of them
py::dict local_layer_variant(int64_t T, int64_t K, int64_t E, int64_t H, int64_t I, bool keep) {
    const tmoe::LocalLayerPlan p = tmoe::local_layer_plan((int)T, (int)K, (int)E, (int)H, (int)I, keep ? 1 : 0);
    py::dict d;
    d["few"] = p.few;
    d["copies_forward"] = p.copies[0] != 0;
    d["copies_backward"] = p.copies[1] != 0;
    return d;
}

// columns per tile, for tests that are about wide ones: [direction][first GEMM, second GEMM, dW_down, dW_gateup]
std::vector<std::vector<int>> local_layer_columns(int64_t T, int64_t K, int64_t E, int64_t H, int64_t I) {
    const tmoe::LocalLayerPlan p = tmoe::local_layer_plan((int)T, (int)K, (int)E, (int)H, (int)I, 1);
    return {{p.cols[0][0], p.cols[0][1]}, {std::begin(p.cols[1]), std::end(p.cols[1])}};
}

// whether units of one 128-row block are multiplied as 128 rows
bool local_layer_halves(int64_t T, int64_t K, int64_t E, int64_t H, int64_t I) {
    return tmoe::local_layer_plan((int)T, (int)K, (int)E, (int)H, (int)I, 0).halves != 0;
}

void check_layer_weights(const torch::Tensor& wg, const torch::Tensor& wd, int64_t E, int64_t H, int64_t I) {
    TORCH_CHECK(wg.is_cuda() && wg.scalar_type() == torch::kBFloat16 && wg.is_contiguous() && wg.dim() == 3 && wg.size(0) == E &&
                wg.size(1) == 2 * I && wg.size(2) == H, "W_gateup must be a contiguous bf16 [E, 2I, H] CUDA tensor");
    TORCH_CHECK(wd.is_cuda() && wd.scalar_type() == torch::kBFloat16 && wd.is_contiguous() && wd.dim() == 3 && wd.size(0) == E &&
                wd.size(1) == H && wd.size(2) == I, "W_down must be a contiguous bf16 [E, H, I] CUDA tensor");
}

// What the calls of one buffer share: the arena (expert outputs in slot order), the status block and its copy in pinned
// memory, and the workspaces of the last forward and backward for whoever asks for their statistics.
class LocalLayer : public std::enable_shared_from_this<LocalLayer> {
  public:
    using Schedule = std::array<int64_t, 4>;      // units per batch, lag percent, least lag in items, SMs

    LocalLayer(torch::Tensor status, torch::Tensor status_host) : status_(status), host_(status_host) {}

    // Returns when no thread is about to launch on the arena before: what is launched later uses the new one.
    void set_arena(int64_t ptr, int64_t bytes) {
        std::lock_guard<std::mutex> lock(arena_mutex_);
        arena_ = ptr;
        arena_bytes_ = bytes;
    }
    int64_t arena() const {
        std::lock_guard<std::mutex> lock(arena_mutex_);
        return arena_;
    }
    void close() { open_ = false; }

    // The conditions under which the kernels take a call; anything else is for the caller's slow path, which also names what is wrong.
    bool takes(const torch::Tensor& x, const torch::Tensor& idx, const torch::Tensor& w, const torch::Tensor& wg, const torch::Tensor& wd,
               int64_t num_experts) const {
        if (!(x.is_cuda() && idx.is_cuda() && w.is_cuda() && wg.is_cuda() && wd.is_cuda())) return false;
        if (x.dim() != 2 || idx.dim() != 2 || wg.dim() != 3 || wd.dim() != 3 || w.sizes() != idx.sizes() || idx.size(0) != x.size(0)) return false;
        if (x.scalar_type() != torch::kBFloat16 || wg.scalar_type() != torch::kBFloat16 || wd.scalar_type() != torch::kBFloat16 ||
            w.scalar_type() != torch::kFloat32 || (idx.scalar_type() != torch::kInt64 && idx.scalar_type() != torch::kInt32))
            return false;
        if (!(x.is_contiguous() && idx.is_contiguous() && w.is_contiguous() && wg.is_contiguous() && wd.is_contiguous())) return false;
        const int64_t E = wg.size(0), H = x.size(1), I = wd.size(2);
        return E == num_experts && E >= 1 && E <= tmoe::kLocalMaxExperts && wg.size(1) == 2 * I && wg.size(2) == H && wd.size(0) == E && wd.size(1) == H &&
               H % 64 == 0 && I % 64 == 0 && idx.size(1) >= 1 && idx.size(1) <= 32;
    }
    // bytes of the arena that a call needs, 0 if it has them
    int64_t wants(int64_t T, int64_t K, int64_t E, int64_t H) const {
        const int64_t need = local_layer_arena_bytes(T, K, E, H);
        std::lock_guard<std::mutex> lock(arena_mutex_);
        return need > arena_bytes_ ? need : 0;
    }

    // Forward and backward passes so far: each writes over the arena, a backward pass without anybody in Python being told.
    int64_t launches() const {
        std::lock_guard<std::mutex> lock(arena_mutex_);
        return launches_;
    }

    // strict: wait for the call's kernels, so that the call whose wait ran out is the one that raises
    void settle(bool strict) {
        if (!strict) return;
        const cudaError_t e = cudaStreamSynchronize(cur_stream());
        TORCH_CHECK(e == cudaSuccess, "teramoe_b200: ", cudaGetErrorString(e));
        check();
    }
    void check() {
        TORCH_CHECK(open_, "Buffer was destroyed");
        volatile int* h = host_.data_ptr<int>();
        if (h[0] == 0) return;
        static const char* names[] = {"", "mbarrier wait", "flag wait", "barrier", "bad argument"};
        const int code = h[0], site = h[1], block = h[2], detail = h[3];
        status_.narrow(0, 0, 4).zero_();
        h[0] = 0;
        TORCH_CHECK(false, "teramoe_b200: a device-side wait ran out on rank 0: ", code >= 1 && code <= 4 ? names[code] : "?", " (site ", site,
                    ", block ", block, ", detail ", detail, ")");
    }

    struct Kept {
        torch::Tensor ws, rows;       // rows: x [T, H], then the pre-activation of every slot (2I values)
    };

    torch::Tensor forward(const torch::Tensor& x, const torch::Tensor& topk_idx, const torch::Tensor& topk_w, const torch::Tensor& w_gateup,
                          const torch::Tensor& w_down, const Schedule& schedule, Kept* kept) {
        check();
        c10::cuda::CUDAGuard guard(x.device());
        const TopK tk = topk_of(topk_idx);
        const int64_t E = w_gateup.size(0), H = x.size(1), I = w_gateup.size(1) / 2;
        TORCH_CHECK(x.is_cuda() && x.scalar_type() == torch::kBFloat16 && x.is_contiguous() && x.dim() == 2 && x.size(0) == tk.T, "x must be a contiguous bf16 [T, H] CUDA tensor");
        TORCH_CHECK(topk_w.is_cuda() && topk_w.scalar_type() == torch::kFloat32 && topk_w.is_contiguous() && topk_w.numel() == (int64_t)tk.T * tk.K,
                    "topk_weights must be a contiguous fp32 [T, K] CUDA tensor");
        check_layer_weights(w_gateup, w_down, E, H, I);
        tmoe::LocalLayerParams p{};
        p.plan = tmoe::local_layer_plan(tk.T, tk.K, (int)E, (int)H, (int)I, kept != nullptr ? 1 : 0);
        const int64_t rows = layer_rows(p.plan);
        auto ws = torch::empty({p.plan.words}, on(x, torch::kInt32));
        auto out = torch::empty({tk.T, H}, x.options());
        // act [rows, I] and, with copies, x in slot order [rows, H]
        auto act = torch::empty({rows * (I + (p.plan.copies[0] ? H : 0))}, x.options());
        if (kept != nullptr) {
            kept->ws = ws;
            kept->rows = torch::empty({tk.T * H + rows * 2 * I}, x.options());
            p.saved_x = kept->rows.data_ptr();
            p.preact = kept->rows.data_ptr<at::BFloat16>() + tk.T * H;
        }
        p.ws = ws.data_ptr<int>();
        p.topk_idx = tk.ptr; p.idx_is64 = tk.is64; p.topk_w = topk_w.data_ptr<float>();
        p.x = x.data_ptr(); p.w_gateup = w_gateup.data_ptr(); p.w_down = w_down.data_ptr();
        p.act = act.data_ptr(); p.out = out.data_ptr();
        if (p.plan.copies[0]) p.slot_rows = act.data_ptr<at::BFloat16>() + rows * I;
        const cudaStream_t stream = cur_stream();
        {
            std::lock_guard<std::mutex> lock(arena_mutex_);
            set_common(p, schedule);
            if (!p.plan.routes) TM_CHECK_CUDA(tmoe::local_layer_route(p, stream));
            TM_CHECK_CUDA(tmoe::local_layer_launch(p, stream));
        }
        note(0, ws, p.plan);
        return out;
    }

    // -> dx [T,H], d(topk_weights) [T,K], dW_gateup, dW_down
    std::array<torch::Tensor, 4> backward(const torch::Tensor& grad_out, const Kept& kept, const torch::Tensor& w_gateup, const torch::Tensor& w_down,
                                          int64_t K, const Schedule& schedule) {
        check();
        c10::cuda::CUDAGuard guard(grad_out.device());
        const int64_t E = w_gateup.size(0), T = grad_out.size(0), H = w_gateup.size(2), I = w_gateup.size(1) / 2;
        TORCH_CHECK(grad_out.is_cuda() && grad_out.scalar_type() == torch::kBFloat16 && grad_out.is_contiguous() && grad_out.dim() == 2 &&
                    grad_out.size(1) == H, "grad_out must be a contiguous bf16 [T, H] CUDA tensor");
        check_layer_weights(w_gateup, w_down, E, H, I);
        tmoe::LocalLayerParams p{};
        p.plan = tmoe::local_layer_plan((int)T, (int)K, (int)E, (int)H, (int)I, 1);
        const int64_t rows = layer_rows(p.plan);
        TORCH_CHECK(kept.ws.numel() == p.plan.words && kept.rows.numel() == T * H + rows * 2 * I && kept.rows.device() == grad_out.device() &&
                    kept.rows.scalar_type() == torch::kBFloat16 && kept.rows.is_contiguous() && aligned16(kept.rows),
                    "saved tensors of another call");
        // act x route [rows, I], dGU [rows, 2I], grad_out and x in slot order [rows, H] (with copies), partial sums of d(route weight): one
        // allocation (rows and I, H are multiples of 64: every part starts on a 16-byte boundary)
        const int64_t copied = p.plan.copies[1] ? 2 * H : 0;
        auto scratch = torch::empty({rows * (3 * I + copied + 4 * ((I + 255) / 256))}, grad_out.options());
        auto* act_w = scratch.data_ptr<at::BFloat16>();
        auto* dgu = act_w + rows * I;
        auto* slot_rows = dgu + rows * 2 * I;
        auto* parts = slot_rows + rows * copied;
        if (copied != 0) {
            p.slot_rows = slot_rows;
            p.slot_x = slot_rows + rows * H;
        }
        auto dx = torch::empty({T, H}, grad_out.options());
        auto dw = torch::empty({T, K}, on(grad_out, torch::kFloat32));
        auto dwg = torch::empty({E, 2 * I, H}, grad_out.options());
        auto dwd = torch::empty({E, H, I}, grad_out.options());
        p.ws = kept.ws.data_ptr<int>();
        p.bwd = 1;
        p.x = grad_out.data_ptr(); p.w_gateup = w_gateup.data_ptr(); p.w_down = w_down.data_ptr();
        p.act = act_w; p.aux = dgu; p.saved_x = kept.rows.data_ptr(); p.out = dx.data_ptr();
        p.preact = kept.rows.data_ptr<at::BFloat16>() + T * H; p.droute_part = reinterpret_cast<float*>(parts);
        p.dw_topk = dw.data_ptr<float>(); p.dw_gateup = dwg.data_ptr(); p.dw_down = dwd.data_ptr();
        {
            std::lock_guard<std::mutex> lock(arena_mutex_);
            set_common(p, schedule);
            TM_CHECK_CUDA(tmoe::local_layer_launch(p, cur_stream()));
        }
        note(1, kept.ws, p.plan);
        return {dx, dw, dwg, dwd};
    }

    // statistics words of the last forward (0) / backward (1), None before the first
    c10::optional<torch::Tensor> stats(int64_t dir) {
        std::lock_guard<std::mutex> lock(mutex_);
        if (!last_[dir].defined()) return c10::nullopt;
        return last_[dir].narrow(0, last_at_[dir], 48).view(torch::kInt64);
    }
    // whether the last forward ran in local_few.cu, and the rows of a unit there (read the workspace back)
    bool ran_few() { return last_meta(tmoe::kMetaFew) != 0; }
    int64_t few_unit() { return last_meta(tmoe::kMetaFewUnit); }

  private:
    // (with arena_mutex_ held, until the launch)
    void set_common(tmoe::LocalLayerParams& p, const Schedule& s) {
        const int64_t rows = layer_rows(p.plan);
        TORCH_CHECK(rows * p.plan.H * 2 <= arena_bytes_, "the arena is too small for this call");
        p.out_rows = (int)rows;
        p.y = reinterpret_cast<void*>(arena_);
        p.group_units = (int)s[0]; p.lag_percent = (int)s[1]; p.min_lag_items = (int)s[2];
        p.num_sms = (int)s[3];
        p.status = status_.data_ptr<int>();
        ++launches_;
    }
    int last_meta(int word) {
        torch::Tensor ws;
        int64_t at;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            ws = last_[0];
            at = last_meta_ + word;
        }
        return ws.defined() ? ws[at].item<int>() : 0;
    }
    void note(int dir, const torch::Tensor& ws, const tmoe::LocalLayerPlan& plan) {
        torch::Tensor before = ws;            // (the one that goes may have to wait for the interpreter: not under the lock)
        std::lock_guard<std::mutex> lock(mutex_);
        std::swap(last_[dir], before);
        last_at_[dir] = plan.stats[dir];
        if (dir == 0) last_meta_ = plan.meta;
    }
    torch::Tensor status_, host_;
    // A backward pass runs without the interpreter's lock, next to a call that replaces the arena.
    mutable std::mutex arena_mutex_;
    int64_t arena_ = 0, arena_bytes_ = 0, launches_ = 0;
    std::atomic<bool> open_{true};
    std::mutex mutex_;
    torch::Tensor last_[2];
    int64_t last_at_[2] = {0, 0}, last_meta_ = 0;
};

// The layer as a native autograd node: a backward pass runs on autograd's worker thread without the interpreter.
class LocalLayerFunction : public torch::autograd::Function<LocalLayerFunction> {
  public:
    static torch::Tensor forward(torch::autograd::AutogradContext* ctx, const torch::Tensor& x, const torch::Tensor& topk_w, const torch::Tensor& w_gateup,
                                 const torch::Tensor& w_down, const torch::Tensor& topk_idx, const c10::optional<torch::Tensor>& grad_topk_w,
                                 std::shared_ptr<LocalLayer> layer, LocalLayer::Schedule schedule, bool strict, std::shared_ptr<PyObject> owner) {
        LocalLayer::Kept kept;
        auto out = layer->forward(x, topk_idx, topk_w, w_gateup, w_down, schedule, &kept);
        // x itself is not kept.  Hooks on saved tensors may move or recompute the rows, or store them in another form; they are not
        // given the workspace, whose words are places in memory.
        ctx->save_for_backward({w_gateup, w_down, kept.rows});
        auto holder = c10::make_intrusive<Holder>();
        holder->ws = kept.ws;
        holder->layer = std::move(layer);
        holder->schedule = schedule;
        holder->K = topk_idx.size(1);
        holder->strict = strict;
        holder->owner = std::move(owner);
        holder->grad_topk_w = grad_topk_w;
        ctx->saved_data["h"] = c10::IValue::make_capsule(std::move(holder));
        return out;
    }
    static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
        const auto saved = ctx->get_saved_variables();
        auto capsule = ctx->saved_data["h"].toCapsule();
        auto* h = static_cast<Holder*>(capsule.get());
        // The counters of the workspace are cleared by the forward's routing kernels only, so the kernel can run on it once.  (The node's own
        // lock covers `spent`.)
        TORCH_CHECK(!h->spent, "teramoe_b200: a second backward pass over the same forward: its workspace is used up, also with retain_graph=True");
        torch::autograd::variable_list res;
        {
            at::AutoGradMode no_grad(false);
            auto r = h->layer->backward(grads[0].contiguous(), LocalLayer::Kept{h->ws, saved[2]}, saved[0], saved[1], h->K, h->schedule);
            h->spent = true;
            h->ws = torch::Tensor();
            if (h->grad_topk_w.has_value()) {
                h->grad_topk_w->copy_(r[1]);
                r[1] = *h->grad_topk_w;
            }
            h->layer->settle(h->strict);
            res = {r[0], r[1], r[2], r[3]};
        }
        if (at::GradMode::is_enabled()) {
            // a graph of this backward pass was asked for: using it raises, as there is no second derivative
            auto err = std::make_shared<torch::autograd::DelayedError>("trying to differentiate twice a function that was marked with @once_differentiable",
                                                                       (int64_t)res.size());
            for (auto& r : res) r = r.detach().requires_grad_(true);
            res = (*err)(std::move(res));
        }
        res.resize(10);
        return res;
    }

  private:
    struct Holder : torch::CustomClassHolder {
        std::shared_ptr<LocalLayer> layer;
        LocalLayer::Schedule schedule;
        int64_t K;
        bool strict, spent = false;
        torch::Tensor ws;
        c10::optional<torch::Tensor> grad_topk_w;
        std::shared_ptr<PyObject> owner;      // the buffer lives at least as long as a graph that needs its arena
    };
};

// -> the layer's output; None: not a call for these kernels; int: the arena has to hold that many bytes first
py::object local_layer_call(std::shared_ptr<LocalLayer> layer, const torch::Tensor& x, const torch::Tensor& topk_idx, const torch::Tensor& topk_w,
                            const torch::Tensor& w_gateup, const torch::Tensor& w_down, int64_t num_experts, LocalLayer::Schedule schedule,
                            bool autograd, const c10::optional<torch::Tensor>& grad_topk_w, bool strict, py::object owner) {
    if (!layer->takes(x, topk_idx, topk_w, w_gateup, w_down, num_experts)) return py::none();
    // Forward-mode derivatives do not exist.  The Python node says so, also for tensors that require no gradient; this node is not asked then.
    if (autograd)
        for (const torch::Tensor* t : {&x, &topk_w, &w_gateup, &w_down})
            if (t->_fw_grad(0).defined()) return py::none();
    if (const int64_t need = layer->wants(x.size(0), topk_idx.size(1), num_experts, x.size(1))) return py::int_(need);
    torch::Tensor out;
    if (autograd && at::GradMode::is_enabled() && (x.requires_grad() || topk_w.requires_grad() || w_gateup.requires_grad() || w_down.requires_grad())) {
        std::shared_ptr<PyObject> keep(owner.release().ptr(), [](PyObject* p) {
            if (p == nullptr || !Py_IsInitialized()) return;
            py::gil_scoped_acquire gil;
            Py_DECREF(p);
        });
        out = LocalLayerFunction::apply(x, topk_w, w_gateup, w_down, topk_idx, grad_topk_w, layer, schedule, strict, std::move(keep));
    } else {
        at::AutoGradMode no_grad(false);
        out = layer->forward(x, topk_idx, topk_w, w_gateup, w_down, schedule, nullptr);
    }
    layer->settle(strict);
    return py::cast(out);
}

}  // namespace

void register_local(pybind11::module_& m) {
    py::class_<LocalLayout, std::shared_ptr<LocalLayout>>(m, "LocalLayout")
        .def_readonly("send_row", &LocalLayout::send_row)
        .def("totals", [](const LocalLayout& l) { return l.scratch.narrow(0, 0, l.E + 1); })
        .def("captured", [](const LocalLayout& l) { return l.capture != 0; })
        .def("rows", &LocalLayout::rows, py::call_guard<py::gil_scoped_release>());
    m.def("ll_local_dispatch", &ll_local_dispatch);
    m.def("ll_local_combine", &ll_local_combine);
    py::class_<LocalLayer, std::shared_ptr<LocalLayer>>(m, "LocalLayer")
        .def(py::init<torch::Tensor, torch::Tensor>())
        .def("set_arena", &LocalLayer::set_arena, py::call_guard<py::gil_scoped_release>())
        .def("arena", &LocalLayer::arena)
        .def("launches", &LocalLayer::launches)
        .def("close", &LocalLayer::close)
        .def("check", &LocalLayer::check)
        .def("stats", &LocalLayer::stats)
        .def("ran_few", &LocalLayer::ran_few, py::call_guard<py::gil_scoped_release>())
        .def("few_unit", &LocalLayer::few_unit, py::call_guard<py::gil_scoped_release>())
        .def("call", &local_layer_call);
    m.def("local_layer_variant", &local_layer_variant);
    m.def("local_layer_halves", &local_layer_halves);
    m.def("local_layer_columns", &local_layer_columns);
    m.def("local_counts", &local_counts);
    m.def("local_scatter", &local_scatter);
    m.def("local_combine", &local_combine);
    py::class_<LocalExchange>(m, "LocalExchange").def(py::init<>()).def("dispatch", &LocalExchange::dispatch);
}
