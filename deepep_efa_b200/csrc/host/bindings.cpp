// Python bindings (module `_dx`): the host runtime, the host-only helpers (Config, Arena, layouts) and
// one launch function per kernel. Launch functions take LISTS of per-rank arguments: one entry in a
// real multi-process job, one entry per emulated rank in the single-GPU emulation (one cooperative
// launch for all of them). All launches go to the CURRENT torch CUDA stream of the rank's device; the
// Python layer chooses the stream (communication stream, compute stream for hook mode).
//
// Reference counterpart: the pybind module at csrc/deep_ep.cpp:4310-4479 and the host halves of
// get_dispatch_layout / intranode_dispatch / intranode_combine (csrc/deep_ep.cpp:517-1035).
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/functional.h>
#include <pybind11/stl.h>
#include <torch/extension.h>

#include "../kernels/gemm_api.h"
#include "runtime.hpp"

namespace py = pybind11;
using dxh::RuntimeCore;

namespace {

#define DX_CHECK(cond, msg)                                                        \
    do {                                                                           \
        if (!(cond)) throw std::invalid_argument(std::string("deepep_efa_b200: ") + (msg)); \
    } while (0)

struct Runtime {
    std::shared_ptr<RuntimeCore> core;
    cudaStream_t comm_stream = nullptr;
    torch::Tensor layout_scratch;  // grows on demand
    bool all_tokens_sent = true;   // by the last dispatch of a lone rank (see normal_dispatch)
    int ll_dispatched = -1;        // parity of the low-latency dispatch that no combine has followed yet

    Runtime(int rank, int num_ranks, int64_t num_nvl_bytes, int64_t num_ll_bytes, int device, double timeout_ms, bool mask_on_timeout)
        : core(std::make_shared<RuntimeCore>(rank, num_ranks, (uint64_t)num_nvl_bytes, (uint64_t)num_ll_bytes, device, timeout_ms,
                                             mask_on_timeout)) {}

    py::bytes ipc_handle() const { return py::bytes(core->ipc_handle()); }
    void open_peers(const std::vector<std::string>& handles) { core->open_peers(handles); }
    void set_comm_stream(int64_t s) { comm_stream = reinterpret_cast<cudaStream_t>(s); }

    // A block of the arena; its memory returns when the last tensor in it dies.
    struct Block {
        std::shared_ptr<RuntimeCore> core;
        uint64_t off;
        cudaStream_t comm;
        Block(std::shared_ptr<RuntimeCore> c, uint64_t at, cudaStream_t s) : core(std::move(c)), off(at), comm(s) {}
        Block(const Block&) = delete;
        ~Block() {
            cudaStream_t streams[2];
            int n = 0;
            try {
                streams[n] = c10::cuda::getCurrentCUDAStream(core->device()).stream();
                ++n;
            } catch (...) {
            }
            if (comm != nullptr && core->comm_stream_shared()) streams[n++] = comm;
            core->arena_release(off, streams, n);
        }
    };
    using BlockPtr = std::shared_ptr<Block>;
    bool alloc_blocks(const uint64_t* bytes, int n, BlockPtr* blocks, uint64_t roomy = 0) {
        uint64_t offs[8];
        DX_CHECK(n <= 8, "at most 8 blocks at a time");
        if (!core->arena_alloc(bytes, n, offs, roomy)) return false;
        for (int i = 0; i < n; ++i) blocks[i] = std::make_shared<Block>(core, offs[i], comm_stream);
        return true;
    }
    BlockPtr alloc_block(uint64_t bytes) {
        BlockPtr b;
        alloc_blocks(&bytes, 1, &b);
        return b;
    }
    torch::Tensor tensor_in(const BlockPtr& block, uint64_t byte_off, at::IntArrayRef sizes, torch::ScalarType dtype) {
        return torch::from_blob(reinterpret_cast<char*>(core->base()) + block->off + byte_off, sizes, [block](void*) {},
                                torch::TensorOptions().dtype(dtype).device(torch::kCUDA, core->device()));
    }

    torch::Tensor alloc_symmetric(std::vector<int64_t> sizes, torch::ScalarType dtype) {
        int64_t numel = 1;
        for (auto s : sizes) numel *= s;
        return tensor_in(alloc_block((uint64_t)numel * c10::elementSize(dtype)), 0, sizes, dtype);
    }

    // Offset of a tensor inside the symmetric buffer, or -1 when it lives elsewhere.
    int64_t symmetric_offset(const torch::Tensor& t) const {
        if (!t.is_cuda() || !t.is_contiguous()) return -1;
        uint64_t off = 0;
        if (!core->in_symmetric(t.data_ptr(), (uint64_t)t.numel() * t.element_size(), &off)) return -1;
        return (int64_t)off;
    }

    // Tensor view over a fixed range of the symmetric buffer (low-latency region). Not owned.
    torch::Tensor view(int64_t off, std::vector<int64_t> sizes, torch::ScalarType dtype) {
        int64_t numel = 1;
        for (auto s : sizes) numel *= s;
        DX_CHECK(off >= 0 && (uint64_t)off + (uint64_t)numel * c10::elementSize(dtype) <= core->total_bytes(), "view out of the symmetric buffer");
        auto keep = core;
        return torch::from_blob(reinterpret_cast<char*>(core->base()) + off, sizes, [keep](void*) {},
                                torch::TensorOptions().dtype(dtype).device(torch::kCUDA, core->device()));
    }

    void set_mask(int rank_to_mask, bool mask) {
        DX_CHECK(rank_to_mask >= 0 && rank_to_mask < core->num_ranks(), "rank_to_mask out of range");
        const int v = mask ? 1 : 0;
        DX_CUDA_CHECK(cudaMemcpyAsync(&core->control()->ll_mask[rank_to_mask], &v, sizeof(int), cudaMemcpyHostToDevice,
                                      c10::cuda::getCurrentCUDAStream(core->device()).stream()));
        DX_CUDA_CHECK(cudaStreamSynchronize(c10::cuda::getCurrentCUDAStream(core->device()).stream()));
    }
    void query_mask(torch::Tensor out) {
        DX_CHECK(out.is_cuda() && out.scalar_type() == torch::kInt32 && out.numel() >= core->num_ranks(), "mask_status must be int32 [num_ranks] on the GPU");
        DX_CUDA_CHECK(cudaMemcpyAsync(out.data_ptr(), core->control()->ll_mask, sizeof(int) * core->num_ranks(), cudaMemcpyDeviceToDevice,
                                      c10::cuda::getCurrentCUDAStream(core->device()).stream()));
    }
    void clean_mask() {
        DX_CUDA_CHECK(cudaMemsetAsync(core->control()->ll_mask, 0, sizeof(int) * dx::kMaxRanks,
                                      c10::cuda::getCurrentCUDAStream(core->device()).stream()));
    }
};

}  // namespace

// used by fused_bindings.cpp, which cannot name the module-local Runtime class
dxh::RuntimeCore* dx_core_of(py::handle runtime) { return runtime.cast<Runtime*>()->core.get(); }

namespace {

cudaStream_t cur_stream(const Runtime* rt) { return c10::cuda::getCurrentCUDAStream(rt->core->device()).stream(); }

void set_local_peers(std::vector<Runtime*> rts) {
    std::vector<RuntimeCore*> cores;
    for (auto* r : rts) cores.push_back(r->core.get());
    for (auto* r : rts) r->core->set_local_peers(cores);
}

template <typename T>
T* ptr_or_null(const c10::optional<torch::Tensor>& t) {
    return t.has_value() && t->defined() ? reinterpret_cast<T*>(t->data_ptr()) : nullptr;
}

void check_launch(cudaError_t e, const char* what) {
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw std::runtime_error(std::string(what) + ": launch failed: " + cudaGetErrorString(e));
    }
}

// Counts, membership and handles come from earlier calls, each allocated on the stream that call ran on. A call that reads them on
// another stream marks them there, so that their memory is not handed out again before its kernels have run, whoever drops them and
// when. On the stream they came from this does nothing.
void used_here(const torch::Tensor& t) {
    if (t.is_cuda()) c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), c10::cuda::getCurrentCUDAStream(t.get_device()));
}

// ---------------------------------------------------------------------------------------------
// layout
// ---------------------------------------------------------------------------------------------
std::tuple<torch::Tensor, torch::Tensor, torch::Tensor> get_dispatch_layout(Runtime* rt, const torch::Tensor& topk_idx, int num_experts) {
    DX_CHECK(topk_idx.dim() == 2 && topk_idx.is_contiguous() && topk_idx.scalar_type() == torch::kInt64, "topk_idx must be contiguous int64 [T,K]");
    const int R = rt->core->num_ranks();
    DX_CHECK(num_experts > 0 && num_experts % R == 0, "num_experts must be a positive multiple of the number of ranks");
    c10::cuda::CUDAGuard guard(rt->core->device());
    const int T = (int)topk_idx.size(0), K = (int)topk_idx.size(1);
    auto i32 = torch::TensorOptions().dtype(torch::kInt32).device(topk_idx.device());
    auto per_rank = torch::empty({R}, i32), per_expert = torch::empty({num_experts}, i32);
    auto in_rank = torch::empty({T, R}, i32.dtype(torch::kBool));
    // The scratch belongs to whichever call runs: it is replaced only behind the previous one, and marked on the stream that uses it,
    // so that an outgrown one is not handed out while a call on another stream is still to use it. A captured call has one of its own
    // in the graph's memory: the shared one may be outgrown by the time of a replay.
    dxh::OrderedCall order(cur_stream(rt));
    order.add(rt->core.get());
    order.enter();
    const int64_t need = (int64_t)dx::layout_scratch_ints(num_experts, R, T);
    torch::Tensor scratch;
    if (order.captured()) {
        scratch = torch::zeros({need}, i32);
    } else {
        if (!rt->layout_scratch.defined() || rt->layout_scratch.numel() < need) rt->layout_scratch = torch::zeros({need}, i32);
        scratch = rt->layout_scratch;
        used_here(scratch);
    }
    dx::LayoutArgs a{};
    a.topk_idx = topk_idx.data_ptr<int64_t>();
    a.num_tokens = T;
    a.num_topk = K;
    a.num_experts = num_experts;
    a.num_ranks = R;
    a.num_tokens_per_rank = per_rank.data_ptr<int>();
    a.num_tokens_per_expert = per_expert.data_ptr<int>();
    a.is_token_in_rank = in_rank.data_ptr<bool>();
    a.scratch = scratch.data_ptr<int>();
    check_launch(dx::launch_layout(a, order.stream), "get_dispatch_layout");
    return {per_rank, per_expert, in_rank};
}

c10::optional<torch::Tensor> opt_tensor(const py::handle& h) {
    if (h.is_none()) return c10::nullopt;
    return h.cast<torch::Tensor>();
}

// ---------------------------------------------------------------------------------------------
// normal-mode dispatch: count exchange, host wait for the receive counts, outputs carved from the arena, dispatch kernel.
// Per rank request: (x, x_scales|None, num_tokens_per_rank|None, num_tokens_per_expert|None, is_token_in_rank|None,
//                    topk_idx|None, topk_weights|None, handle|None)
// Per rank result:  (recv_x, recv_scales|None, recv_topk_idx|None, recv_topk_weights|None, rows per local expert (list),
//                    (rank_prefix_matrix, channel_prefix_matrix, recv_channel_prefix_matrix, recv_src_idx, is_token_in_rank, send_head))
// ---------------------------------------------------------------------------------------------
struct DispatchCall {
    torch::Tensor x, in_rank, rpm, cpm, rcpm, send_head;
    c10::optional<torch::Tensor> x_scales, topk_idx, topk_w;
    int T = 0, H = 0, K = 0, num_recv = 0;
    torch::ScalarType out_type;
    bool has_scales = false;
    std::vector<int> per_expert;
    // Outputs with lives of their own (the source indices live on in the handle, the weights in a backward pass) are blocks of their
    // own; the scales are in front of the rows they belong to.
    struct Out {
        uint64_t head_bytes = 0, row_bytes = 0;  // per row: what lies in front (of all rows), and the rows
        bool there = false;
        Runtime::BlockPtr block;
        uint64_t head_rows = 0;  // rows the front part was sized for
        uint64_t bytes(int rows) const { return there ? front(rows) + (uint64_t)rows * row_bytes : 0; }
        uint64_t front(uint64_t rows) const { return dxh::align_up(rows * head_bytes, 1024); }
        uint64_t off() const { return there ? block->off + front(head_rows) : 0; }
    };
    enum { kRecvX, kRecvIdx, kRecvW, kSrcIdx, kOuts };
    Out outs[kOuts];

    void describe() {
        outs[kRecvX] = {has_scales ? (uint64_t)(H / 128) * 4 : 0, (uint64_t)H * c10::elementSize(out_type), true};
        outs[kRecvIdx] = {0, (uint64_t)K * 8, topk_idx.has_value()};
        outs[kRecvW] = {0, (uint64_t)K * 4, topk_w.has_value()};
        outs[kSrcIdx] = {0, 4, true};
    }
    // With `only_if_roomy`: only where they take at most a quarter of the largest free block.
    bool allocate(Runtime* rt, int rows, bool only_if_roomy = false) {
        uint64_t bytes[kOuts], sum = 0;
        Out* of[kOuts];
        int n = 0;
        for (Out& o : outs)
            if (o.there) {
                of[n] = &o;
                bytes[n] = o.bytes(rows);
                sum += dxh::align_up(bytes[n] + 1, 1024);
                ++n;
            }
        Runtime::BlockPtr blocks[kOuts];
        if (!rt->alloc_blocks(bytes, n, blocks, only_if_roomy ? 4 * sum : 0)) return false;
        for (int i = 0; i < n; ++i) {
            of[i]->block = std::move(blocks[i]);
            of[i]->head_rows = (uint64_t)rows;
        }
        return true;
    }
    // The kernel writes no row past the received ones, so the rest is as good as never allocated.
    void trim(Runtime* rt, int rows) {
        for (Out& o : outs) {
            if (o.there) rt->core->arena_shrink(o.block->off, o.front(o.head_rows) + (uint64_t)rows * o.row_bytes);
        }
    }
};

// Lets other host threads run: the caller has left its OrderedCall.
void wait_counts(Runtime* rt, DispatchCall& q, int num_local_experts) {
    py::gil_scoped_release rel;
    q.num_recv = rt->core->wait_recv_counts(num_local_experts, &q.per_expert);
}

py::list normal_dispatch(std::vector<Runtime*> rts, const std::vector<py::tuple>& reqs, int num_channels, int expert_alignment, bool quantize,
                         bool round_scale, int num_worst_tokens, int num_sms) {
    const int V = (int)rts.size();
    DX_CHECK(V >= 1 && V <= dx::kMaxVirtualRanks && (int)reqs.size() == V, "dispatch: one entry per rank");
    DX_CHECK(num_sms >= 1, "num_sms must be >= 1");
    DX_CHECK(num_channels >= 1 && num_channels <= dx::kMaxChannels, "num_channels out of range");
    DX_CHECK(expert_alignment >= 1, "expert_alignment must be >= 1");
    c10::cuda::CUDAGuard guard(rts[0]->core->device());
    const int R = rts[0]->core->num_ranks();
    std::vector<DispatchCall> calls(V);
    std::vector<dx::NotifyArgs> nargs(V);
    std::vector<dx::DispatchArgs> dargs(V);
    dxh::OrderedCall order(cur_stream(rts[0]));
    for (Runtime* rt : rts) order.add(rt->core.get());
    bool cached = false;
    int E = R;  // a cached call carries no expert ids to remap
    for (int v = 0; v < V; ++v) {
        Runtime* rt = rts[v];
        const py::tuple& t = reqs[v];
        DispatchCall& q = calls[v];
        DX_CHECK(t.size() == 8, "dispatch: per-rank tuple must have 8 entries");
        DX_CHECK(rt->core->available(), "runtime is not synchronised with its peers");
        q.x = t[0].cast<torch::Tensor>().contiguous();
        q.x_scales = opt_tensor(t[1]);
        if (q.x_scales.has_value()) q.x_scales = q.x_scales->contiguous();  // column-major scales are accepted (the reference's tests pass them)
        q.topk_idx = opt_tensor(t[5]);
        q.topk_w = opt_tensor(t[6]);
        DX_CHECK(q.x.dim() == 2 && q.x.is_cuda(), "x must be [T,hidden] on the GPU");
        q.T = (int)q.x.size(0);
        q.H = (int)q.x.size(1);
        const int T = q.T, H = q.H;
        DX_CHECK((H * q.x.element_size()) % 16 == 0, "hidden bytes must be a multiple of 16");
        q.has_scales = quantize || q.x_scales.has_value();
        q.out_type = quantize ? torch::kFloat8_e4m3fn : q.x.scalar_type();
        if (quantize) {
            DX_CHECK(q.x.scalar_type() == torch::kBFloat16 && H % 128 == 0 && H <= 8192, "fused FP8 dispatch needs bf16 x with hidden % 128 == 0 and hidden <= 8192");
        } else if (q.x_scales.has_value()) {
            DX_CHECK(q.x.element_size() == 1 && q.x_scales->scalar_type() == torch::kFloat32 && q.x_scales->size(0) == T, "x_scales must be f32 [T,hidden/128]");
            DX_CHECK(H % 128 == 0 && q.x_scales->size(1) == H / 128, "x_scales must have hidden/128 columns");
        } else {
            DX_CHECK(q.x.scalar_type() == torch::kBFloat16, "x must be bf16 (or an (e4m3, scales) pair)");
        }
        if (q.topk_idx.has_value()) {
            DX_CHECK(q.topk_idx->scalar_type() == torch::kInt64 && q.topk_idx->is_contiguous() && q.topk_idx->dim() == 2 && q.topk_idx->size(0) == T, "topk_idx must be int64 [T,K]");
            q.K = (int)q.topk_idx->size(1);
            DX_CHECK(q.K <= dx::kMaxTopk, "num_topk too large");
            if (q.topk_w.has_value())
                DX_CHECK(q.topk_w->scalar_type() == torch::kFloat32 && q.topk_w->is_contiguous() && q.topk_w->numel() == q.topk_idx->numel(), "topk_weights must be f32 [T,K]");
        }  // (weights without ids do not travel: the result is [rows, 0])
        q.describe();
        cached = !t[7].is_none();
        q.outs[DispatchCall::kSrcIdx].there = !(cached && R == 1);  // (with peers, every rank's place is published)
        if (cached) {
            const py::tuple h(py::reinterpret_borrow<py::object>(t[7]));  // any sequence: a saved handle may come back as a list
            DX_CHECK(h.size() == 6, "a normal-mode handle has 6 entries");
            q.rpm = h[0].cast<torch::Tensor>();
            q.cpm = h[1].cast<torch::Tensor>();
            q.rcpm = h[2].cast<torch::Tensor>();
            q.num_recv = (int)h[3].cast<torch::Tensor>().size(0);
            q.in_rank = h[4].cast<torch::Tensor>();
            q.send_head = h[5].cast<torch::Tensor>();
            DX_CHECK(q.send_head.scalar_type() == torch::kInt32 && q.send_head.is_contiguous() && q.send_head.dim() == 2 && q.send_head.size(0) == T && q.send_head.size(1) == R, "send_head must be int32 [T,R]");
            DX_CHECK(q.rpm.scalar_type() == torch::kInt32 && q.rpm.is_contiguous() && q.rpm.numel() == R * R, "rank_prefix_matrix must be int32 [R,R]");
            used_here(q.rpm);
            used_here(q.send_head);
            continue;
        }
        auto ntpr = t[2].cast<torch::Tensor>(), ntpe = t[3].cast<torch::Tensor>();
        q.in_rank = t[4].cast<torch::Tensor>();
        DX_CHECK(ntpr.scalar_type() == torch::kInt32 && ntpr.numel() == R && ntpr.is_contiguous(), "num_tokens_per_rank must be int32 [R]");
        DX_CHECK(ntpe.scalar_type() == torch::kInt32 && ntpe.is_contiguous() && ntpe.numel() % R == 0, "num_tokens_per_expert must be int32 [E]");
        DX_CHECK(q.in_rank.scalar_type() == torch::kBool && q.in_rank.dim() == 2 && q.in_rank.size(1) == R && q.in_rank.is_contiguous(), "is_token_in_rank must be bool [T,R]");
        DX_CHECK(q.in_rank.size(0) == T, "is_token_in_rank must have one row per token of x");
        E = (int)ntpe.numel();
        DX_CHECK(E / R <= dx::kMaxLocalExperts, "too many local experts");
        used_here(ntpr);
        used_here(ntpe);
        used_here(q.in_rank);
        auto i32 = torch::TensorOptions().dtype(torch::kInt32).device(q.in_rank.device());
        q.rpm = torch::empty({R, R}, i32);
        q.cpm = torch::empty({R, num_channels}, i32);
        q.rcpm = torch::empty({R, num_channels}, i32);
        q.send_head = torch::empty({T, R}, i32);
        if (num_worst_tokens == 0) rt->core->reset_recv_counters(E / R);
        dx::NotifyArgs& a = nargs[v];
        a.ctx = rt->core->ctx();
        a.num_tokens_per_rank = ntpr.data_ptr<int>();
        a.num_tokens_per_expert = ntpe.data_ptr<int>();
        a.is_token_in_rank = q.in_rank.data_ptr<bool>();
        a.num_tokens = T;
        a.num_experts = E;
        a.num_channels = num_channels;
        a.expert_alignment = expert_alignment;
        a.rank_prefix_matrix = q.rpm.data_ptr<int>();
        a.channel_prefix_matrix = q.cpm.data_ptr<int>();
        a.recv_channel_prefix_matrix = q.rcpm.data_ptr<int>();
        a.send_head = q.send_head.data_ptr<int>();
        // A call whose host does not wait must not publish: its words could land after a later call has reset them.
        dxh::HostWords* hw = reinterpret_cast<dxh::HostWords*>(a.ctx.status);  // status is the first member
        a.host_recv_counter = num_worst_tokens > 0 ? nullptr : &hw->recv_counter;
        a.host_expert_counter = num_worst_tokens > 0 ? nullptr : hw->expert_counter;
    }
    if (!cached) {
        order.enter();
        check_launch(dx::launch_notify(nargs.data(), V, order.stream), "notify");
    }

    // How many rows arrive is known on the host only when the count exchange has run, except that a lone rank receives at most
    // its own tokens: its outputs are sized for them and cut to what has arrived afterwards; the dispatch kernel is queued at once
    // and the host waits beside it. Cutting leaves holes in the arena, so this is done only where a row per token is a small part of
    // it (a quarter of the largest free block) and while all tokens are sent: a caller whose last dispatch left some out waits first.
    const bool exact = !cached && num_worst_tokens == 0;
    bool waited = !exact;
    for (int v = 0; v < V; ++v) {
        DispatchCall& q = calls[v];
        int rows = cached ? q.num_recv : num_worst_tokens;
        if (exact && R == 1 && rts[v]->all_tokens_sent && q.allocate(rts[v], q.T, true)) continue;
        if (exact) {
            order.leave();
            wait_counts(rts[v], q, E / R);
            rows = q.num_recv;
            waited = true;
        }
        q.num_recv = rows;
        q.allocate(rts[v], rows);
    }
    for (int v = 0; v < V; ++v) {
        DispatchCall& q = calls[v];
        dx::DispatchArgs& a = dargs[v];
        a.ctx = rts[v]->core->ctx();
        a.x = q.x.data_ptr();
        a.x_elem_bytes = (int)q.x.element_size();
        a.x_scales = (!quantize && q.x_scales.has_value()) ? q.x_scales->data_ptr<float>() : nullptr;
        a.quantize = quantize ? 1 : 0;
        a.round_scale = round_scale ? 1 : 0;
        a.topk_idx = ptr_or_null<int64_t>(q.topk_idx);
        a.topk_weights = q.topk_idx.has_value() ? ptr_or_null<float>(q.topk_w) : nullptr;
        a.num_topk = q.K;
        a.send_head = q.send_head.data_ptr<int>();
        a.rank_prefix_matrix = q.rpm.data_ptr<int>();
        a.num_tokens = q.T;
        a.hidden = q.H;
        a.num_experts = E;
        a.num_sms = num_sms;
        a.recv_x_off = q.outs[DispatchCall::kRecvX].off();
        a.recv_scales_off = q.has_scales ? q.outs[DispatchCall::kRecvX].block->off : 0;
        a.recv_topk_idx_off = q.outs[DispatchCall::kRecvIdx].off();
        a.recv_topk_w_off = q.outs[DispatchCall::kRecvW].off();
        a.recv_src_idx_off = q.outs[DispatchCall::kSrcIdx].there ? q.outs[DispatchCall::kSrcIdx].off() : dx::kNoOffset;
        a.num_worst_tokens = num_worst_tokens;
    }
    order.enter();
    check_launch(dx::launch_dispatch(dargs.data(), V, order.stream), "dispatch");
    order.leave();

    py::list out;
    for (int v = 0; v < V; ++v) {
        Runtime* rt = rts[v];
        DispatchCall& q = calls[v];
        if (!waited) {
            wait_counts(rt, q, E / R);
            if (q.num_recv < q.T) q.trim(rt, q.num_recv);
        }
        if (exact && R == 1) rt->all_tokens_sent = q.num_recv == q.T;
        const int64_t n = q.num_recv, H = q.H, K = q.K;
        auto tensor = [&](int which, std::initializer_list<int64_t> sizes, torch::ScalarType dtype, bool front = false) -> py::object {
            const DispatchCall::Out& o = q.outs[which];
            return o.there && (!front || q.has_scales) ? py::cast(rt->tensor_in(o.block, front ? 0 : o.front(o.head_rows), sizes, dtype)) : py::object(py::none());
        };
        out.append(py::make_tuple(tensor(DispatchCall::kRecvX, {n, H}, q.out_type), tensor(DispatchCall::kRecvX, {n, H / 128}, torch::kFloat32, true),
                                  tensor(DispatchCall::kRecvIdx, {n, K}, torch::kInt64), tensor(DispatchCall::kRecvW, {n, K}, torch::kFloat32), q.per_expert,
                                  py::make_tuple(q.rpm, q.cpm, q.rcpm, tensor(DispatchCall::kSrcIdx, {n}, torch::kInt32), q.in_rank, q.send_head)));
    }
    return out;
}

// ---------------------------------------------------------------------------------------------
// normal-mode combine. Per rank call: (x, topk_weights|None, send_head, rank_prefix_matrix, bias0|None, bias1|None,
// out|None, out_topk_weights|None); outputs that are not given are allocated on the current stream.
// Per rank result: (out, out_topk_weights|None)
// ---------------------------------------------------------------------------------------------
py::list normal_combine(std::vector<Runtime*> rts, const std::vector<py::tuple>& per_rank, int num_sms) {
    const int V = (int)rts.size();
    DX_CHECK(V >= 1 && V <= dx::kMaxVirtualRanks && (int)per_rank.size() == V, "combine: one entry per rank");
    c10::cuda::CUDAGuard guard(rts[0]->core->device());
    std::vector<dx::CombineArgs> args(V);
    std::vector<torch::Tensor> keep;
    py::list results;
    dxh::OrderedCall order(cur_stream(rts[0]));
    for (Runtime* rt : rts) order.add(rt->core.get());
    for (int v = 0; v < V; ++v) {
        Runtime* rt = rts[v];
        const py::tuple& t = per_rank[v];
        DX_CHECK(t.size() == 8, "combine: per-rank tuple must have 8 entries");
        const int R = rt->core->num_ranks();
        auto x = t[0].cast<torch::Tensor>();
        auto w = opt_tensor(t[1]);
        auto send_head = t[2].cast<torch::Tensor>();
        auto rpm = t[3].cast<torch::Tensor>();
        auto b0 = opt_tensor(t[4]);
        auto b1 = opt_tensor(t[5]);
        DX_CHECK(x.is_cuda() && x.dim() == 2 && x.scalar_type() == torch::kBFloat16, "combine: x must be bf16 [N,hidden] on the GPU");
        if (w.has_value()) {
            // weights of another type, or on the host, are converted on the way to where the peers read them
            if (rt->symmetric_offset(*w) < 0) w = w->to(x.device(), torch::kFloat32);
            DX_CHECK(w->scalar_type() == torch::kFloat32 && w->dim() == 2, "combine: topk_weights must be [N,K], and f32 in the symmetric buffer");
        }
        const int H = (int)x.size(1), T = (int)send_head.size(0);
        DX_CHECK(H % 8 == 0, "hidden must be a multiple of 8");
        DX_CHECK(send_head.scalar_type() == torch::kInt32 && send_head.is_contiguous() && send_head.size(1) == R, "send_head must be int32 [T,R]");
        used_here(send_head);
        used_here(rpm);
        // What the peers read must lie in symmetric memory; anything else is staged there. A lone rank reads its own tensor where
        // it is (an offset that leaves the buffer, which the debug range check would refuse), given a row for every row of x.
        auto place = [&](const torch::Tensor& given) -> uint64_t {
            torch::Tensor tt = given.contiguous();
            int64_t off = rt->symmetric_offset(tt);
            const bool in_place = R == 1 && !rt->core->debug_checks() && tt.size(0) >= x.size(0) && (reinterpret_cast<uintptr_t>(tt.data_ptr()) & 15) == 0;
            if (off < 0 && !in_place) {
                const uint64_t bytes = (uint64_t)tt.numel() * tt.element_size();
                auto staged = rt->tensor_in(rt->alloc_block(bytes), 0, tt.sizes(), tt.scalar_type());
                DX_CUDA_CHECK(cudaMemcpyAsync(staged.data_ptr(), tt.data_ptr(), bytes, cudaMemcpyDeviceToDevice, order.stream));
                off = rt->symmetric_offset(staged);
                keep.push_back(staged);
            }
            keep.push_back(tt);
            return off >= 0 ? (uint64_t)off : (uint64_t)(reinterpret_cast<uintptr_t>(tt.data_ptr()) - reinterpret_cast<uintptr_t>(rt->core->base()));
        };
        torch::Tensor out = t[6].is_none() ? torch::empty({T, H}, x.options()) : t[6].cast<torch::Tensor>();
        DX_CHECK(out.scalar_type() == torch::kBFloat16 && out.is_contiguous() && out.size(0) == T && out.size(1) == H, "out must be bf16 [T,hidden]");
        c10::optional<torch::Tensor> out_w;
        dx::CombineArgs& a = args[v];
        a.ctx = rt->core->ctx();
        a.x_off = place(x);
        a.topk_w_off = ~0ull;
        a.num_topk = 0;
        a.out_topk_w = nullptr;
        if (w.has_value()) {
            a.topk_w_off = place(*w);
            a.num_topk = (int)w->size(1);
            out_w = t[7].is_none() ? torch::empty({T, a.num_topk}, x.options().dtype(torch::kFloat32)) : t[7].cast<torch::Tensor>();
            DX_CHECK(out_w->scalar_type() == torch::kFloat32 && out_w->is_contiguous() && out_w->numel() == (int64_t)T * a.num_topk, "combine: out_topk_weights must be f32 [T,K]");
            a.out_topk_w = out_w->data_ptr<float>();
        }
        a.send_head = send_head.data_ptr<int>();
        a.rank_prefix_matrix = rpm.data_ptr<int>();
        auto bias_ptr = [&](const c10::optional<torch::Tensor>& b) -> const __nv_bfloat16* {
            if (!b.has_value()) return nullptr;
            DX_CHECK(b->scalar_type() == torch::kBFloat16 && b->is_contiguous() && b->size(0) == T && b->size(1) == H, "bias must be bf16 [T,hidden]");
            return reinterpret_cast<const __nv_bfloat16*>(b->data_ptr());
        };
        a.bias0 = bias_ptr(b0);
        a.bias1 = bias_ptr(b1);
        a.out = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
        a.num_tokens = T;
        a.hidden = H;
        a.num_sms = num_sms;
        results.append(py::make_tuple(out, out_w));
    }
    order.enter();
    check_launch(dx::launch_combine(args.data(), V, order.stream), "combine");
    return results;
}

// ---------------------------------------------------------------------------------------------
// One rank's call on the communication stream (buffer.py: _CommScope says what it keeps in order). The stream waits for the event `previous` (none: for
// the caller's stream; 0: an event that was never recorded), the call runs with the stream as the current one, and afterwards either the caller's stream waits or,
// with `async_finish`, what both streams use is recorded on the other one. The same in Python took 20 us of a call's 35.
// ---------------------------------------------------------------------------------------------
class OnCommStream {
public:
    OnCommStream(const py::tuple& stream, py::object previous, bool async_finish)
        : comm_(c10::cuda::CUDAStream::unpack3(stream[0].cast<int64_t>(), (c10::DeviceIndex)stream[1].cast<int>(), c10::DeviceType::CUDA)),
          caller_(c10::cuda::getCurrentCUDAStream()), async_(async_finish) {
        if (previous.is_none()) {
            follow(comm_, caller_);
        } else if (const auto event = reinterpret_cast<cudaEvent_t>(previous.cast<uintptr_t>())) {
            DX_CUDA_CHECK(cudaStreamWaitEvent(comm_.stream(), event, 0));
        }
    }
    const c10::cuda::CUDAStream& stream() const { return comm_; }
    // Allocated on the communication stream and handed to the caller.
    void output(const torch::Tensor& t) const { t.record_stream(caller_); }
    // Allocated on the caller's stream; with nothing to wait for there, the memory must not be reused before the communication stream is done.
    void input(const py::handle& h) const {
        if (!async_ || !THPVariable_Check(h.ptr())) return;
        const torch::Tensor& t = THPVariable_Unpack(h.ptr());
        if (t.is_cuda()) t.record_stream(comm_);
    }
    void finish() const {
        if (!async_) follow(caller_, comm_);
    }

private:
    static void follow(const c10::cuda::CUDAStream& later, const c10::cuda::CUDAStream& first) {
        at::cuda::CUDAEvent event(cudaEventDisableTiming);
        event.record(first);
        event.block(later);
    }
    c10::cuda::CUDAStream comm_, caller_;
    bool async_;
};

py::tuple normal_dispatch_on(const py::tuple& stream, py::object previous, bool async_finish, Runtime* rt, const py::tuple& req, int num_channels, int expert_alignment,
                             bool quantize, bool round_scale, int num_worst_tokens, int num_sms) {
    OnCommStream scope(stream, previous, async_finish);
    py::list outs;
    {
        c10::cuda::CUDAStreamGuard guard(scope.stream());
        outs = normal_dispatch({rt}, {req}, num_channels, expert_alignment, quantize, round_scale, num_worst_tokens, num_sms);
    }
    const py::tuple out = outs[0];
    if (req[7].is_none()) {
        const py::tuple handle = out[5];
        for (const int i : {0, 1, 2, 5}) scope.output(handle[i].cast<torch::Tensor>());
    }
    for (int i = 0; i < 7; ++i) scope.input(req[i]);
    scope.finish();
    return out;
}

// req: (x, topk_weights|None, send_head, rank_prefix_matrix, bias0|None, bias1|None)
py::tuple normal_combine_on(const py::tuple& stream, py::object previous, bool async_finish, bool results_on_stream, Runtime* rt, const py::tuple& req, int num_sms) {
    OnCommStream scope(stream, previous, async_finish);
    py::object out = py::none(), out_w = py::none();
    // Results of a call that follows the caller's stream are allocated there, freed on which they are reusable at once. Behind an event they are the communication
    // stream's: a block that the caller's stream gave up after the event may still be in use there.
    results_on_stream = results_on_stream || !previous.is_none();
    if (!results_on_stream) {
        const auto x = req[0].cast<torch::Tensor>();
        const int64_t rows = req[2].cast<torch::Tensor>().size(0);
        out = py::cast(torch::empty({rows, x.size(1)}, x.options().dtype(torch::kBFloat16)));
        if (!req[1].is_none()) out_w = py::cast(torch::empty({rows, req[1].cast<torch::Tensor>().size(1)}, x.options().dtype(torch::kFloat32)));
    }
    py::list results;
    {
        c10::cuda::CUDAStreamGuard guard(scope.stream());
        results = normal_combine({rt}, {py::make_tuple(req[0], req[1], req[2], req[3], req[4], req[5], out, out_w)}, num_sms);
    }
    const py::tuple result = results[0];
    for (const py::handle& h : result) {
        if (h.is_none()) continue;
        if (results_on_stream) scope.output(py::cast<torch::Tensor>(h));
        else scope.input(h);
    }
    for (const int i : {0, 1, 4, 5}) scope.input(req[i]);
    scope.finish();
    return result;
}

void barrier(std::vector<Runtime*> rts) {
    const int V = (int)rts.size();
    c10::cuda::CUDAGuard guard(rts[0]->core->device());
    std::vector<dx::BarrierArgs> args(V);
    for (int v = 0; v < V; ++v) args[v].ctx = rts[v]->core->ctx();
    check_launch(dx::launch_barrier(args.data(), V, cur_stream(rts[0])), "barrier");
}

void timeout_probe(Runtime* rt) {
    c10::cuda::CUDAGuard guard(rt->core->device());
    check_launch(dx::launch_timeout_probe(rt->core->ctx(), rt->core->never_set_flag(), cur_stream(rt)), "timeout_probe");
}

// ---------------------------------------------------------------------------------------------
// FP8 cast
// ---------------------------------------------------------------------------------------------
std::tuple<torch::Tensor, torch::Tensor> per_token_cast_to_fp8(const torch::Tensor& x, bool round_scale, bool use_ue8m0,
                                                               c10::optional<torch::Tensor> group_counts, int rows_per_group,
                                                               c10::optional<torch::Tensor> out_q, c10::optional<torch::Tensor> out_s,
                                                               c10::optional<torch::Tensor> num_rows_dev, bool atoms) {
    DX_CHECK(x.is_cuda() && x.dim() == 2 && x.is_contiguous() && x.scalar_type() == torch::kBFloat16, "x must be contiguous bf16 [M,hidden] on the GPU");
    const int M = (int)x.size(0), H = (int)x.size(1);
    DX_CHECK(H % 128 == 0 && (!use_ue8m0 || H % 512 == 0), "hidden must be a multiple of 128 (512 for UE8M0 scales)");
    c10::cuda::CUDAGuard guard(x.device());
    auto out = out_q.has_value() ? *out_q : torch::empty({M, H}, x.options().dtype(torch::kFloat8_e4m3fn));
    // atoms: the scales leave as the UE8M0 scale atoms of the natively block-scaled GEMM, uint8 [ceil(M/128), hidden/128, 512]
    DX_CHECK(!atoms || !use_ue8m0, "atoms and use_ue8m0 are two different scale formats");
    torch::Tensor scales = out_s.has_value() ? *out_s
                           : atoms ? torch::empty({(M + 127) / 128, H / 128, 512}, x.options().dtype(torch::kUInt8))
                           : (use_ue8m0 ? torch::empty({M, H / 512}, x.options().dtype(torch::kInt32))
                                        : torch::empty({M, H / 128}, x.options().dtype(torch::kFloat32)));
    DX_CHECK(out.is_cuda() && scales.is_cuda() && out.device() == x.device() && scales.device() == x.device(), "outputs must live on x's GPU");
    DX_CHECK(out.is_contiguous() && out.numel() == (int64_t)M * H && out.element_size() == 1, "out_q must be a contiguous 1-byte [M,hidden] tensor");
    if (atoms)
        DX_CHECK(scales.is_contiguous() && scales.element_size() == 1 && scales.numel() >= (int64_t)((M + 127) / 128) * (H / 128) * 512, "out_s must be uint8 [ceil(M/128), hidden/128, 512]");
    else
        DX_CHECK(scales.is_contiguous() && scales.numel() == (int64_t)M * (use_ue8m0 ? H / 512 : H / 128) && scales.element_size() == 4, "out_s has the wrong shape");
    dx::Fp8CastArgs a{};
    a.x = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr());
    a.out = reinterpret_cast<uint8_t*>(out.data_ptr());
    a.scales = (use_ue8m0 || atoms) ? nullptr : scales.data_ptr<float>();
    a.scales_ue8m0 = use_ue8m0 ? scales.data_ptr<int32_t>() : nullptr;
    a.sf_atoms = atoms ? scales.data_ptr<uint8_t>() : nullptr;
    if (num_rows_dev.has_value()) {
        DX_CHECK(num_rows_dev->is_cuda() && num_rows_dev->device() == x.device() && num_rows_dev->scalar_type() == torch::kInt32 && num_rows_dev->numel() >= 1,
                 "num_rows_dev must be an int32 tensor on x's GPU");
        a.num_rows_dev = num_rows_dev->data_ptr<int>();
    }
    a.num_rows = M;
    a.hidden = H;
    a.round_scale = round_scale ? 1 : 0;
    a.ue8m0 = use_ue8m0 ? 1 : 0;
    a.group_counts = nullptr;
    a.rows_per_group = 1;
    if (group_counts.has_value()) {
        DX_CHECK(group_counts->is_cuda() && group_counts->scalar_type() == torch::kInt32 && group_counts->is_contiguous() && rows_per_group > 0 &&
                     group_counts->numel() * (int64_t)rows_per_group == M, "group_counts must be int32 [M / rows_per_group]");
        a.group_counts = group_counts->data_ptr<int>();
        a.rows_per_group = rows_per_group;
    }
    check_launch(dx::launch_fp8_cast(a, c10::cuda::getCurrentCUDAStream(x.device().index()).stream()), "per_token_cast_to_fp8");
    return {out, scales};
}

// ---------------------------------------------------------------------------------------------
// low latency
// ---------------------------------------------------------------------------------------------
dx::LLRegion make_region(const dxh::LowLatencyLayout& l) {
    dx::LLRegion r;
    for (int p = 0; p < 2; ++p) {
        r.counts_off[p] = l.counts_off[p];
        r.recv_x_off[p] = l.recv_x_off[p];
        r.recv_scales_off[p] = l.recv_scales_off[p];
        r.recv_src_info_off[p] = l.recv_src_info_off[p];
        r.combine_stage_off[p] = l.combine_stage_off[p];
        r.combine_src_off[p] = l.combine_src_off[p];
    }
    return r;
}

using OptTensor = c10::optional<torch::Tensor>;

void fill_ll_dispatch(dx::LLDispatchArgs& a, Runtime* rt, const torch::Tensor& x, const torch::Tensor& topk_idx, const torch::Tensor& count,
                      const torch::Tensor& range, const OptTensor& cum, const OptTensor& wait, const OptTensor& slot, int num_max_tokens, int num_experts,
                      bool use_fp8, bool round_scale, bool use_ue8m0, int parity, int phases, int num_sms) {
    const int R = rt->core->num_ranks();
    // x may also sit in pinned host memory: the token CTAs then read their rows over PCIe themselves (each row is read
    // exactly once), which is the host-to-device transfer without a copy in front of the kernel
    const bool x_on_gpu = x.is_cuda() && x.device().index() == rt->core->device();
    const bool x_pinned = x.device().is_cpu() && x.is_pinned();
    DX_CHECK((x_on_gpu || x_pinned) && x.dim() == 2 && x.is_contiguous() && x.scalar_type() == torch::kBFloat16,
             "x must be contiguous bf16 [T,hidden] on this rank's GPU or in pinned host memory");
    DX_CHECK(topk_idx.is_cuda() && topk_idx.device().index() == rt->core->device() && count.is_cuda() && range.is_cuda(),
             "low_latency_dispatch: every tensor but x must live on this rank's GPU");
    const int T = (int)x.size(0), H = (int)x.size(1);
    DX_CHECK(T <= num_max_tokens, "more tokens than num_max_dispatch_tokens_per_rank");
    DX_CHECK(num_max_tokens <= 65535, "num_max_dispatch_tokens_per_rank must fit the 16-bit count field of the count exchange");
    DX_CHECK((int64_t)R * num_max_tokens < 65535, "rows per expert (ranks x num_max_dispatch_tokens_per_rank) must fit the 16-bit row field of send_row");
    DX_CHECK(H % 128 == 0 && (!use_ue8m0 || H % 512 == 0), "hidden must be a multiple of 128 (512 with UE8M0)");
    DX_CHECK(topk_idx.scalar_type() == torch::kInt64 && topk_idx.is_contiguous() && topk_idx.dim() == 2 && topk_idx.size(0) == T, "topk_idx must be int64 [T,K]");
    DX_CHECK(topk_idx.size(1) <= dx::kMaxTopk, "num_topk too large");
    DX_CHECK(num_experts % R == 0 && count.numel() == num_experts / R && range.numel() == (int64_t)(num_experts / R) * R, "bad output shapes");
    dxh::LowLatencyLayout lay(rt->core->ll_base(), num_max_tokens, H, R, num_experts);
    DX_CHECK(lay.total_bytes <= rt->core->ll_bytes(), "low-latency region too small: create the Buffer with num_rdma_bytes >= get_low_latency_rdma_size_hint(...)");
    a.ctx = rt->core->ctx();
    a.parity = parity;
    a.region = make_region(lay);
    a.x = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr());
    a.topk_idx = topk_idx.data_ptr<int64_t>();
    a.num_tokens = T;
    a.hidden = H;
    a.num_topk = (int)topk_idx.size(1);
    a.num_experts = num_experts;
    a.num_max_tokens = num_max_tokens;
    a.use_fp8 = use_fp8;
    a.round_scale = round_scale;
    a.use_ue8m0 = use_ue8m0;
    a.phases = phases;
    a.packed_recv_count = count.data_ptr<int>();
    a.layout_range = range.data_ptr<int64_t>();
    a.cumulative_stats = ptr_or_null<int>(cum);
    a.wait_cost_stats = ptr_or_null<int64_t>(wait);
    if (slot.has_value())
        DX_CHECK(slot->is_cuda() && slot->scalar_type() == torch::kInt32 && slot->is_contiguous() && slot->numel() >= (int64_t)T * topk_idx.size(1), "send_row must be int32 [T,K] on the GPU");
    a.send_row = ptr_or_null<int>(slot);
    a.num_sms = num_sms;
    rt->ll_dispatched = parity;
}

// Per rank tuple: (x, topk_idx, packed_recv_count, layout_range, cumulative_stats|None, wait_stats|None, send_row|None)
void ll_dispatch(std::vector<Runtime*> rts, std::vector<py::tuple> per_rank, int num_max_tokens, int num_experts, bool use_fp8,
                 bool round_scale, bool use_ue8m0, int parity, int phases, int num_sms) {
    const int V = (int)rts.size();
    DX_CHECK(V >= 1 && V <= dx::kMaxVirtualRanks && (int)per_rank.size() == V, "ll_dispatch: one entry per rank");
    c10::cuda::CUDAGuard guard(rts[0]->core->device());
    std::vector<dx::LLDispatchArgs> args(V);
    for (int v = 0; v < V; ++v) {
        const py::tuple& t = per_rank[v];
        DX_CHECK(t.size() == 7, "ll_dispatch: per-rank tuple must have 7 entries");
        fill_ll_dispatch(args[v], rts[v], t[0].cast<torch::Tensor>(), t[1].cast<torch::Tensor>(), t[2].cast<torch::Tensor>(), t[3].cast<torch::Tensor>(),
                         opt_tensor(t[4]), opt_tensor(t[5]), opt_tensor(t[6]), num_max_tokens, num_experts, use_fp8, round_scale, use_ue8m0, parity, phases, num_sms);
    }
    check_launch(dx::launch_ll_dispatch(args.data(), V, cur_stream(rts[0])), "low_latency_dispatch");
}

// One rank and both halves, the call of a decode step: its arguments come one by one instead of in lists and tuples.
void ll_dispatch_one(Runtime* rt, const torch::Tensor& x, const torch::Tensor& topk_idx, const torch::Tensor& count, const torch::Tensor& range,
                     const OptTensor& cum, const OptTensor& wait, const torch::Tensor& slot, int num_max_tokens, int num_experts, bool use_fp8,
                     bool round_scale, bool use_ue8m0, int parity, int num_sms) {
    c10::cuda::CUDAGuard guard(rt->core->device());
    dx::LLDispatchArgs a{};
    fill_ll_dispatch(a, rt, x, topk_idx, count, range, cum, wait, slot, num_max_tokens, num_experts, use_fp8, round_scale, use_ue8m0, parity, 3, num_sms);
    check_launch(dx::launch_ll_dispatch(&a, 1, cur_stream(rt)), "low_latency_dispatch");
}

// pull: x of every rank lives in its symmetric buffer and send_row comes from the dispatch of the same handle; the home
// ranks read the rows in place. close_barrier: readers report back before the kernel ends (x is not the zero-copy buffer).
void fill_ll_combine(dx::LLCombineArgs& a, Runtime* rt, const torch::Tensor& x, const torch::Tensor& topk_idx, const torch::Tensor& topk_w,
                     const torch::Tensor& src_info, const torch::Tensor& range, const torch::Tensor& out, const OptTensor& wait, const OptTensor& send_row,
                     int num_max_tokens, int num_experts, int parity, int phases, int num_sms, bool pull, bool close_barrier) {
    const int R = rt->core->num_ranks();
    const int L = num_experts / R;
    DX_CHECK(x.is_cuda() && x.dim() == 3 && x.is_contiguous() && x.scalar_type() == torch::kBFloat16 && x.size(0) == L && x.size(1) == (int64_t)R * num_max_tokens, "x must be contiguous bf16 [L, R*max_tokens, hidden] on the GPU");
    DX_CHECK(x.device().index() == rt->core->device() && topk_idx.is_cuda() && topk_w.is_cuda() && src_info.is_cuda() && range.is_cuda() &&
                 topk_idx.device() == x.device() && topk_w.device() == x.device(), "low_latency_combine: inputs must live on this rank's GPU");
    // the result may go to device memory or straight to pinned (page-locked, device-mapped) host memory
    DX_CHECK((out.is_cuda() && out.device() == x.device()) || (out.device().is_cpu() && out.is_pinned()), "out must be on this rank's GPU or in pinned host memory");
    const int H = (int)x.size(2);
    DX_CHECK(topk_idx.scalar_type() == torch::kInt64 && topk_idx.is_contiguous() && topk_idx.dim() == 2, "topk_idx must be int64 [T,K]");
    const int T = (int)topk_idx.size(0);
    DX_CHECK(T <= num_max_tokens && topk_idx.size(1) <= dx::kMaxTopk, "too many tokens or top-k entries");
    DX_CHECK(topk_w.scalar_type() == torch::kFloat32 && topk_w.is_contiguous() && topk_w.numel() == topk_idx.numel(), "topk_weights must be f32 [T,K]");
    DX_CHECK(src_info.scalar_type() == torch::kInt32 && src_info.is_contiguous() && src_info.numel() == (int64_t)L * R * num_max_tokens, "src_info must be int32 [L,N]");
    DX_CHECK(range.scalar_type() == torch::kInt64 && range.is_contiguous() && range.numel() == (int64_t)L * R, "layout_range must be int64 [L,R]");
    DX_CHECK(out.scalar_type() == torch::kBFloat16 && out.is_contiguous() && out.size(0) == T && out.size(1) == H, "out must be bf16 [T,hidden]");
    // A result that overwrites expert outputs: the staged form has copied every row before it stores one. (With peers the forms are
    // different protocols, which a rank cannot choose by itself.)
    const char *x0 = static_cast<const char*>(x.data_ptr()), *out0 = static_cast<const char*>(out.data_ptr());
    a.in_place = R == 1 && out0 < x0 + x.nbytes() && out0 + out.nbytes() > x0 ? 1 : 0;
    if (a.in_place) pull = close_barrier = false;
    dxh::LowLatencyLayout lay(rt->core->ll_base(), num_max_tokens, H, R, num_experts);
    DX_CHECK(lay.total_bytes <= rt->core->ll_bytes(), "low-latency region too small");
    a.ctx = rt->core->ctx();
    a.parity = parity;
    a.region = make_region(lay);
    a.x = reinterpret_cast<const __nv_bfloat16*>(x.data_ptr());
    a.topk_idx = topk_idx.data_ptr<int64_t>();
    a.topk_weights = topk_w.data_ptr<float>();
    a.src_info = src_info.data_ptr<int>();
    a.layout_range = range.data_ptr<int64_t>();
    a.out = reinterpret_cast<__nv_bfloat16*>(out.data_ptr());
    a.wait_cost_stats = ptr_or_null<int64_t>(wait);
    a.num_tokens = T;
    a.hidden = H;
    a.num_topk = (int)topk_idx.size(1);
    a.num_experts = num_experts;
    a.num_max_tokens = num_max_tokens;
    a.phases = phases;
    a.num_sms = num_sms;
    a.pull = pull ? 1 : 0;
    a.close_barrier = (pull && close_barrier) ? 1 : 0;
    a.x_off = 0;
    a.settled = 0;
    a.send_row = nullptr;
    if (send_row.has_value()) {
        DX_CHECK(send_row->is_cuda() && send_row->scalar_type() == torch::kInt32 && send_row->is_contiguous() &&
                     send_row->numel() >= (int64_t)T * topk_idx.size(1), "send_row must be int32 [T,K] on the GPU");
        a.send_row = send_row->data_ptr<int>();
    }
    if (pull) {
        const int64_t xo = rt->symmetric_offset(x);
        DX_CHECK(xo >= 0 && xo % 16 == 0, "pull combine: x must live in this rank's symmetric buffer");
        DX_CHECK(send_row.has_value(), "pull combine: send_row is missing");
        a.x_off = (uint64_t)xo;
        // Rows may be gathered beside the dispatch of their handle unless that dispatch is what writes them: of the low-latency region (where
        // x may be the landing zone itself, as in a round trip without experts) only the combine buffers are the caller's to fill.
        const uint64_t begin = (uint64_t)xo, end = begin + (uint64_t)x.numel() * x.element_size();
        const bool in_region = begin < rt->core->ll_base() + rt->core->ll_bytes() && end > rt->core->ll_base();
        // Nor where another combine came in between: it lets its successor start before its result is written, and that may be part of x.
        a.settled = (rt->ll_dispatched == parity && (!in_region || begin == lay.combine_src_off[0] || begin == lay.combine_src_off[1])) ? 1 : 0;
    }
    rt->ll_dispatched = -1;
}

// Per rank tuple: (x, topk_idx, topk_weights, src_info, layout_range, out, wait_stats|None, send_row|None)
void ll_combine(std::vector<Runtime*> rts, std::vector<py::tuple> per_rank, int num_max_tokens, int num_experts, int parity, int phases,
                int num_sms, bool pull, bool close_barrier) {
    const int V = (int)rts.size();
    DX_CHECK(V >= 1 && V <= dx::kMaxVirtualRanks && (int)per_rank.size() == V, "ll_combine: one entry per rank");
    c10::cuda::CUDAGuard guard(rts[0]->core->device());
    std::vector<dx::LLCombineArgs> args(V);
    for (int v = 0; v < V; ++v) {
        const py::tuple& t = per_rank[v];
        DX_CHECK(t.size() == 8, "ll_combine: per-rank tuple must have 8 entries");
        fill_ll_combine(args[v], rts[v], t[0].cast<torch::Tensor>(), t[1].cast<torch::Tensor>(), t[2].cast<torch::Tensor>(), t[3].cast<torch::Tensor>(),
                        t[4].cast<torch::Tensor>(), t[5].cast<torch::Tensor>(), opt_tensor(t[6]), opt_tensor(t[7]), num_max_tokens, num_experts, parity, phases,
                        num_sms, pull, close_barrier);
    }
    check_launch(dx::launch_ll_combine(args.data(), V, cur_stream(rts[0])), "low_latency_combine");
}

// One rank and both halves; `zero_copy` is this parity's zero-copy buffer. Returns the result, allocated here unless given.
torch::Tensor ll_combine_one(Runtime* rt, const torch::Tensor& x, const torch::Tensor& topk_idx, const torch::Tensor& topk_w, const torch::Tensor& src_info,
                             const torch::Tensor& range, const OptTensor& out, const OptTensor& wait, const torch::Tensor& send_row,
                             const torch::Tensor& zero_copy, int num_max_tokens, int num_experts, int parity, int num_sms) {
    c10::cuda::CUDAGuard guard(rt->core->device());
    const bool pull = rt->symmetric_offset(x) >= 0;
    // a caller-owned tensor: its owner may rewrite it as soon as the call returns
    const bool close_barrier = pull && x.data_ptr() != zero_copy.data_ptr();
    const torch::Tensor result = out.has_value() ? *out : torch::empty({topk_idx.size(0), zero_copy.size(2)}, topk_idx.options().dtype(torch::kBFloat16));
    dx::LLCombineArgs a{};
    fill_ll_combine(a, rt, x, topk_idx, topk_w, src_info, range, result, wait, send_row, num_max_tokens, num_experts, parity, 3, num_sms, pull, close_barrier);
    check_launch(dx::launch_ll_combine(&a, 1, cur_stream(rt)), "low_latency_combine");
    return result;
}

// Offsets of the low-latency region for the Python layer (views are created there once and cached).
py::dict ll_layout(Runtime* rt, int num_max_tokens, int hidden, int num_experts) {
    dxh::LowLatencyLayout l(rt->core->ll_base(), num_max_tokens, hidden, rt->core->num_ranks(), num_experts);
    py::dict d;
    auto put = [&](const char* k, const uint64_t* v) { d[k] = py::make_tuple((int64_t)v[0], (int64_t)v[1]); };
    put("counts", l.counts_off);
    put("recv_x", l.recv_x_off);
    put("recv_scales", l.recv_scales_off);
    put("recv_src_info", l.recv_src_info_off);
    put("combine_stage", l.combine_stage_off);
    put("combine_src", l.combine_src_off);
    d["total_bytes"] = (int64_t)l.total_bytes;
    d["available_bytes"] = (int64_t)rt->core->ll_bytes();
    return d;
}

}  // namespace

void bind_gemm(py::module_& m);  // gemm_bindings.cpp
void bind_hier(py::module_& m);  // hier_bindings.cpp
void bind_fused(py::module_& m); // fused_bindings.cpp

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
    m.doc() = "deepep_efa_b200 native runtime (sm_100a)";

    py::class_<dxh::Config>(m, "Config")
        .def(py::init<int, int, int, int, int>(), py::arg("num_sms") = 32, py::arg("num_max_nvl_chunked_send_tokens") = 6,
             py::arg("num_max_nvl_chunked_recv_tokens") = 256, py::arg("num_max_rdma_chunked_send_tokens") = 6,
             py::arg("num_max_rdma_chunked_recv_tokens") = 256)
        .def_readwrite("num_sms", &dxh::Config::num_sms)
        .def_readonly("num_max_nvl_chunked_send_tokens", &dxh::Config::num_max_nvl_chunked_send_tokens)
        .def_readonly("num_max_nvl_chunked_recv_tokens", &dxh::Config::num_max_nvl_chunked_recv_tokens)
        .def_readonly("num_max_rdma_chunked_send_tokens", &dxh::Config::num_max_rdma_chunked_send_tokens)
        .def_readonly("num_max_rdma_chunked_recv_tokens", &dxh::Config::num_max_rdma_chunked_recv_tokens)
        .def("get_nvl_buffer_size_hint", &dxh::Config::get_nvl_buffer_size_hint, py::arg("hidden_bytes"), py::arg("num_ranks"),
             py::arg("max_tokens_per_rank") = dxh::kDefaultHintTokens)
        .def("get_rdma_buffer_size_hint", &dxh::Config::get_rdma_buffer_size_hint, py::arg("hidden_bytes"), py::arg("num_ranks"));
    m.def("get_low_latency_rdma_size_hint", &dxh::get_low_latency_rdma_size_hint, py::arg("num_max_dispatch_tokens_per_rank"),
          py::arg("hidden"), py::arg("num_ranks"), py::arg("num_experts"));
    m.attr("CONTROL_BYTES") = (int64_t)dxh::kControlBytes;
    py::class_<dxh::LowLatencyLayout>(m, "LowLatencyLayout")
        .def(py::init<uint64_t, int, int, int, int>(), py::arg("base"), py::arg("num_max_dispatch_tokens_per_rank"), py::arg("hidden"),
             py::arg("num_ranks"), py::arg("num_experts"))
        .def_readonly("total_bytes", &dxh::LowLatencyLayout::total_bytes)
        .def_property_readonly("counts_off", [](const dxh::LowLatencyLayout& l) { return std::make_pair(l.counts_off[0], l.counts_off[1]); })
        .def_property_readonly("recv_x_off", [](const dxh::LowLatencyLayout& l) { return std::make_pair(l.recv_x_off[0], l.recv_x_off[1]); })
        .def_property_readonly("recv_scales_off", [](const dxh::LowLatencyLayout& l) { return std::make_pair(l.recv_scales_off[0], l.recv_scales_off[1]); })
        .def_property_readonly("recv_src_info_off", [](const dxh::LowLatencyLayout& l) { return std::make_pair(l.recv_src_info_off[0], l.recv_src_info_off[1]); })
        .def_property_readonly("combine_stage_off", [](const dxh::LowLatencyLayout& l) { return std::make_pair(l.combine_stage_off[0], l.combine_stage_off[1]); })
        .def_property_readonly("combine_src_off", [](const dxh::LowLatencyLayout& l) { return std::make_pair(l.combine_src_off[0], l.combine_src_off[1]); });

    py::class_<dxh::Arena>(m, "Arena")
        .def(py::init<uint64_t, uint64_t, uint64_t>(), py::arg("base"), py::arg("size"), py::arg("align") = 1024)
        .def("alloc", &dxh::Arena::alloc)
        .def("free", &dxh::Arena::free)
        .def("shrink", &dxh::Arena::shrink)
        .def("owns", &dxh::Arena::owns)
        .def_property_readonly("capacity", &dxh::Arena::capacity)
        .def_property_readonly("in_use", &dxh::Arena::in_use)
        .def_property_readonly("high_water", &dxh::Arena::high_water)
        .def_property_readonly("num_free_blocks", &dxh::Arena::num_free_blocks)
        .def_property_readonly("largest_free", &dxh::Arena::largest_free);

    m.def("status_name", [](int code) { return std::string(dxh::status_name(code)); });

    py::class_<Runtime>(m, "Runtime")
        .def(py::init<int, int, int64_t, int64_t, int, double, bool>(), py::arg("rank"), py::arg("num_ranks"), py::arg("num_nvl_bytes"),
             py::arg("num_ll_bytes"), py::arg("device"), py::arg("timeout_ms") = 10000.0, py::arg("mask_on_timeout") = false)
        .def("ipc_handle", &Runtime::ipc_handle)
        .def("open_peers", &Runtime::open_peers)
        .def("set_comm_stream", &Runtime::set_comm_stream)
        .def("share_comm_stream", [](Runtime& r) { r.core->share_comm_stream(); })
        .def("alloc_symmetric", &Runtime::alloc_symmetric)
        .def("symmetric_offset", &Runtime::symmetric_offset)
        .def("view", &Runtime::view)
        .def("set_mask", &Runtime::set_mask)
        .def("query_mask", &Runtime::query_mask)
        .def("clean_mask", &Runtime::clean_mask)
        .def("set_timeout_ms", [](Runtime& r, double ms) { r.core->set_timeout_ms(ms); })
        .def("set_debug_checks", [](Runtime& r, bool on) { r.core->set_debug_checks(on); })
        .def("debug_checks", [](Runtime& r) { return r.core->debug_checks(); })
        .def("set_debug_extent", [](Runtime& r, int64_t bytes) { r.core->set_debug_extent((uint64_t)bytes); })
        .def("timeout_ms", [](Runtime& r) { return r.core->timeout_ms(); })
        .def("status_code", [](Runtime& r) { return r.core->status_code(); })
        .def("status_string", [](Runtime& r) { return r.core->status_string(); })
        .def("clear_status", [](Runtime& r) { r.core->clear_status(); })
        .def("enable_trace", [](Runtime& r, bool on) { r.core->enable_trace(on); })
        .def("read_trace", [](Runtime& r) { return r.core->read_trace(); })
        .def("reset_control", [](Runtime& r) { r.core->reset_control(); })
        .def("release", [](Runtime& r) { r.core->release(); })
        .def("is_available", [](Runtime& r) { return r.core->available(); })
        .def("rank", [](Runtime& r) { return r.core->rank(); })
        .def("num_ranks", [](Runtime& r) { return r.core->num_ranks(); })
        .def("device", [](Runtime& r) { return r.core->device(); })
        .def("total_bytes", [](Runtime& r) { return (int64_t)r.core->total_bytes(); })
        .def("arena_capacity", [](Runtime& r) { return (int64_t)r.core->arena().capacity(); })
        .def("arena_in_use", [](Runtime& r) { return (int64_t)r.core->arena().in_use(); })
        .def("arena_high_water", [](Runtime& r) { return (int64_t)r.core->arena().high_water(); })
        .def("ll_bytes", [](Runtime& r) { return (int64_t)r.core->ll_bytes(); });

    m.def("set_local_peers", &set_local_peers);
    m.def("get_dispatch_layout", &get_dispatch_layout);
    m.def("normal_dispatch", &normal_dispatch);
    m.def("normal_combine", &normal_combine);
    m.def("normal_dispatch_on", &normal_dispatch_on);
    m.def("normal_combine_on", &normal_combine_on);
    m.def("barrier", &barrier);
    m.def("timeout_probe", &timeout_probe);
    m.def("per_token_cast_to_fp8", &per_token_cast_to_fp8, py::arg("x"), py::arg("round_scale") = false, py::arg("use_ue8m0") = false,
          py::arg("group_counts") = py::none(), py::arg("rows_per_group") = 1, py::arg("out_q") = py::none(), py::arg("out_s") = py::none(),
          py::arg("num_rows_dev") = py::none(), py::arg("atoms") = false);
    m.def("ll_dispatch", &ll_dispatch);
    m.def("ll_dispatch_one", &ll_dispatch_one);
    m.def("ll_combine_one", &ll_combine_one);
    m.def("ll_combine", &ll_combine, py::arg("runtimes"), py::arg("per_rank"), py::arg("num_max_tokens"), py::arg("num_experts"),
          py::arg("parity"), py::arg("phases"), py::arg("num_sms"), py::arg("pull") = false, py::arg("close_barrier") = false);
    m.def("ll_layout", &ll_layout);
    bind_gemm(m);
    bind_hier(m);
    bind_fused(m);
}
