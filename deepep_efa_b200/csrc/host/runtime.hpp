// Per-rank host runtime: owns the symmetric buffer (cudaMalloc + CUDA IPC), the arena carved out of
// it, the mapped host words the kernels report through, and the rank-local device state (tickets,
// sequence counters). One instance per rank; a single process may own several (single-GPU emulation
// of a multi-rank job, where "peers" are simply the other instances' buffers).
//
// Reference counterparts: deep_ep::Buffer constructor / sync / destroy (csrc/deep_ep.cpp:206-515),
// SharedMemoryAllocator (csrc/deep_ep.cpp:93-202), mapped counters (csrc/deep_ep.cpp:281-296).
// Differences: no NVSHMEM/EFA state, no workspace, outputs are carved from the symmetric arena, errors
// come back through a status block instead of a device trap.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <deque>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>

#include "../kernels/api.h"
#include "arena.hpp"
#include "config.hpp"

namespace dxh {

#define DX_CUDA_CHECK(expr)                                                                              \
    do {                                                                                                 \
        cudaError_t _e = (expr);                                                                         \
        if (_e != cudaSuccess) {                                                                         \
            char _buf[512];                                                                              \
            std::snprintf(_buf, sizeof(_buf), "CUDA error %s (%s) at %s:%d: %s", cudaGetErrorName(_e),   \
                          cudaGetErrorString(_e), __FILE__, __LINE__, #expr);                            \
            cudaGetLastError();                                                                          \
            throw std::runtime_error(_buf);                                                              \
        }                                                                                                \
    } while (0)

inline const char* status_name(int code) {
    switch (code) {
        case dx::kOk: return "ok";
        case dx::kTimeoutBarrier: return "timeout in cross-rank barrier";
        case dx::kTimeoutNotify: return "timeout waiting for token counts (notify)";
        case dx::kTimeoutDescriptor: return "timeout waiting for a peer's receive descriptor";
        case dx::kTimeoutLLCount: return "timeout waiting for low-latency expert counts";
        case dx::kTimeoutLLData: return "timeout waiting for low-latency dispatch rows";
        case dx::kTimeoutCombineReady: return "timeout waiting for a peer's combine source";
        case dx::kTimeoutCombineData: return "timeout waiting for low-latency combine rows";
        case dx::kTimeoutGemm: return "timeout inside grouped GEMM pipeline";
        case dx::kBadArgument: return "kernel rejected its arguments";
        case dx::kTimeoutTest: return "timeout probe (expected in tests)";
        case dx::kTimeoutFusedNotify: return "timeout waiting for expert counts (expert-major dispatch)";
        case dx::kBadPeerAccess: return "debug bounds check: a row address fell outside the peer's symmetric buffer (access skipped)";
        default: return "unknown status";
    }
}

// Host words the device writes; all in one mapped pinned allocation.
struct HostWords {
    dx::StatusBlock status;
    volatile int recv_counter;                         // -1 = not yet, -2 = notify failed
    volatile int expert_counter[dx::kMaxLocalExperts];
};

constexpr int kLocalScratchInts = 64;
// sequences + low-latency expected arrivals + expected rows per local expert of the expert-major dispatch
constexpr int kLocalSeqWords = dx::kNumLocalSeqWords;

class RuntimeCore {
  public:
    RuntimeCore(int rank, int num_ranks, uint64_t num_nvl_bytes, uint64_t num_ll_bytes, int device, double timeout_ms,
                bool mask_on_timeout)
        : rank_(rank), num_ranks_(num_ranks), device_(device), mask_on_timeout_(mask_on_timeout) {
        if (num_ranks < 1 || num_ranks > dx::kMaxRanks) throw std::invalid_argument("num_ranks must be in [1, 8]: one NVSwitch domain");
        if (rank < 0 || rank >= num_ranks) throw std::invalid_argument("rank out of range");
        DX_CUDA_CHECK(cudaSetDevice(device_));
        ll_base_ = kControlBytes;
        ll_bytes_ = align_up(num_ll_bytes, 1024);
        const uint64_t arena_base = ll_base_ + ll_bytes_;
        const uint64_t arena_bytes = num_nvl_bytes > kControlBytes ? align_up(num_nvl_bytes - kControlBytes, 1024) : 0;
        total_bytes_ = arena_base + arena_bytes;
        DX_CUDA_CHECK(cudaMalloc(&base_, total_bytes_));
        // control block, and the low-latency region: its count words carry validity tags and must not start with stale ones
        DX_CUDA_CHECK(cudaMemset(base_, 0, kControlBytes + ll_bytes_));
        arena_.reset(arena_base, arena_bytes);
        DX_CUDA_CHECK(cudaMalloc(&local_scratch_, kLocalScratchInts * sizeof(int)));
        DX_CUDA_CHECK(cudaMemset(local_scratch_, 0, kLocalScratchInts * sizeof(int)));
        DX_CUDA_CHECK(cudaMalloc(&local_seq_, kLocalSeqWords * sizeof(uint64_t)));
        DX_CUDA_CHECK(cudaMemset(local_seq_, 0, kLocalSeqWords * sizeof(uint64_t)));
        DX_CUDA_CHECK(cudaMalloc(&never_set_flag_, sizeof(uint64_t)));
        DX_CUDA_CHECK(cudaMemset(never_set_flag_, 0, sizeof(uint64_t)));
        DX_CUDA_CHECK(cudaHostAlloc(reinterpret_cast<void**>(&host_), sizeof(HostWords), cudaHostAllocMapped));
        std::memset((void*)host_, 0, sizeof(HostWords));
        host_->recv_counter = -1;
        DX_CUDA_CHECK(cudaHostGetDevicePointer(reinterpret_cast<void**>(&host_dev_), (void*)host_, 0));
        int khz = 0;
        DX_CUDA_CHECK(cudaDeviceGetAttribute(&khz, cudaDevAttrClockRate, device_));
        clock_khz_ = khz > 0 ? khz : 1965000;
        set_timeout_ms(timeout_ms);
        if (const char* e = std::getenv("DEEPEP_DEBUG_CHECKS"); e != nullptr && e[0] == '1') debug_checks_ = true;
        for (int i = 0; i < dx::kMaxRanks; ++i) peers_[i] = nullptr;
        peers_[rank_] = base_;
        DX_CUDA_CHECK(cudaDeviceSynchronize());
    }

    ~RuntimeCore() { release(); }

    void set_debug_checks(bool on) { debug_checks_ = on; }
    bool debug_checks() const { return debug_checks_; }
    // Test hook: check row addresses against a smaller extent than the real allocation (0 = the real size), so that a test
    // can provoke a violation with an address that still lies inside this rank's own buffer.
    void set_debug_extent(uint64_t bytes) { debug_extent_override_ = bytes; }

    void set_timeout_ms(double ms) {
        timeout_ms_ = ms;
        timeout_cycles_ = (long long)(ms * (double)clock_khz_);
    }
    double timeout_ms() const { return timeout_ms_; }

    std::string ipc_handle() const {
        cudaIpcMemHandle_t h;
        DX_CUDA_CHECK(cudaIpcGetMemHandle(&h, base_));
        return std::string(reinterpret_cast<const char*>(&h), sizeof(h));
    }

    // Real multi-process bootstrap: handles[r] is rank r's IPC handle, device_ids[r] its CUDA device.
    void open_peers(const std::vector<std::string>& handles) {
        if ((int)handles.size() != num_ranks_) throw std::invalid_argument("open_peers: need one handle per rank");
        DX_CUDA_CHECK(cudaSetDevice(device_));
        for (int r = 0; r < num_ranks_; ++r) {
            if (r == rank_) continue;
            if (handles[r].size() != sizeof(cudaIpcMemHandle_t)) throw std::invalid_argument("open_peers: bad handle size");
            cudaIpcMemHandle_t h;
            std::memcpy(&h, handles[r].data(), sizeof(h));
            void* p = nullptr;
            DX_CUDA_CHECK(cudaIpcOpenMemHandle(&p, h, cudaIpcMemLazyEnablePeerAccess));
            peers_[r] = p;
            ipc_opened_[r] = true;
        }
        available_ = true;
    }

    // Single-process emulation: the peers are other RuntimeCore objects on the same device.
    void set_local_peers(const std::vector<RuntimeCore*>& all) {
        if ((int)all.size() != num_ranks_) throw std::invalid_argument("set_local_peers: need one runtime per rank");
        for (int r = 0; r < num_ranks_; ++r) peers_[r] = all[r]->base_;
        available_ = true;
    }

    void release() {
        if (released_) return;
        released_ = true;
        cudaSetDevice(device_);
        cudaDeviceSynchronize();
        drain_pending(Drain::kWait);
        order_ = capture_order_ = Order{};
        for (cudaEvent_t ev : event_pool_) cudaEventDestroy(ev);
        event_pool_.clear();
        for (int r = 0; r < num_ranks_; ++r)
            if (ipc_opened_[r]) cudaIpcCloseMemHandle(peers_[r]);
        if (base_) cudaFree(base_);
        if (local_scratch_) cudaFree(local_scratch_);
        if (local_seq_) cudaFree(local_seq_);
        if (never_set_flag_) cudaFree(never_set_flag_);
        if (trace_) cudaFree(trace_);
        trace_ = nullptr;
        if (host_) cudaFreeHost((void*)host_);
        base_ = nullptr;
        available_ = false;
    }

    dx::RankCtx ctx() const {
        dx::RankCtx c;
        c.rank = rank_;
        c.num_ranks = num_ranks_;
        for (int i = 0; i < dx::kMaxRanks; ++i) c.peers[i] = peers_[i];
        c.status = &host_dev_->status;
        c.local_scratch = local_scratch_;
        c.seq = local_seq_;
        c.trace = trace_;
        c.timeout_cycles = timeout_cycles_;
        c.mask_on_timeout = mask_on_timeout_ ? 1 : 0;
        c.debug_extent = debug_checks_ ? (unsigned long long)(debug_extent_override_ != 0 ? debug_extent_override_ : total_bytes_) : 0ull;
        return c;
    }

    // ---- arena ------------------------------------------------------------------------------
    // Fresh blocks of the given sizes. Blocks released earlier become reusable once the streams that may still touch them have passed
    // the events recorded at release time. With `roomy`, nothing happens and false is returned unless the largest free block is at
    // least that large.
    bool arena_alloc(const uint64_t* bytes, int n, uint64_t* offs, uint64_t roomy = 0) {
        std::lock_guard<std::mutex> g(mu_);
        for (Drain how : {Drain::kFront, Drain::kAll, Drain::kWait}) {
            drain_pending(how);
            if (roomy > 0 && arena_.largest_free() < roomy) {
                if (how == Drain::kFront) continue;
                return false;
            }
            int i = 0;
            for (; i < n; ++i) {
                const int64_t off = arena_.alloc(bytes[i]);
                if (off < 0) break;
                offs[i] = (uint64_t)off;
            }
            if (i == n) return true;
            const uint64_t need = bytes[i];
            while (i-- > 0) arena_.free(offs[i]);
            if (how != Drain::kWait) continue;
            char buf[512];
            std::snprintf(buf, sizeof(buf),
                          "symmetric arena exhausted: need %llu B, capacity %llu B, in use %llu B, largest free block %llu B. "
                          "Create the Buffer with a larger num_nvl_bytes (Config.get_nvl_buffer_size_hint) or drop references "
                          "to earlier dispatch results.",
                          (unsigned long long)need, (unsigned long long)arena_.capacity(), (unsigned long long)arena_.in_use(),
                          (unsigned long long)arena_.largest_free());
            throw std::runtime_error(buf);
        }
        return false;
    }

    // Gives back the end of a block that nothing has used or will use.
    void arena_shrink(uint64_t off, uint64_t bytes) {
        std::lock_guard<std::mutex> g(mu_);
        if (!released_) arena_.shrink(off, bytes);
    }

    // Called when the last tensor of a block dies (any thread). `streams` (up to two, nullptr = the default stream) are the
    // streams whose queued work may still use the block. So may the ordered calls (below), on whatever stream they ran: the last of
    // them is behind all others, so when it was on neither of these streams its event is waited for as well. Events come from a
    // pool: creating and destroying them cost more than everything else here.
    void arena_release(uint64_t off, const cudaStream_t* streams, int num_streams) {
        std::lock_guard<std::mutex> g(mu_);
        if (released_) return;
        Pending p;
        p.off = off;
        int prev = -1;
        cudaGetDevice(&prev);
        if (prev != device_) cudaSetDevice(device_);
        bool covered = order_.event == nullptr;
        for (int i = 0; i < num_streams; ++i) {
            if (i == 1 && streams[1] == streams[0]) break;
            cudaEvent_t ev = take_event();
            if (ev == nullptr) continue;
            if (cudaEventRecord(ev, streams[i]) == cudaSuccess) {
                p.events[p.num_events++] = ev;
                covered = covered || streams[i] == order_.stream;
            } else {
                event_pool_.push_back(ev);
            }
        }
        if (!covered) p.last_call = order_.event;
        cudaGetLastError();
        if (prev != device_ && prev >= 0) cudaSetDevice(prev);
        pending_.push_back(p);
    }

    // ---- order of the normal-mode and expert-major kernels ------------------------------------
    // They share state (sequence numbers, tickets, count words, the layout scratch), so one must not overlap the next one. A call runs on the
    // caller's stream, or on the communication stream when the caller asked for an event; a call on another stream than the
    // last one waits for that one's event first. Enter before the first launch of a call and leave after the last one, with
    // nothing in between that lets another host thread in (a wait for the GPU): a call that waits leaves before it does.
    // Calls under stream capture are ordered among those of the same capture. With calls outside of it they are not: an event
    // from outside may not be waited for there, and the graph's owner orders its replays.
    struct Order;
    struct Place {  // of one call, from enter to leave
        Order* order = nullptr;
        unsigned long long capture = 0;
        bool captured = false;
    };
    Place order_enter(cudaStream_t s) {
        std::lock_guard<std::mutex> g(mu_);
        const Place at = place_of(s);
        const Order* o = at.order;
        if (o != nullptr && o->event != nullptr && o->capture == at.capture && o->stream != s) DX_CUDA_CHECK(cudaStreamWaitEvent(s, *o->event, 0));
        return at;
    }
    void order_leave(cudaStream_t s, const Place& at) {
        std::lock_guard<std::mutex> g(mu_);
        Order* o = at.order;
        if (o == nullptr) return;
        if (o->event == nullptr || o->event.use_count() > 1) {  // a block released meanwhile waits for that call, not for this one
            const cudaEvent_t ev = take_event();
            o->event = ev == nullptr ? nullptr : std::shared_ptr<cudaEvent_t>(new cudaEvent_t(ev), [this](cudaEvent_t* e) {
                event_pool_.push_back(*e);  // (under mu_, like every use of these pointers)
                delete e;
            });
        }
        if (o->event != nullptr) cudaEventRecord(*o->event, s);
        else comm_shared_ = true;
        o->stream = s;
        o->capture = at.capture;
        cudaGetLastError();
    }
    struct Order {
        std::shared_ptr<cudaEvent_t> event;  // end of the last call, recorded on `stream`
        cudaStream_t stream = nullptr;
        unsigned long long capture = 0;  // the capture it belongs to, 0 = none
    };

    // The communication stream runs ordered calls, which a release waits for by their event. Once it is shared (a caller has asked for it,
    // or other kernels of this library run there) a release records an event of its own on it.
    void share_comm_stream() { comm_shared_ = true; }
    bool comm_stream_shared() const { return comm_shared_; }

    bool in_symmetric(const void* p, uint64_t bytes, uint64_t* off) const {
        const char* b = reinterpret_cast<const char*>(base_);
        const char* q = reinterpret_cast<const char*>(p);
        if (q < b || q + bytes > b + total_bytes_) return false;
        *off = (uint64_t)(q - b);
        return true;
    }

    // ---- host <-> device words ----------------------------------------------------------------
    void reset_recv_counters(int num_local_experts) {
        host_->recv_counter = -1;
        for (int i = 0; i < num_local_experts; ++i) host_->expert_counter[i] = -1;
    }

    // Spins until the notify kernel has published the receive counts. Bounded by the host timeout.
    int wait_recv_counts(int num_local_experts, std::vector<int>* per_expert) {
        const auto t0 = std::chrono::steady_clock::now();
        const double limit_ms = timeout_ms_ * 2 + 1000.0;
        while (true) {
            const int n = host_->recv_counter;
            bool ready = n >= 0;
            if (n == -2) raise_status("dispatch");
            if (ready)
                for (int i = 0; i < num_local_experts; ++i) ready = ready && host_->expert_counter[i] >= 0;
            if (ready) {
                per_expert->resize(num_local_experts);
                for (int i = 0; i < num_local_experts; ++i) (*per_expert)[i] = host_->expert_counter[i];
                return n;
            }
            const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
            if (ms > limit_ms) {
                if (host_->status.code != 0) raise_status("dispatch");
                throw std::runtime_error("dispatch: host timed out waiting for the receive counts (did every rank call dispatch?)");
            }
        }
    }

    // ---- tracing -------------------------------------------------------------------------------
    // Kernels stamp the GPU global timer at phase boundaries of their first and last CTA.
    void enable_trace(bool on) {
        DX_CUDA_CHECK(cudaSetDevice(device_));
        if (on && trace_ == nullptr) {
            DX_CUDA_CHECK(cudaMalloc(&trace_, kTraceWords * sizeof(unsigned long long)));
            DX_CUDA_CHECK(cudaMemset(trace_, 0, kTraceWords * sizeof(unsigned long long)));
        } else if (!on && trace_ != nullptr) {
            DX_CUDA_CHECK(cudaDeviceSynchronize());
            cudaFree(trace_);
            trace_ = nullptr;
        }
    }
    std::vector<unsigned long long> read_trace() {
        std::vector<unsigned long long> v(kTraceWords, 0);
        if (trace_ != nullptr) {
            DX_CUDA_CHECK(cudaSetDevice(device_));
            DX_CUDA_CHECK(cudaDeviceSynchronize());
            DX_CUDA_CHECK(cudaMemcpy(v.data(), trace_, kTraceWords * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
        }
        return v;
    }

    int status_code() const { return read_word(&host_->status.code); }
    std::string status_string() const {
        const int code = read_word(&host_->status.code), rank = read_word(&host_->status.rank);
        const int peer = read_word(&host_->status.peer), detail = read_word(&host_->status.detail);
        char buf[256];
        std::snprintf(buf, sizeof(buf), "%s [code %d, rank %d, peer %d, detail %d]", status_name(code), code, rank, peer, detail);
        return std::string(buf);
    }
    void clear_status() { std::memset((void*)&host_->status, 0, sizeof(dx::StatusBlock)); }
    void raise_status(const char* where) {
        std::string m = std::string(where) + ": " + status_string();
        throw std::runtime_error("EPTimeoutError: " + m);
    }

    // Zeroes the control block and the rank-local sequence state. Call on every rank, between two
    // host-level barriers, with no kernel of this Buffer in flight.
    void reset_control() {
        DX_CUDA_CHECK(cudaSetDevice(device_));
        DX_CUDA_CHECK(cudaDeviceSynchronize());
        DX_CUDA_CHECK(cudaMemset(base_, 0, kControlBytes + ll_bytes_));  // sequences restart, so no tagged count word may survive
        DX_CUDA_CHECK(cudaMemset(local_scratch_, 0, kLocalScratchInts * sizeof(int)));
        DX_CUDA_CHECK(cudaMemset(local_seq_, 0, kLocalSeqWords * sizeof(uint64_t)));
        DX_CUDA_CHECK(cudaDeviceSynchronize());
        clear_status();
    }

    int rank() const { return rank_; }
    int num_ranks() const { return num_ranks_; }
    int device() const { return device_; }
    bool available() const { return available_; }
    void* base() const { return base_; }
    uint64_t total_bytes() const { return total_bytes_; }
    uint64_t ll_base() const { return ll_base_; }
    uint64_t ll_bytes() const { return ll_bytes_; }
    const Arena& arena() const { return arena_; }
    uint64_t* never_set_flag() const { return never_set_flag_; }
    uint64_t* local_seq() const { return local_seq_; }
    dx::ControlBlock* control() const { return reinterpret_cast<dx::ControlBlock*>(base_); }

  private:
    static int read_word(const int* p) { return *reinterpret_cast<const volatile int*>(p); }

    struct Pending {
        uint64_t off = 0;
        cudaEvent_t events[2];
        int num_events = 0;
        std::shared_ptr<cudaEvent_t> last_call;  // of the ordered calls, where the events do not cover it
    };

    // What a call on `s` is ordered by; nothing when the driver will not say (the default stream while another stream captures).
    Place place_of(cudaStream_t s) {
        Place at;
        cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &st) != cudaSuccess) cudaGetLastError();
        else if (st == cudaStreamCaptureStatusNone) at.order = &order_;
        else if (cudaStreamGetCaptureInfo(s, &st, &at.capture) == cudaSuccess && st == cudaStreamCaptureStatusActive) at.order = &capture_order_;
        at.captured = st != cudaStreamCaptureStatusNone;
        return at;
    }

    cudaEvent_t take_event() {
        cudaEvent_t ev = nullptr;
        if (!event_pool_.empty()) {
            ev = event_pool_.back();
            event_pool_.pop_back();
        } else if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
            ev = nullptr;
        }
        return ev;
    }

    // kFront stops at the first release that has not passed: they pass nearly in order, and every look at an event costs the host more
    // than the rest of an allocation.
    enum class Drain { kFront, kAll, kWait };
    void drain_pending(Drain how) {
        const bool wait = how == Drain::kWait;
        for (auto it = pending_.begin(); it != pending_.end();) {
            auto passed = [&](cudaEvent_t ev) { return (wait ? cudaEventSynchronize(ev) : cudaEventQuery(ev)) != cudaErrorNotReady; };
            bool done = it->last_call == nullptr || passed(*it->last_call);
            for (int i = 0; done && i < it->num_events; ++i) done = passed(it->events[i]);
            if (done) {
                for (int i = 0; i < it->num_events; ++i) event_pool_.push_back(it->events[i]);
                arena_.free(it->off);
                it = pending_.erase(it);
            } else if (how == Drain::kFront) {
                break;
            } else {
                ++it;
            }
        }
        cudaGetLastError();
    }

    int rank_, num_ranks_, device_;
    bool mask_on_timeout_ = false;
    uint64_t debug_extent_override_ = 0;
    bool debug_checks_ = false;  // range-check row addresses on the device (env DEEPEP_DEBUG_CHECKS=1 or set_debug_checks)
    bool available_ = false, released_ = false;
    void* base_ = nullptr;
    uint64_t total_bytes_ = 0, ll_base_ = 0, ll_bytes_ = 0;
    void* peers_[dx::kMaxRanks];
    bool ipc_opened_[dx::kMaxRanks] = {false, false, false, false, false, false, false, false};
    int* local_scratch_ = nullptr;
    uint64_t* local_seq_ = nullptr;
    uint64_t* never_set_flag_ = nullptr;
    unsigned long long* trace_ = nullptr;
    static constexpr int kTraceWords = dx::kNumFamilies * 2 * dx::kTraceStampsPerSlot;
    HostWords* host_ = nullptr;
    HostWords* host_dev_ = nullptr;
    int clock_khz_ = 1965000;
    double timeout_ms_ = 10000.0;
    long long timeout_cycles_ = 0;
    Arena arena_;
    std::deque<Pending> pending_;
    std::vector<cudaEvent_t> event_pool_;  // bounded by the number of blocks that were ever pending at once
    Order order_, capture_order_;
    std::atomic<bool> comm_shared_{false};
    std::mutex mu_;
};

// The launches of one call on one stream, ordered behind the previous call's (RuntimeCore::order_enter) of every rank that takes part.
class OrderedCall {
  public:
    explicit OrderedCall(cudaStream_t s) : stream(s) {}
    OrderedCall(const OrderedCall&) = delete;
    ~OrderedCall() { leave(); }
    void add(RuntimeCore* core) {
        if (n_ == dx::kMaxRanks) throw std::invalid_argument("OrderedCall: too many ranks");
        cores_[n_++] = core;
    }
    void enter() {
        if (inside_) return;
        for (int i = 0; i < n_; ++i) places_[i] = cores_[i]->order_enter(stream);
        inside_ = true;
    }
    void leave() {
        if (!inside_) return;
        for (int i = 0; i < n_; ++i) cores_[i]->order_leave(stream, places_[i]);
        inside_ = false;
    }
    bool captured() const { return inside_ && places_[0].captured; }
    const cudaStream_t stream;

  private:
    RuntimeCore* cores_[dx::kMaxRanks];
    RuntimeCore::Place places_[dx::kMaxRanks];
    int n_ = 0;
    bool inside_ = false;
};

}  // namespace dxh
