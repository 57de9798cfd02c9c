// Staged copies of the host entry points.
//
// A pageable cudaMemcpy goes through the driver's own staging buffer on the
// calling thread: 11.7 GB/s for dgemm_ 2048^3 (67 MB up, 34 MB down), a quarter
// of the PCIe link and most of a call whose product takes 0.55 ms.  Here up to
// eight host threads copy 512 KB chunks into pinned slots and enqueue each
// chunk's device copy themselves; with two slots a thread fills one while the
// other is on the link.  dgemm_ 2048^3 8.1 -> 4.0 ms a call, 1024^3 2.2 -> 1.4.
// Page-locked memory keeps cudaMemcpy2DAsync, and so do transfers under 2 MB and
// a call's only larger one up to 8 MB: starting the threads would not pay.
#include "host_copy.h"

#include <algorithm>
#include <chrono>
#include <cstring>
#include <exception>

namespace zb {

namespace {
// Threads are started per call.  Two transfers of 2 MB repay it (dgemm_ 512^3, three: 460 ->
// 420 us; C of 520 x 520 up and down: 500 -> 340), one does from about 8 MB (one upload of 4 MB
// 335 -> 395 us, of 11 MB 690 -> 650; one download of 2 MB 208 -> 245, of 8 MB 560 -> 530).
constexpr size_t kStagedMinBytes = size_t(2) << 20;
constexpr size_t kLoneMinBytes = size_t(8) << 20;

bool pageable(const void* host) {
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, host) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return attr.type == cudaMemoryTypeUnregistered;
}

// The driver's calls on the current context.  The caller's need not be the device's primary
// one, which is what the runtime gives a new thread.
struct ContextCalls {
    CUresult(CUDAAPI* get)(CUcontext*) = nullptr;
    CUresult(CUDAAPI* set)(CUcontext) = nullptr;
};
const ContextCalls& context_calls() {
    static const ContextCalls calls = [] {
        ContextCalls c;
        cudaDriverEntryPointQueryResult q;
        void *get = nullptr, *set = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &get, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess &&
            cudaGetDriverEntryPoint("cuCtxSetCurrent", &set, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess) {
            c.get = reinterpret_cast<decltype(c.get)>(get);
            c.set = reinterpret_cast<decltype(c.set)>(set);
        }
        return c;
    }();
    return calls;
}
}  // namespace

cudaError_t PinnedSlots::reserve() {
    if (base) return cudaSuccess;
    void* p = nullptr;
    cudaError_t e = cudaHostAlloc(&p, 2 * kThreads * kSlotBytes, cudaHostAllocDefault);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return e;
    }
    base = static_cast<char*>(p);
    for (cudaEvent_t& ev : done)
        if ((e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess) {
            cudaGetLastError();
            release();
            return e;
        }
    return cudaSuccess;
}

void PinnedSlots::release() {
    for (cudaEvent_t& ev : done) {
        if (ev) {
            cudaEventSynchronize(ev);
            cudaEventDestroy(ev);
        }
        ev = nullptr;
    }
    if (base) cudaFreeHost(base);
    base = nullptr;
}

CopyTeam::CopyTeam(PinnedSlots& slots, std::initializer_list<Transfer> transfers) : slots_(slots) {
    int large = 0;
    for (const Transfer& t : transfers) large += t.bytes >= kStagedMinBytes && pageable(t.host);
    min_bytes_ = large > 1 ? kStagedMinBytes : kLoneMinBytes;
}

CopyTeam::~CopyTeam() {
    {
        std::lock_guard<std::mutex> lock(mu_);
        quit_ = true;
        posted_.store(-1, std::memory_order_release);
    }
    start_.notify_all();
    for (std::thread& t : threads_) t.join();
}

// Whether this transfer goes through the slots; starts the threads the first time.
bool CopyTeam::staged(const void* host, size_t width, size_t height) {
    const size_t bytes = width * height, slot = PinnedSlots::kSlotBytes;
    if (bytes < min_bytes_ || !pageable(host)) return false;
    int want = std::min<int>(PinnedSlots::kThreads, (int)std::thread::hardware_concurrency() / 2);
    want = (int)std::min<size_t>(want, (bytes + slot - 1) / slot);  // no more than there are chunks
    if (want < 2 || slots_.reserve() != cudaSuccess) return false;
    if (!context_) {
        const ContextCalls& calls = context_calls();
        if (!calls.set || calls.get(&context_) != CUDA_SUCCESS || !context_) return false;
    }
    try {
        threads_.reserve(want - 1);
        while ((int)threads_.size() < want - 1) {
            const int id = (int)threads_.size() + 1;
            const long seen = generation_;  // no transfer is running: the first one it takes part in is the next
            threads_.emplace_back([this, id, seen] { loop(id, seen); });
        }
    } catch (const std::exception&) {  // no more threads: those that started, and this one, do the work
    }
    return true;
}

void CopyTeam::loop(int id, long seen) {
    const bool bound = context_calls().set(context_) == CUDA_SUCCESS;  // if not, the others do its share
    for (;;) {
        // the transfers of one call follow each other within microseconds: poll for the next
        // one for a while before sleeping (a wake-up costs 50 to 100 us here)
        const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(200);
        while (posted_.load(std::memory_order_acquire) == seen && std::chrono::steady_clock::now() < until)
            std::this_thread::yield();
        {
            std::unique_lock<std::mutex> lock(mu_);
            start_.wait(lock, [&] { return quit_ || generation_ != seen; });
            if (quit_) return;
            seen = generation_;
        }
        if (bound) work(id);
        std::lock_guard<std::mutex> lock(mu_);
        if (--busy_ == 0) finish_.notify_one();
    }
}

// This thread's share of the current job: chunks claimed from a counter, alternating
// between the thread's two slots.  A download's chunk is copied out of its slot while
// the next one is on the link.
void CopyTeam::work(int id) {
    const Job& j = job_;
    struct Chunk {
        size_t col, cols, at, bytes;  // bytes at .. at + bytes of columns col .. col + cols
    } held{};
    int held_slot = -1, turn = 0;
    auto fail = [&](cudaError_t e) {
        int none = 0;
        if (e != cudaSuccess) error_.compare_exchange_strong(none, (int)e);
        return e != cudaSuccess;
    };
    auto rows = [&](const Chunk& c, char* slot, bool in) {
        for (size_t q = 0; q < c.cols; ++q) {
            char* h = j.host + (c.col + q) * j.hpitch + c.at;
            if (in)
                std::memcpy(slot + q * c.bytes, h, c.bytes);
            else
                std::memcpy(h, slot + q * c.bytes, c.bytes);
        }
    };
    // slot <-> device: one run of bytes where the device columns are packed
    auto link = [&](char* dst, size_t dp, const char* src, size_t sp, const Chunk& c, cudaMemcpyKind kind) {
        if (c.cols == 1 || dp == sp) return cudaMemcpyAsync(dst, src, c.bytes * c.cols, kind, j.st);
        return cudaMemcpy2DAsync(dst, dp, src, sp, c.bytes, c.cols, kind, j.st);
    };
    auto flush = [&]() {  // copy the held chunk of a download out
        if (held_slot < 0) return;
        if (!fail(cudaEventSynchronize(slots_.done[held_slot])))
            rows(held, slots_.base + held_slot * PinnedSlots::kSlotBytes, false);
        held_slot = -1;
    };
    for (;;) {
        const size_t n = next_.fetch_add(1);
        if (n >= j.chunks || error_.load()) break;
        Chunk c;
        if (j.pieces > 1) {
            const size_t piece = PinnedSlots::kSlotBytes;
            c = {n / j.pieces, 1, (n % j.pieces) * piece, 0};
            c.bytes = std::min(piece, j.width - c.at);
        } else {
            c = {n * j.cols_per_chunk, 0, 0, j.width};
            c.cols = std::min(j.cols_per_chunk, j.height - c.col);
        }
        const int s = 2 * id + (turn++ & 1);
        char* slot = slots_.base + s * PinnedSlots::kSlotBytes;
        char* dev = j.dev + c.col * j.dpitch + c.at;
        if (fail(cudaEventSynchronize(slots_.done[s]))) break;  // the slot's last device copy
        if (j.up) {
            rows(c, slot, true);
            if (fail(link(dev, j.dpitch, slot, c.bytes, c, cudaMemcpyHostToDevice))) break;
            if (fail(cudaEventRecord(slots_.done[s], j.st))) break;
        } else {
            if (fail(link(slot, c.bytes, dev, j.dpitch, c, cudaMemcpyDeviceToHost))) break;
            if (fail(cudaEventRecord(slots_.done[s], j.st))) break;
            flush();
            held = c;
            held_slot = s;
        }
    }
    flush();
}

cudaError_t CopyTeam::run(Job j) {
    j.cols_per_chunk = std::max<size_t>(1, PinnedSlots::kSlotBytes / std::max<size_t>(1, j.width));
    j.pieces = j.width > PinnedSlots::kSlotBytes ? (j.width + PinnedSlots::kSlotBytes - 1) / PinnedSlots::kSlotBytes : 1;
    j.chunks = j.pieces > 1 ? j.height * j.pieces : (j.height + j.cols_per_chunk - 1) / j.cols_per_chunk;
    {
        std::lock_guard<std::mutex> lock(mu_);
        job_ = j;
        next_.store(0);
        error_.store(0);
        busy_ = (int)threads_.size();
        posted_.store(++generation_, std::memory_order_release);
    }
    start_.notify_all();
    work(0);
    std::unique_lock<std::mutex> lock(mu_);
    finish_.wait(lock, [&] { return busy_ == 0; });
    return static_cast<cudaError_t>(error_.load());
}

cudaError_t CopyTeam::upload(void* dev, size_t dpitch, const void* host, size_t hpitch, size_t width, size_t height,
                             cudaStream_t st) {
    if (!staged(host, width, height))
        return cudaMemcpy2DAsync(dev, dpitch, host, hpitch, width, height, cudaMemcpyHostToDevice, st);
    Job j;
    j.up = true;
    j.host = static_cast<char*>(const_cast<void*>(host));
    j.dev = static_cast<char*>(dev);
    j.hpitch = hpitch;
    j.dpitch = dpitch;
    j.width = width;
    j.height = height;
    j.st = st;
    return run(j);
}

cudaError_t CopyTeam::download(void* host, size_t hpitch, const void* dev, size_t dpitch, size_t width, size_t height,
                               cudaStream_t st) {
    if (!staged(host, width, height))
        return cudaMemcpy2DAsync(host, hpitch, dev, dpitch, width, height, cudaMemcpyDeviceToHost, st);
    Job j;
    j.up = false;
    j.host = static_cast<char*>(host);
    j.dev = static_cast<char*>(const_cast<void*>(dev));
    j.hpitch = hpitch;
    j.dpitch = dpitch;
    j.width = width;
    j.height = height;
    j.st = st;
    return run(j);
}

}  // namespace zb
