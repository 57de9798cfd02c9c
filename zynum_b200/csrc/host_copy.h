// Copies between pageable host matrices and device buffers by several host threads.
#pragma once

#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <initializer_list>
#include <mutex>
#include <thread>
#include <vector>

#include <cuda.h>
#include <cuda_runtime.h>

namespace zb {

// Pinned staging slots of the host entry points (kept by the context, released
// by its shutdown): two per copying thread.
struct PinnedSlots {
    static constexpr int kThreads = 8;              // most copying threads
    static constexpr size_t kSlotBytes = 1 << 19;
    char* base = nullptr;
    cudaEvent_t done[2 * kThreads] = {};            // last device copy out of / into each slot
    cudaError_t reserve();
    void release();
};

// The copying threads of one host call: started on the first transfer that takes
// them, in the calling thread's CUDA context, joined by the destructor.  The caller
// holds the context's mutex, so one team uses the slots at a time.
class CopyTeam {
  public:
    struct Transfer {
        const void* host;
        size_t bytes;
    };
    // transfers: what the call will copy, for the decision whether threads pay.
    CopyTeam(PinnedSlots& slots, std::initializer_list<Transfer> transfers);
    ~CopyTeam();
    CopyTeam(const CopyTeam&) = delete;
    CopyTeam& operator=(const CopyTeam&) = delete;

    // width x height bytes (height columns of `width` bytes, pitches in bytes), ordered after
    // earlier work on `st`.  upload: on return the source has been read (staged copies) or the
    // copy is enqueued (cudaMemcpy2DAsync).  download: on return the staged form has written
    // the destination; otherwise the copy is enqueued.
    cudaError_t upload(void* dev, size_t dpitch, const void* host, size_t hpitch, size_t width, size_t height,
                       cudaStream_t st);
    cudaError_t download(void* host, size_t hpitch, const void* dev, size_t dpitch, size_t width, size_t height,
                         cudaStream_t st);

  private:
    struct Job {
        bool up = true;
        char* host = nullptr;
        char* dev = nullptr;
        size_t hpitch = 0, dpitch = 0, width = 0, height = 0;
        size_t cols_per_chunk = 1, pieces = 1, chunks = 0;  // a column longer than a slot goes in pieces
        cudaStream_t st = nullptr;
    };
    bool staged(const void* host, size_t width, size_t height);
    cudaError_t run(Job j);
    void work(int id);
    void loop(int id, long seen);

    PinnedSlots& slots_;
    size_t min_bytes_;             // smallest transfer that takes the threads
    CUcontext context_ = nullptr;  // the calling thread's, for the copying threads
    std::vector<std::thread> threads_;
    std::mutex mu_;
    std::condition_variable start_, finish_;
    Job job_;
    long generation_ = 0;            // jobs posted so far (under mu_)
    std::atomic<long> posted_{0};    // the same for polling; -1: leave
    int busy_ = 0;
    bool quit_ = false;
    std::atomic<size_t> next_{0};
    std::atomic<int> error_{0};
};

}  // namespace zb
