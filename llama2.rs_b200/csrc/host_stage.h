// Host <-> device copies of the callers' ordinary (pageable) arrays through pinned staging memory.
//
// The driver's own path for pageable memory stages through one buffer and waits for it: 57 us up and 65 us down for the 757 KB of a
// 37-row batch, 23 us of it DMA.  Here the array goes through a ring of chunks, so that copying one chunk and the DMA of the others
// overlap (5120 x 5120, 37 rows on host arrays: 177 -> 161 us a call).  Arrays that are pinned already are copied directly.
#pragma once

#include <cuda_runtime.h>

#include <cstring>
#include <memory>
#include <mutex>
#include <vector>

#include "host_common.h"

namespace l2 {

class HostStage {
public:
    static constexpr size_t CHUNK = (size_t)256 << 10;
    static constexpr int SLOTS = 4;
    ~HostStage();
    int init(int device);
    int device() const { return device_; }
    // The copies of a call are on one stream.  src stays as it is until a download has returned, or drain.
    int upload(void* dst, const void* src, size_t bytes, cudaStream_t st);
    // returns when dst holds the data; word_dev (may be null): one more int that comes along
    int download(void* dst, const void* src, size_t bytes, cudaStream_t st, const int* word_dev = nullptr, int* word = nullptr);
    void drain();  // waits for an upload without a download behind it, or a copy that failed in the middle
private:
    int device_ = -1;
    bool busy_ = false;               // copies may be in flight ...
    cudaStream_t busy_on_ = nullptr;  // ... on this stream
    char* pin_ = nullptr;
    cudaEvent_t done_[SLOTS] = {};
};

// Staging rings not in use right now, at most KEPT of them, given back when the last handle that may use them is closed.  A call takes
// one for its duration, so calls on several threads and streams never share one.
class StagePool {
public:
    static void retain();   // a handle that will use staging was made ...
    static void release();  // ... and closed
    class Lease {
    public:
        Lease() = default;
        ~Lease();
        int take(int device);
        HostStage* operator->() const { return s_.get(); }
    private:
        std::unique_ptr<HostStage> s_;
    };
private:
    static constexpr int KEPT = 4;
    static std::mutex mu_;
    static std::vector<std::unique_ptr<HostStage>> free_;
    static int users_;
};

}  // namespace l2
