// Pinned staging of the callers' arrays (see host_stage.h).
#include "host_stage.h"

#include "model.h"

namespace l2 {

// Pinned arrays need no staging; a device pointer is left to the copy, which refuses it.
static bool direct_copy(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type == cudaMemoryTypeHost || a.type == cudaMemoryTypeDevice;
}

HostStage::~HostStage() {
    for (cudaEvent_t e : done_) if (e) { cudaEventSynchronize(e); cudaEventDestroy(e); }
    if (pin_) cudaFreeHost(pin_);
}

int HostStage::init(int device) {
    device_ = device;
    L2_CUDA(cudaMallocHost(reinterpret_cast<void**>(&pin_), CHUNK * SLOTS + 64));
    for (cudaEvent_t& e : done_) L2_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return L2_OK;
}

int HostStage::upload(void* dst, const void* src, size_t bytes, cudaStream_t st) {
    busy_ = true; busy_on_ = st;
    if (direct_copy(src)) {  // the caller's array itself is the staging memory
        L2_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st));
        return L2_OK;
    }
    int slot = 0;
    for (size_t off = 0; off < bytes; off += CHUNK, slot = (slot + 1) % SLOTS) {
        const size_t n = std::min(CHUNK, bytes - off);
        L2_CUDA(cudaEventSynchronize(done_[slot]));  // the copy that used this slot last has finished
        memcpy(pin_ + slot * CHUNK, static_cast<const char*>(src) + off, n);
        L2_CUDA(cudaMemcpyAsync(static_cast<char*>(dst) + off, pin_ + slot * CHUNK, n, cudaMemcpyHostToDevice, st));
        L2_CUDA(cudaEventRecord(done_[slot], st));
    }
    return L2_OK;
}

void HostStage::drain() {
    if (busy_) cudaStreamSynchronize(busy_on_);
    busy_ = false;
}

int HostStage::download(void* dst, const void* src, size_t bytes, cudaStream_t st, const int* word_dev, int* word) {
    busy_ = true; busy_on_ = st;
    volatile int* pin_word = reinterpret_cast<int*>(pin_ + CHUNK * SLOTS);  // (in front of the data on the stream: there when the data is)
    if (word_dev) L2_CUDA(cudaMemcpyAsync(pin_ + CHUNK * SLOTS, word_dev, sizeof(int), cudaMemcpyDeviceToHost, st));
    if (direct_copy(dst)) {
        L2_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
        L2_CUDA(cudaStreamSynchronize(st));
        busy_ = false;
        if (word_dev) *word = *pin_word;
        return L2_OK;
    }
    const int chunks = (int)((bytes + CHUNK - 1) / CHUNK);
    auto request = [&](int i) -> int {
        const size_t off = (size_t)i * CHUNK, n = std::min(CHUNK, bytes - off);
        L2_CUDA(cudaMemcpyAsync(pin_ + (i % SLOTS) * CHUNK, static_cast<const char*>(src) + off, n, cudaMemcpyDeviceToHost, st));
        L2_CUDA(cudaEventRecord(done_[i % SLOTS], st));
        return L2_OK;
    };
    // (an upload of the same call may still use the slots: its copies come first on the stream)
    for (int i = 0; i < chunks && i < SLOTS; i++)
        if (int rc = request(i)) return rc;
    for (int i = 0; i < chunks; i++) {
        L2_CUDA(cudaEventSynchronize(done_[i % SLOTS]));
        memcpy(static_cast<char*>(dst) + (size_t)i * CHUNK, pin_ + (i % SLOTS) * CHUNK, std::min(CHUNK, bytes - (size_t)i * CHUNK));
        if (i + SLOTS < chunks)
            if (int rc = request(i + SLOTS)) return rc;
    }
    busy_ = false;  // the last copy has been waited for, and with it everything in front of it on the stream
    if (word_dev) *word = *pin_word;
    return L2_OK;
}

std::mutex StagePool::mu_;
std::vector<std::unique_ptr<HostStage>> StagePool::free_;
int StagePool::users_ = 0;

void StagePool::retain() {
    std::lock_guard<std::mutex> g(mu_);
    users_++;
}
void StagePool::release() {
    std::vector<std::unique_ptr<HostStage>> gone;
    std::lock_guard<std::mutex> g(mu_);
    if (--users_ == 0) gone.swap(free_);
}
int StagePool::Lease::take(int device) {
    {
        std::lock_guard<std::mutex> g(mu_);
        for (size_t i = 0; i < free_.size(); i++)
            if (free_[i]->device() == device) {
                s_ = std::move(free_[i]);
                free_.erase(free_.begin() + (long)i);
                return L2_OK;
            }
    }
    std::unique_ptr<HostStage> s(new HostStage);
    if (int rc = s->init(device)) return rc;
    s_ = std::move(s);
    return L2_OK;
}
StagePool::Lease::~Lease() {
    if (!s_) return;
    s_->drain();  // a call that ended in an error: the next owner of the ring, and the caller with its array, find nothing in flight
    std::lock_guard<std::mutex> g(mu_);
    if ((int)free_.size() < KEPT && users_ > 0) free_.push_back(std::move(s_));
}

}  // namespace l2
