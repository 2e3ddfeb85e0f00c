// Drives HostStage and StagePool (host_stage.cu) over a stand-in for the CUDA runtime in which copies stay in flight until somebody
// waits for them, so that memory handed on too early is seen.  Exit code 0: all checks hold.
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <map>
#include <set>

#include "../llama2.rs_b200/csrc/host_stage.h"

namespace {
struct Op { void* dst; const void* src; size_t n; size_t mark; };  // a copy, or the mark of an event record
std::map<cudaStream_t, std::deque<Op>> queues;        // work in flight per stream
struct Mark { cudaStream_t st; size_t mark; };
std::map<cudaEvent_t, Mark> recorded;                  // an event's latest record
std::set<const char*> pinned;                          // what cudaPointerGetAttributes calls pinned
int copies_until_error = -1;
size_t events = 0, marks = 0;

void run(cudaStream_t st, size_t until) {  // until: stop behind this mark (0: everything)
    auto& q = queues[st];
    while (!q.empty()) {
        const Op op = q.front();
        q.pop_front();
        if (op.mark) { if (op.mark == until) return; }
        else memcpy(op.dst, op.src, op.n);
    }
}
size_t in_flight() {
    size_t n = 0;
    for (auto& q : queues) for (auto& op : q.second) n += op.mark == 0;
    return n;
}
int errors = 0;
void check(bool ok, const char* what) {
    if (!ok) { printf("FAILED: %s\n", what); errors++; }
}
}  // namespace

extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    a->type = pinned.count(static_cast<const char*>(p)) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { *p = malloc(n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = reinterpret_cast<cudaEvent_t>(++events * 16); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) { queues[st].push_back({nullptr, nullptr, 0, ++marks}); recorded[e] = {st, marks}; return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (!recorded.count(e)) return cudaSuccess;
    const Mark m = recorded[e];
    for (auto& op : queues[m.st]) if (op.mark == m.mark) { run(m.st, m.mark); break; }
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) { run(st, 0); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t st) {
    if (copies_until_error >= 0 && copies_until_error-- == 0) return cudaErrorUnknown;
    queues[st].push_back({dst, src, n, 0});
    return cudaSuccess;
}
}
namespace l2 {
int fail(int code, const char*, ...) { return code; }
}

using namespace l2;

int main() {
    const cudaStream_t s1 = reinterpret_cast<cudaStream_t>(1), s2 = reinterpret_cast<cudaStream_t>(2);
    StagePool::retain();
    auto filled = [](size_t n, int seed) { std::vector<char> v(n); for (size_t i = 0; i < n; i++) v[i] = (char)(i * 31 + i / 251 + seed); return v; };

    // round trips: less than a chunk, whole chunks, more than the ring, odd ends; with a word
    for (size_t n : {(size_t)1, HostStage::CHUNK - 3, HostStage::CHUNK, HostStage::CHUNK * HostStage::SLOTS, HostStage::CHUNK * 9 + 5}) {
        StagePool::Lease l;
        check(l.take(0) == L2_OK, "lease");
        std::vector<char> a = filled(n, 1), dev(n), b(n);
        int word_dev = 77, word = 0;
        check(l->upload(dev.data(), a.data(), n, s1) == L2_OK, "upload");
        check(l->download(b.data(), dev.data(), n, s1, &word_dev, &word) == L2_OK, "download");
        check(a == b && word == 77, "what comes back is what went up");
        check(in_flight() == 0, "a download returns with the stream drained");
    }

    // a call that ends between its upload and its download: nothing of it is in flight when it has returned its error
    for (bool pin : {false, true}) {
        const size_t n = HostStage::CHUNK * 2 + 7;
        std::vector<char> a = filled(n, 2), dev1(n), dev2 = filled(n, 5), b(n);
        const std::vector<char> want1 = a, want2 = dev2;
        if (pin) pinned.insert(a.data());
        {
            StagePool::Lease l;
            l.take(0);
            l->upload(dev1.data(), a.data(), n, s1);
        }  // (the launch behind the upload failed)
        check(in_flight() == 0, "no copy is in flight behind a failed call");
        std::fill(a.begin(), a.end(), 0);  // the caller may use its array again
        {
            StagePool::Lease l;
            l.take(0);
            check(l->download(b.data(), dev2.data(), n, s2) == L2_OK && b == want2, "the next call gets its own data");
        }
        run(s1, 0);
        check(dev1 == want1, "the failed call's upload took the array as it was");
        pinned.clear();
    }

    // copies that fail in the middle of an upload or a download
    for (int at = 0; at < 9; at++)
        for (bool down : {false, true}) {
            const size_t n = HostStage::CHUNK * 8;
            std::vector<char> a = filled(n, 3), dev(n);
            {
                StagePool::Lease l;
                l.take(0);
                copies_until_error = at;
                const int rc = down ? l->download(a.data(), dev.data(), n, s1) : l->upload(dev.data(), a.data(), n, s1);
                check((rc != L2_OK) == (at < 8), "the failure is reported");
                copies_until_error = -1;
            }
            check(in_flight() == 0, "no copy is in flight behind a failed copy");
            queues.clear();
        }
    StagePool::release();
    return errors ? 1 : 0;
}
