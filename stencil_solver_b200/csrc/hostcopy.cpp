// Device -> pageable host copies of whole fields.
//
// The driver stages such a copy through its own pinned buffer with one thread, and that
// thread also takes the page faults of a freshly allocated destination: 38 MB arrive in 2.0
// ms when the pages are not new, in 8.5 when they are (huge pages; 18 ms in small ones).
// Here several threads touch the destination a chunk ahead of the copy: 5.2 ms and 12.5 ms
// with chunks of 16 MB (4 MB: 5.5 and 20).  Nothing outlives the call; pinned buffers of
// the library's own and as many copying threads took 3.5 ms, but pinning them first took
// 2 to 9 ms.  A destination whose pages are in place is copied to in one call: starting
// the threads for it cost 0.2 ms and the chunks 1 to 10 % (5.6 MB 0.53 instead of 0.37 ms).
#include <cuda_runtime.h>
#include <sched.h>
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <memory>
#include <thread>
#include <vector>

#include "kernels.h"

namespace sb200 {

namespace {

constexpr size_t kChunk = size_t(16) << 20;  // one copy
constexpr size_t kDirect = size_t(4) << 20;  // shorter copies go straight to the driver
constexpr size_t kPage = 4096;

bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Whether the pages of [p, p + n) are in place, judged by 16 of them.  (A new page
// among the others costs its fault, nothing else.)
bool in_place(const char* p, size_t n) {
    const uintptr_t first = reinterpret_cast<uintptr_t>(p) & ~(kPage - 1);
    const size_t last = (reinterpret_cast<uintptr_t>(p) + n - 1 - first) / kPage;
    for (size_t k = 0; k < 16; ++k) {
        unsigned char in = 0;
        if (mincore(reinterpret_cast<void*>(first + last * k / 15 * kPage), kPage, &in) != 0 || !(in & 1))
            return false;
    }
    return true;
}

// Threads that touch pages: the process' CPUs less the copying one, at most 8.
int touch_threads() {
    cpu_set_t set;
    CPU_ZERO(&set);
    if (sched_getaffinity(0, sizeof(set), &set) != 0) return 0;
    return std::max(0, std::min(8, CPU_COUNT(&set) - 1));
}

// Threads that write one byte of each page of dst back, chunk by chunk; `wait(c)` returns
// once chunk c has been touched (by every thread that could be started).
class Toucher {
public:
    Toucher(char* dst, size_t bytes)
        : dst_(dst), bytes_(bytes), chunks_((bytes + kChunk - 1) / kChunk) {
        const int n = touch_threads();
        try {
            done_.reset(new std::atomic<int>[chunks_]());
            threads_.reserve(n);
            for (int k = 0; k < n; ++k) threads_.emplace_back([this, k, n] { touch(k, n); });
        } catch (...) {  // no memory or no thread: the copy takes the remaining faults
        }
    }
    ~Toucher() {
        for (std::thread& t : threads_) t.join();
    }
    void wait(size_t c) {
        while (!threads_.empty() && done_[c].load(std::memory_order_acquire) < int(threads_.size()))
            std::this_thread::yield();
    }

private:
    void touch(int k, int n) {
        for (size_t c = 0; c < chunks_; ++c) {
            const size_t len = std::min(kChunk, bytes_ - c * kChunk), part = (len + n - 1) / n;
            const size_t b = std::min(len, part * k), e = std::min(len, b + part);
            volatile char* p = dst_ + c * kChunk;
            for (size_t i = b; i < e; i += kPage) p[i] = p[i];
            done_[c].fetch_add(1, std::memory_order_release);
        }
    }

    char* dst_;
    size_t bytes_, chunks_;
    std::unique_ptr<std::atomic<int>[]> done_;
    std::vector<std::thread> threads_;
};

}  // namespace

cudaError_t download(void* host, const void* dev, size_t bytes, cudaStream_t st) {
    if (bytes <= kDirect || !pageable(host) || in_place(static_cast<const char*>(host), bytes)) {
        const cudaError_t e = cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, st);
        return e != cudaSuccess ? e : cudaStreamSynchronize(st);
    }
    char* dst = static_cast<char*>(host);
    const char* src = static_cast<const char*>(dev);
    Toucher pages(dst, bytes);
    cudaError_t e = cudaSuccess;
    for (size_t o = 0; o < bytes && e == cudaSuccess; o += kChunk) {
        pages.wait(o / kChunk);
        e = cudaMemcpyAsync(dst + o, src + o, std::min(kChunk, bytes - o), cudaMemcpyDeviceToHost, st);
    }
    const cudaError_t s = cudaStreamSynchronize(st);
    return e != cudaSuccess ? e : s;
}

}  // namespace sb200
