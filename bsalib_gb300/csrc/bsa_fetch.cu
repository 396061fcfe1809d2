// bsa_fetch.cu -- large results to the caller's (pageable) memory.
//
// A device-to-host copy into fresh pageable memory faults its pages in one by one behind the copy:
// 31 MB of listed bispectra took 26 ms, 15 MB of a materialised grid 12 ms, against 0.2 ms over the
// link.  Here the link fills a pinned block and several host threads copy it on, so the page faults
// and the copy run on many cores.  Memory whose pages are there already takes the plain copy (3 MB in
// about 0.1 ms, which starting the threads alone costs).
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "bsa_engine.cuh"

namespace bsa {
namespace {

constexpr size_t kDirect = 1 << 20;    // smaller results: one plain copy
constexpr size_t kThreads = 8;
constexpr size_t kBlockMax = 64 << 20; // pinned block, at most

// One pinned block for the process, grown on demand to kBlockMax; bsa_gpu_releaseDeviceCache frees it.
struct Pinned {
    std::mutex m;
    void *p = nullptr;
    size_t bytes = 0;
};
Pinned &pinned() {
    static Pinned b;
    return b;
}

// Whether sixteen pages spread over the range are in memory.
bool resident(const void *p, size_t n) {
    static const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    for (int k = 0; k < 16; ++k) {
        const uintptr_t a = ((uintptr_t)p + (n - 1) / 15 * k) & ~(page - 1);
        unsigned char v = 0;
        if (mincore((void *)a, page, &v) != 0 || !(v & 1)) return false;
    }
    return true;
}

void copy_threads(char *dst, const char *src, size_t n) {
    const size_t nt = std::max<size_t>(1, std::min<size_t>({kThreads, n >> 20, std::thread::hardware_concurrency()}));
    const size_t step = ((n + nt - 1) / nt + 4095) & ~(size_t)4095;
    std::vector<std::thread> ts;
    size_t o = step;
    try {
        for (; o < n; o += step)
            ts.emplace_back([=] { std::memcpy(dst + o, src + o, std::min(step, n - o)); });
    } catch (...) {  // no more threads: the rest here
        std::memcpy(dst + o, src + o, n - o);
    }
    std::memcpy(dst, src, std::min(step, n));
    for (std::thread &t : ts) t.join();
}

}  // namespace

// dst = n bytes at src (device) as they are after the work queued on st; waits for it.
cudaError_t fetch(cudaStream_t st, void *dst, const void *src, size_t n) {
    cudaError_t e;
    Pinned &b = pinned();
    std::unique_lock<std::mutex> lk(b.m, std::defer_lock);
    const bool direct = n < kDirect || resident(dst, n);
    if (!direct) lk.lock();
    if (!direct && b.bytes < std::min(n, kBlockMax)) {
        if (b.p) cudaFreeHost(b.p);
        b.p = nullptr;
        b.bytes = 0;
        const size_t want = std::min((n + kDirect - 1) / kDirect * kDirect, kBlockMax);
        if (cudaHostAlloc(&b.p, want, cudaHostAllocDefault) == cudaSuccess) b.bytes = want;
        else {
            b.p = nullptr;
            cudaGetLastError();  // no pinned memory: plain copy
        }
    }
    if (direct || !b.p) {
        if ((e = cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, st))) return e;
        return cudaStreamSynchronize(st);
    }
    for (size_t o = 0; o < n; o += b.bytes) {
        const size_t c = std::min(b.bytes, n - o);
        if ((e = cudaMemcpyAsync(b.p, (const char *)src + o, c, cudaMemcpyDeviceToHost, st)) ||
            (e = cudaStreamSynchronize(st)))
            return e;
        copy_threads((char *)dst + o, (const char *)b.p, c);
    }
    return cudaSuccess;
}

void release_fetch_block() {
    Pinned &b = pinned();
    std::lock_guard<std::mutex> lk(b.m);
    if (b.p) cudaFreeHost(b.p);
    b.p = nullptr;
    b.bytes = 0;
}

}  // namespace bsa
