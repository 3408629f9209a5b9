// capi.cu -- library-wide C entry points: error strings, launch accounting, version.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <stdio.h>
#include <thread>
#include <vector>

#include "hype_common.cuh"

namespace hype {
static thread_local char g_last_error[512] = "";
static std::atomic<long long> g_launches{0};

void set_last_error(const char* where, cudaError_t e) {
    snprintf(g_last_error, sizeof(g_last_error), "%s: %s (%s)", where, cudaGetErrorName(e), cudaGetErrorString(e));
}

// A state that a program downloads goes to memory it has just allocated, none of it present.  The copy then takes
// its page faults one by one (128 MB: 3.9 ms beside a 0.8 ms transfer).  Here up to 4 threads (1.6 ms; 8 take 3.0)
// make the pages present, and do so while the GPU still runs what the stream holds.  Nothing is kept; memory
// that is present already (a buffer in use, pinned memory) and small copies are left alone, and where the kernel
// does not know the request the copy faults the pages in as before.
static void make_present(void* p, size_t bytes) {
    constexpr size_t kLeast = 8u << 20, kPart = 2u << 20;
    if (bytes < kLeast) return;
#ifdef MADV_POPULATE_WRITE
    const size_t page = (size_t)sysconf(_SC_PAGESIZE);
    const size_t lo = ((size_t)p + page - 1) / page * page, hi = ((size_t)p + bytes) / page * page;
    int present = 0;
    for (size_t at : {lo, lo + (hi - lo) / 2 / page * page, hi - page}) {
        unsigned char v = 0;
        present += mincore((void*)at, page, &v) == 0 && (v & 1);
    }
    if (present == 3) return;
    const size_t n = std::max<size_t>(1, std::min<size_t>(4, std::thread::hardware_concurrency() / 2));
    const size_t part = ((hi - lo) / n / kPart + 1) * kPart;
    auto populate = [=](size_t a) { madvise((void*)a, std::min(part, hi - a), MADV_POPULATE_WRITE); };
    std::vector<std::thread> team;
    size_t a = lo;
    try {
        for (; a + part < hi; a += part) team.emplace_back(populate, a);
    } catch (...) {  // no more threads: the rest here
    }
    for (; a < hi; a += part) populate(a);
    for (auto& t : team) t.join();
#endif
}

cudaError_t copy_to_host(void* dst, const void* src, size_t bytes, cudaStream_t stream) {
    make_present(dst, bytes);
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, stream);
}

void count_launch(long long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
}  // namespace hype

extern "C" const char* hype_strerror(int code) {
    switch (code) {
        case HYPE_OK: return "ok";
        case HYPE_ERR_ARG: return "invalid argument";
        case HYPE_ERR_STATE: return "inadmissible state (density or pressure below floor)";
        case HYPE_ERR_CUDA: return "CUDA error";
        case HYPE_ERR_NOMEM: return "device allocation failed";
        case HYPE_ERR_UNSUPPORTED: return "unsupported option";
        default: return "unknown status";
    }
}
extern "C" const char* hype_last_error(void) { return hype::g_last_error; }
extern "C" long long hype_launch_count(void) { return hype::g_launches.load(); }
extern "C" const char* hype_version(void) { return "hype-gb300 0.1 (sm_103a)"; }

extern "C" int hype_set_device(int device) {
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) {
        hype::set_last_error("cudaSetDevice", e);
        return HYPE_ERR_CUDA;
    }
    return HYPE_OK;
}

extern "C" int hype_device_count(int* n) {
    if (!n) return HYPE_ERR_ARG;
    cudaError_t e = cudaGetDeviceCount(n);
    if (e != cudaSuccess) {
        *n = 0;
        hype::set_last_error("cudaGetDeviceCount", e);
        return HYPE_ERR_CUDA;
    }
    return HYPE_OK;
}
