// Host-side runtime pieces shared by the translation units: launch wrapper (PDL + per-kernel event profile +
// launch counter), device buffer RAII, thread-local error slot.
#pragma once
#include <sys/mman.h>
#include <unistd.h>

#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"

namespace fl {

extern thread_local std::string g_last_error;
extern std::atomic<uint64_t> g_launches;

struct ProfEntry {
    std::string tag;
    uint64_t bytes;
    cudaEvent_t e0, e1;
};
struct Profiler {
    bool on = false;
    std::vector<ProfEntry> entries;
};
extern Profiler g_prof;

inline bool env_flag(const char* name) {
    const char* v = std::getenv(name);
    return v != nullptr && v[0] != '\0' && v[0] != '0';
}

struct LaunchCtx {
    cudaStream_t stream = nullptr;
    bool pdl = true;          // programmatic dependent launch on every kernel of the step
    bool capturing = false;   // inside cudaStreamBeginCapture: no events, no profile
    uint64_t captured = 0;    // kernels recorded into the graph being captured
    bool exact = false;       // layered models, exact mode: GEMMs accumulate in f64
};

// Launches `kern` with optional PDL.  `tag`/`bytes` feed the per-kernel profile (algorithmic bytes of that launch).
template <typename... KArgs, typename... Args>
inline void launch(LaunchCtx& lc, const char* tag, uint64_t bytes, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem,
                   Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = lc.stream;
    cudaLaunchAttribute attr[1];
    const bool prof = g_prof.on && !lc.capturing;
    if (lc.pdl && !prof) {
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
    ProfEntry pe;
    if (prof) {
        pe.tag = tag;
        pe.bytes = bytes;
        FL_CUDA(cudaEventCreate(&pe.e0));
        FL_CUDA(cudaEventCreate(&pe.e1));
        FL_CUDA(cudaEventRecord(pe.e0, lc.stream));
    }
    FL_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...));
    if (prof) {
        FL_CUDA(cudaEventRecord(pe.e1, lc.stream));
        g_prof.entries.push_back(pe);
    }
    if (lc.capturing)
        lc.captured++;
    else
        g_launches.fetch_add(1, std::memory_order_relaxed);
}

// a start / stop event pair that cannot leak when something between create and destroy throws
struct EventPair {
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    EventPair() {
        FL_CUDA(cudaEventCreate(&e0));
        if (cudaEventCreate(&e1) != cudaSuccess) {
            cudaEventDestroy(e0);
            throw Error(-2, "cudaEventCreate failed");
        }
    }
    EventPair(const EventPair&) = delete;
    EventPair& operator=(const EventPair&) = delete;
    ~EventPair() {
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
    }
};

template <typename T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    DevBuf(DevBuf&& o) noexcept : p(o.p), n(o.n) { o.p = nullptr; o.n = 0; }      // lets containers of buffers grow
    ~DevBuf() { release(); }
    void alloc(size_t count, bool zero = false) {
        release();
        if (count == 0) return;
        FL_CUDA(cudaMalloc(&p, count * sizeof(T)));
        if (zero) {                             // the streams of models and caches do not wait for the default one
            FL_CUDA(cudaMemset(p, 0, count * sizeof(T)));
            FL_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
        }
        n = count;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
};

// Memory of the process's own, page-locked.  cudaMallocHost hands out a shared mapping: a forked child would see in it what the device writes later
// (registered pages are copied at a fork like any others).  From 1 MB on huge pages, which are locked in 0.13 ms per MB; 4 KB pages and cudaMallocHost
// take 0.5 to 0.8.  Whole pages: no neighbour shares one.
inline void* lock_host(size_t bytes) {
    const size_t page = bytes >= (size_t)1 << 20 ? (size_t)2 << 20 : (size_t)sysconf(_SC_PAGESIZE);
    FL_CHECK(bytes <= SIZE_MAX - page, FL_ERR_INVALID, "bad size");
    const size_t size = (bytes + page - 1) / page * page;
    std::unique_ptr<void, decltype(&std::free)> p(std::aligned_alloc(page, size), &std::free);
    FL_CHECK(p != nullptr, FL_ERR_INVALID, "out of host memory");
    if (bytes >= (size_t)1 << 20) madvise(p.get(), size, MADV_HUGEPAGE);
    FL_CUDA(cudaHostRegister(p.get(), size, cudaHostRegisterDefault));
    return p.release();
}
inline void unlock_host(void* p) {
    FL_CUDA(cudaHostUnregister(p));
    std::free(p);
}

// Page-locked memory that copies alone reach, nobody outside sees and a large buffer may need: below 1 MB from cudaMallocHost, which cuts small pieces
// out of what it has locked already.
template <typename T>
struct HostBuf {
    T* p = nullptr;
    size_t n = 0;
    HostBuf() = default;
    HostBuf(const HostBuf&) = delete;
    HostBuf& operator=(const HostBuf&) = delete;
    ~HostBuf() { release(); }
    void alloc(size_t count) {
        release();
        own = count * sizeof(T) >= (size_t)1 << 20;
        if (own) p = static_cast<T*>(lock_host(count * sizeof(T)));
        else if (count) FL_CUDA(cudaMallocHost(&p, count * sizeof(T)));
        n = count;
    }
    void release() {
        if (p && !own) cudaFreeHost(p);
        if (p && own && cudaHostUnregister(p) == cudaSuccess) std::free(p);
        p = nullptr;
        n = 0;
    }

private:
    bool own = false;
};

template <typename T>
struct PinnedBuf {
    T* p = nullptr;
    size_t n = 0;
    PinnedBuf() = default;
    PinnedBuf(const PinnedBuf&) = delete;
    PinnedBuf& operator=(const PinnedBuf&) = delete;
    ~PinnedBuf() {
        if (p) cudaFreeHost(p);
    }
    void alloc(size_t count) {
        if (p) cudaFreeHost(p);
        p = nullptr;
        n = 0;
        if (count) FL_CUDA(cudaMallocHost(&p, count * sizeof(T)));
        n = count;
    }
};

}  // namespace fl
