// hostio.cu - host arrays in and out: large uploads from pageable memory, and
// row indices, which are 64-bit at the interface and 32-bit on the device.
#include <algorithm>
#include <new>
#include <thread>

#include "kernels.cuh"

namespace umapb {
namespace {

// ------------------------------------------------------- staged uploads
// A copy from pageable memory goes through the driver's own pinned buffer on
// one thread: 128 MB take 10.9 ms, 12 GB/s, on a link that carries over 50.
// Four threads that fill pinned buffers of 1 MB, two each, and queue a copy
// per buffer take 3.6 ms (two threads 5.5, six 3.8, eight 4.0; 512 KB buffers
// 5.0, 2 MB 3.3 at twice the pinned memory).  Below kStagedBytes the driver's
// copy is kept: 8 MB are level (0.43 ms to 0.45), 32 MB would gain 0.7 ms,
// and pinning the buffers for the first time costs 4 to 5 ms, about what one
// copy of kStagedBytes gains.
constexpr size_t kStagedBytes = static_cast<size_t>(64) << 20;
constexpr size_t kStageBuf = static_cast<size_t>(1) << 20;
constexpr int kStageThreads = 4;
constexpr int kStageBufs = 2;
// Pinned sets in use at once; a further upload takes the driver's copy.  One
// (8 MB) is kept when idle, also by calls that make no model, until
// umapb_destroy next leaves no model alive.
constexpr int kStageSets = 2;

struct StageSet {
    int device = 0;
    char* mem = nullptr;
    cudaEvent_t ev[kStageThreads * kStageBufs] = {};

    StageSet() {
        bool ok = cudaGetDevice(&device) == cudaSuccess &&
                  cudaHostAlloc(reinterpret_cast<void**>(&mem),
                                kStageBuf * kStageThreads * kStageBufs,
                                cudaHostAllocDefault) == cudaSuccess;
        for (auto& e : ev)
            ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
        if (!ok) {
            cudaGetLastError();  // the driver's copy serves instead
            clear();
        }
    }
    ~StageSet() { clear(); }
    void clear() {
        for (auto& e : ev) {
            if (e) cudaEventDestroy(e);
            e = nullptr;
        }
        if (mem) cudaFreeHost(mem);
        mem = nullptr;
    }
    StageSet(const StageSet&) = delete;
    StageSet& operator=(const StageSet&) = delete;
};

struct StagePool {
    std::mutex mu;
    StageSet* idle = nullptr;
    int in_use = 0;
    // never destroyed: the driver may be gone when static objects are
    static StagePool& get() {
        static StagePool* p = new StagePool;
        return *p;
    }
};

// A set for the current device, or none.
struct StageLease {
    StageSet* set = nullptr;
    StageLease() {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return;
        StagePool& p = StagePool::get();
        StageSet* other = nullptr;
        {
            std::lock_guard<std::mutex> lk(p.mu);
            if (p.in_use >= kStageSets) return;
            ++p.in_use;
            if (p.idle) (p.idle->device == dev ? set : other) = p.idle;
            p.idle = nullptr;
        }
        delete other;
        if (!set) set = new (std::nothrow) StageSet;
        if (set && !set->mem) {
            delete set;
            set = nullptr;
        }
        if (!set) {
            std::lock_guard<std::mutex> lk(p.mu);
            --p.in_use;
        }
    }
    ~StageLease() {
        if (!set) return;
        StagePool& p = StagePool::get();
        {
            std::lock_guard<std::mutex> lk(p.mu);
            --p.in_use;
            if (!p.idle) std::swap(p.idle, set);
        }
        delete set;
    }
    StageLease(const StageLease&) = delete;
    StageLease& operator=(const StageLease&) = delete;
};

bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

cudaError_t upload_staged(StageSet& set, char* dst, const char* src, size_t bytes, int threads,
                          cudaStream_t s) {
    std::atomic<size_t> next{0};
    std::atomic<int> error{cudaSuccess};
    auto work = [&](int t) {
        auto check = [&](cudaError_t e) {
            if (e != cudaSuccess) error.store(e);
            return e == cudaSuccess;
        };
        if (!check(cudaSetDevice(set.device))) return;
        bool used[kStageBufs] = {};
        for (int b = 0; error.load() == cudaSuccess; b = (b + 1) % kStageBufs) {
            const size_t at = next.fetch_add(1) * kStageBuf;
            if (at >= bytes) return;
            const size_t len = std::min(kStageBuf, bytes - at);
            char* buf = set.mem + (t * kStageBufs + b) * kStageBuf;
            cudaEvent_t ev = set.ev[t * kStageBufs + b];
            if (used[b] && !check(cudaEventSynchronize(ev))) return;
            std::memcpy(buf, src + at, len);
            if (!check(cudaMemcpyAsync(dst + at, buf, len, cudaMemcpyHostToDevice, s))) return;
            if (!check(cudaEventRecord(ev, s))) return;
            used[b] = true;
        }
    };
    run_threads(threads, work);
    // the buffers go back to the pool, so their copies must have been made
    const cudaError_t done = cudaStreamSynchronize(s);
    return error.load() != cudaSuccess ? static_cast<cudaError_t>(error.load()) : done;
}

// ------------------------------------------------------- 64-bit indices
// Widened or narrowed on the device, through the memory of the floats that go
// with them (one a index), so the host makes no pass over them and nothing is
// allocated.  With 1.8M indices out (60,013 rows, k = 30) the call takes 7.3 ms;
// through a host vector of 32-bit indices it took 9.1.  Up to kHostIndices the
// host vector is kept: two more copies and launches are as long.
constexpr int64_t kHostIndices = 1 << 14;

template <typename From, typename To>
__global__ void convert_kernel(const From* __restrict__ in, int64_t n, To* __restrict__ out) {
    const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i < n) out[i] = static_cast<To>(in[i]);
}

}  // namespace

int host_threads() {
    return static_cast<int>(
        std::min<unsigned>(kStageThreads, std::max(1u, std::thread::hardware_concurrency())));
}

void upload_host(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    if (bytes == 0) return;
    // an error of the call, as cudaMemcpyAsync makes it: staging would read it
    if (!src) throw_cuda(cudaErrorInvalidValue, "upload of a null host array", __FILE__, __LINE__);
    const int threads = host_threads();
    if (bytes >= kStagedBytes && threads > 1 && pageable(src)) {
        StageLease lease;
        if (lease.set) {
            UMAPB_CUDA(upload_staged(*lease.set, static_cast<char*>(dst),
                                     static_cast<const char*>(src), bytes, threads, s));
            return;
        }
    }
    UMAPB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
}

void trim_host_staging() {
    StagePool& p = StagePool::get();
    StageSet* set = nullptr;
    {
        std::lock_guard<std::mutex> lk(p.mu);
        std::swap(set, p.idle);
    }
    delete set;
}

void download_neighbors(int64_t* idx_out, float* dist_out, const int32_t* idx, float* dist,
                        int64_t n, cudaStream_t s) {
    if (!idx_out) throw_cuda(cudaErrorInvalidValue, "download to a null host array", __FILE__, __LINE__);
    UMAPB_CUDA(cudaMemcpyAsync(dist_out, dist, n * 4, cudaMemcpyDeviceToHost, s));
    if (n <= kHostIndices) {
        std::vector<int32_t> narrow(n);  // pageable: the copy has been made when the call returns
        UMAPB_CUDA(cudaMemcpyAsync(narrow.data(), idx, n * 4, cudaMemcpyDeviceToHost, s));
        std::copy(narrow.begin(), narrow.end(), idx_out);
        return;
    }
    int64_t* wide = reinterpret_cast<int64_t*>(dist);
    for (int64_t at = 0, len = n / 2; at < n; at += len) {
        len = std::min(len, n - at);
        convert_kernel<<<static_cast<unsigned>(ceil_div(len, 256)), 256, 0, s>>>(idx + at, len, wide);
        UMAPB_LAUNCH_CHECK();
        UMAPB_CUDA(cudaMemcpyAsync(idx_out + at, wide, len * 8, cudaMemcpyDeviceToHost, s));
    }
}

void upload_columns(int32_t* idx, float* values, const int64_t* idx_in, const float* values_in,
                    int64_t n, cudaStream_t s) {
    if (n <= kHostIndices) {
        std::vector<int32_t> narrow(idx_in, idx_in + n);
        if (n > 0)
            UMAPB_CUDA(cudaMemcpyAsync(idx, narrow.data(), n * 4, cudaMemcpyHostToDevice, s));
    } else {
        int64_t* wide = reinterpret_cast<int64_t*>(values);
        for (int64_t at = 0, len = n / 2; at < n; at += len) {
            len = std::min(len, n - at);
            upload_host(wide, idx_in + at, len * 8, s);
            convert_kernel<<<static_cast<unsigned>(ceil_div(len, 256)), 256, 0, s>>>(wide, len, idx + at);
            UMAPB_LAUNCH_CHECK();
        }
    }
    upload_host(values, values_in, n * 4, s);
}

}  // namespace umapb
