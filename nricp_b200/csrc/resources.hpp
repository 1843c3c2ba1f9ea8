// What calls would otherwise create and destroy every time: streams, device
// memory and small page-locked blocks.  Each kind is kept up to a bound, per
// device where it belongs to one, behind a mutex, and handed back when its
// lease ends (never freed at process exit, after the CUDA runtime has shut
// down).  A lease belongs to one call or object, so calls on several threads
// never share one.  (cudaMalloc, cudaFree, stream creation and page-locking
// took 0.7 of the 0.8 ms of a 5,000-pair rigid fit, and 5 to 13 ms of a
// six-wrap solve_batch.)
#pragma once

#include <cstddef>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

namespace nricp_b200 {

void check(cudaError_t status, const char* what);  // throws CudaError (session.cu)

// Device memory: a stream-ordered pool per device that keeps up to 8 GB
// between calls, so that repeated calls allocate and free without waiting for
// the device; release_pools gives back what no call holds.
struct DevicePools {
    std::mutex mu;
    std::map<int, cudaMemPool_t> of_device;
    static DevicePools& all() {
        static DevicePools& pools = *new DevicePools;
        return pools;
    }
};
inline cudaMemPool_t batch_pool(int device) {
    DevicePools& pools = DevicePools::all();
    std::lock_guard<std::mutex> lk(pools.mu);
    auto it = pools.of_device.find(device);
    if (it != pools.of_device.end()) return it->second;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool = nullptr;
    check(cudaMemPoolCreate(&pool, &props), "cudaMemPoolCreate");
    uint64_t keep = 8ull << 30;
    check(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep), "pool");
    pools.of_device[device] = pool;
    return pool;
}

// Waits for each device that has a pool, so that every free has taken place.
inline void release_pools() {
    DevicePools& pools = DevicePools::all();
    std::lock_guard<std::mutex> lk(pools.mu);
    int current = 0;
    if (!pools.of_device.empty()) check(cudaGetDevice(&current), "device");
    for (const auto& [device, pool] : pools.of_device) {
        check(cudaSetDevice(device), "cudaSetDevice");
        const cudaError_t done = cudaDeviceSynchronize();
        const cudaError_t trimmed = cudaMemPoolTrimTo(pool, 0);
        check(cudaSetDevice(current), "cudaSetDevice");
        check(done, "release memory");
        check(trimmed, "release memory");
    }
}

inline cudaMemPool_t current_pool() {
    int device = 0;
    check(cudaGetDevice(&device), "device");
    return batch_pool(device);
}

// Pool memory freed in the stream's order when it goes out of scope.
class PoolBuffer {
public:
    PoolBuffer(size_t bytes, cudaStream_t stream, const char* what) : stream_(stream) {
        check(cudaMallocFromPoolAsync(&base_, bytes > 0 ? bytes : 1, current_pool(), stream), what);
    }
    PoolBuffer(const PoolBuffer&) = delete;
    PoolBuffer& operator=(const PoolBuffer&) = delete;
    ~PoolBuffer() { cudaFreeAsync(base_, stream_); }
    char* data() const { return static_cast<char*>(base_); }

private:
    void* base_ = nullptr;
    cudaStream_t stream_;
};

// A non-blocking stream of the current device; at most 32 idle ones are kept
// per device.  Work still queued when a lease ends only delays the next one's.
class StreamLease {
public:
    StreamLease() = default;
    StreamLease(StreamLease&& o) noexcept : stream_(o.stream_), device_(o.device_) { o.stream_ = nullptr; }
    StreamLease& operator=(StreamLease&& o) noexcept {
        std::swap(stream_, o.stream_);
        std::swap(device_, o.device_);
        return *this;
    }
    ~StreamLease() {
        if (!stream_) return;
        {
            std::lock_guard<std::mutex> lk(mutex());
            auto& kept = idle()[device_];
            if (kept.size() < 32) {
                kept.push_back(stream_);
                return;
            }
        }
        cudaStreamDestroy(stream_);
    }
    static StreamLease take() {
        StreamLease s;
        check(cudaGetDevice(&s.device_), "device");
        {
            std::lock_guard<std::mutex> lk(mutex());
            auto& kept = idle()[s.device_];
            if (!kept.empty()) {
                s.stream_ = kept.back();
                kept.pop_back();
                return s;
            }
        }
        check(cudaStreamCreateWithFlags(&s.stream_, cudaStreamNonBlocking), "cudaStreamCreate");
        return s;
    }
    operator cudaStream_t() const { return stream_; }

private:
    static std::mutex& mutex() {
        static std::mutex& m = *new std::mutex;
        return m;
    }
    static std::map<int, std::vector<cudaStream_t>>& idle() {
        static auto& kept = *new std::map<int, std::vector<cudaStream_t>>;
        return kept;
    }
    cudaStream_t stream_ = nullptr;
    int device_ = 0;
};

// A small page-locked block; at most 32 idle ones of 64 KB are kept, larger
// blocks are not.
class PinnedLease {
public:
    PinnedLease() = default;
    explicit PinnedLease(size_t bytes) {
        kept_size_ = bytes <= kBlock;
        if (kept_size_) {
            std::lock_guard<std::mutex> lk(mutex());
            if (!idle().empty()) {
                base_ = idle().back();
                idle().pop_back();
                return;
            }
        }
        check(cudaHostAlloc(&base_, kept_size_ ? kBlock : bytes, cudaHostAllocPortable), "cudaHostAlloc");
    }
    PinnedLease(PinnedLease&& o) noexcept : base_(o.base_), kept_size_(o.kept_size_) { o.base_ = nullptr; }
    PinnedLease& operator=(PinnedLease&& o) noexcept {
        std::swap(base_, o.base_);
        std::swap(kept_size_, o.kept_size_);
        return *this;
    }
    ~PinnedLease() {
        if (!base_) return;
        if (kept_size_) {
            std::lock_guard<std::mutex> lk(mutex());
            if (idle().size() < 32) {
                idle().push_back(base_);
                return;
            }
        }
        cudaFreeHost(base_);
    }
    void* data() const { return base_; }

private:
    static constexpr size_t kBlock = 64 * 1024;
    static std::mutex& mutex() {
        static std::mutex& m = *new std::mutex;
        return m;
    }
    static std::vector<void*>& idle() {
        static auto& kept = *new std::vector<void*>;
        return kept;
    }
    void* base_ = nullptr;
    bool kept_size_ = false;
};

}  // namespace nricp_b200
