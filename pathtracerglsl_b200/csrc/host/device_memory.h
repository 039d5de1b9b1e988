// device_memory.h — device memory of a context's objects.
#pragma once
#include <cuda_runtime.h>
#include <map>
#include <mutex>
#include <set>

namespace ptx_host {

// A scene, program or build takes a few dozen blocks, and cudaMalloc / cudaFree cost 0.1 to
// several ms each (38 of each made 18 of the 25 ms of uploading a 327,680-triangle scene).  So the
// contexts on one device share a stream-ordered pool: allocating and freeing is then a few
// microseconds while it holds enough.  It keeps at most kPoolKeep bytes that no object uses and
// goes with the device's last context.  Blocks above kPoolMax come from cudaMalloc: the pool maps
// memory in small pieces, and the 8.7 GB path pool of a 2^25-path wave took 80 ms from it against
// 5.  So does every block of a device that makes no pool.  A block freed on one stream goes to
// another only once it is idle: streams of the pool never wait for one another.
constexpr unsigned long long kPoolKeep = 512ull << 20;
constexpr size_t kPoolMax = 256ull << 20;

class DevicePools {
public:
    // The device's pool, or null where it makes none.  Each acquire is released once.
    cudaMemPool_t acquire(int device) {
        std::lock_guard<std::mutex> lock(mutex_);
        Pool& d = pools_[device];
        if (d.users++ == 0) d.pool = create(device);
        return d.pool;
    }
    // The stream that uploads of an acquired device's contexts share (one of a context's own
    // cost 50 to 300 us to create); null if it cannot be made.
    cudaStream_t upload_stream(int device) {
        std::lock_guard<std::mutex> lock(mutex_);
        Pool& d = pools_[device];
        if (!d.upload && cudaStreamCreateWithFlags(&d.upload, cudaStreamNonBlocking) != cudaSuccess) {
            cudaGetLastError();
            d.upload = nullptr;
        }
        return d.upload;
    }
    void release(int device) {
        std::lock_guard<std::mutex> lock(mutex_);
        const auto it = pools_.find(device);
        if (--it->second.users > 0) return;
        if (it->second.upload) cudaStreamDestroy(it->second.upload);
        if (it->second.pool) cudaMemPoolDestroy(it->second.pool);
        pools_.erase(it);
    }
    static DevicePools& all() {
        static DevicePools* pools = new DevicePools;   // outlives contexts that are destroyed at exit
        return *pools;
    }

private:
    struct Pool { cudaMemPool_t pool = nullptr; cudaStream_t upload = nullptr; int users = 0; };
    static cudaMemPool_t create(int device) {
        int supported = 0;
        if (cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, device) != cudaSuccess || !supported) {
            cudaGetLastError();
            return nullptr;
        }
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = device;
        unsigned long long keep = kPoolKeep;
        int wait = 0;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
            cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &wait) != cudaSuccess) {
            cudaGetLastError();
            cudaMemPoolDestroy(pool);
            return nullptr;
        }
        return pool;
    }
    std::mutex mutex_;
    std::map<int, Pool> pools_;
};

// Allocations of one of a context's streams, ordered on it: every use is, or follows a wait for it.
class DeviceMemory {
public:
    void open(int device, cudaStream_t stream) {
        device_ = device;
        stream_ = stream;
        pool_ = DevicePools::all().acquire(device);
    }
    void close() { DevicePools::all().release(device_); }
    cudaError_t alloc(void** out, size_t bytes) {
        const bool pooled = pool_ && bytes <= kPoolMax;
        cudaError_t e = take(out, bytes, pooled);
        if (e == cudaErrorMemoryAllocation && pool_) {   // what the pool keeps idle may be what is missing
            cudaDeviceSynchronize();   // frees on every stream
            cudaMemPoolTrimTo(pool_, 0);
            e = take(out, bytes, pooled);
        }
        if (e == cudaSuccess && !pooled) direct_.insert(*out);
        return e;
    }
    void free(void* p) {
        if (!p) return;
        if (direct_.erase(p)) cudaFree(p);
        else cudaFreeAsync(p, stream_);
    }

private:
    cudaError_t take(void** out, size_t bytes, bool pooled) {
        void* p = nullptr;
        const cudaError_t e = pooled ? cudaMallocFromPoolAsync(&p, bytes, pool_, stream_) : cudaMalloc(&p, bytes);
        if (e != cudaSuccess) cudaGetLastError();
        *out = e == cudaSuccess ? p : nullptr;
        return e;
    }
    int device_ = 0;
    cudaStream_t stream_ = nullptr;
    cudaMemPool_t pool_ = nullptr;
    std::set<void*> direct_;   // from cudaMalloc
};

}  // namespace ptx_host
