// alloc.cu -- device memory behind dbuf.
//
// A build makes dozens of small allocations.  cudaMalloc takes 0.18 to 0.38 ms
// each and cudaFree as much again (4 KB as well as 16 MB, measured on a B200:
// 36 of the 48 ms of a build of 1M elements), a block of a memory pool that
// already holds its pages 2 us.  So blocks of up to kPoolBlock come from a pool
// of the library's own, one per device.  Larger ones stay with cudaMalloc,
// which maps a gigabyte in 0.4 ms where a pool that has to grow takes 6.5.
//
// The pool keeps at most kPoolKept bytes that nobody uses (CUDA gives back what
// is above that at the next synchronisation) and all of it is given back when an
// allocation fails.  Allocations and frees go through a stream of the library's;
// a block is handed out after that stream has been waited for and goes back
// after the device has been waited for, as cudaFree does, so it may be used on
// any stream and by any thread in between.
#include <mutex>

#include "common.cuh"

namespace abhsf {

namespace {

constexpr size_t kPoolBlock = size_t(32) << 20;
constexpr uint64_t kPoolKept = uint64_t(256) << 20;
constexpr int kMaxDevices = 64;

struct device_pool {
    bool tried = false;
    cudaMemPool_t pool = nullptr;
    cudaStream_t st = nullptr;
};

std::mutex g_pool_mutex;
device_pool g_pools[kMaxDevices];  // the pools live as long as the process

// The current device's pool (null where it has none).
device_pool pool_of(int dev)
{
    if (dev < 0 || dev >= kMaxDevices)
        return {};
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    device_pool& p = g_pools[dev];
    if (!p.tried) {
        p.tried = true;
        int supported = 0;
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        uint64_t kept = kPoolKept;
        cudaMemPool_t pool = nullptr;
        cudaStream_t st = nullptr;
        if (cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, dev) == cudaSuccess && supported &&
            cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess &&
            cudaMemPoolCreate(&pool, &props) == cudaSuccess &&
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &kept) == cudaSuccess) {
            p.pool = pool;
            p.st = st;
        } else {
            cudaGetLastError();  // no pool: cudaMalloc serves
        }
    }
    return p;
}

}  // namespace

void* device_alloc(size_t bytes, int& pool_dev)
{
    pool_dev = -1;
    int dev = 0;
    ABHSF_CUDA(cudaGetDevice(&dev));
    const device_pool p = pool_of(dev);
    void* ptr = nullptr;
    if (p.pool && bytes <= kPoolBlock) {
        if (cudaMallocFromPoolAsync(&ptr, bytes, p.pool, p.st) == cudaSuccess &&
            cudaStreamSynchronize(p.st) == cudaSuccess) {
            pool_dev = dev;
            return ptr;
        }
        cudaGetLastError();
    }
    cudaError_t e = cudaMalloc(&ptr, bytes);
    if (e == cudaErrorMemoryAllocation && p.pool) {
        cudaGetLastError();
        cudaMemPoolTrimTo(p.pool, 0);
        e = cudaMalloc(&ptr, bytes);
    }
    cuda_check(e, "cudaMalloc");
    return ptr;
}

void device_free(void* ptr, int pool_dev) noexcept
{
    if (pool_dev < 0) {
        cudaFree(ptr);
        return;
    }
    int dev = pool_dev;
    cudaGetDevice(&dev);
    if (dev != pool_dev)
        cudaSetDevice(pool_dev);
    cudaDeviceSynchronize();
    cudaFreeAsync(ptr, g_pools[pool_dev].st);
    if (dev != pool_dev)
        cudaSetDevice(dev);
}

}  // namespace abhsf
