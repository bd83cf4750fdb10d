// alloc.cu -- device memory behind dbuf.
//
// A build makes dozens of small allocations.  cudaMalloc takes 0.18 to 0.38 ms
// each and cudaFree as much again (4 KB as well as 16 MB, measured on a B200:
// 36 of the 48 ms of a build of 1M elements), a block of a memory pool that
// already holds its pages 2 us.  So blocks of up to kPoolBlock come from a pool
// of the library's own, one per device.  Larger ones stay with cudaMalloc,
// which maps a gigabyte in 0.4 ms where a pool that has to grow takes 6.5.
//
// The pool keeps at most kPoolKept bytes that nobody uses: its release threshold
// (CUDA gives back what the pool holds above it at the next synchronisation) is
// moved along with the bytes in use.  All that is unused is given back when an
// allocation fails.  Allocations and frees go through a stream of the library's;
// a block is handed out after that stream has been waited for and goes back
// after the device has been waited for, as cudaFree does, so it may be used on
// any stream and by any thread in between.
#include <mutex>

#include "common.cuh"

namespace abhsf {

namespace {

constexpr size_t kPoolBlock = size_t(1) << 30;
constexpr uint64_t kPoolKept = uint64_t(2) << 30;
constexpr int kMaxDevices = 64;

struct device_pool {
    bool tried = false;
    cudaMemPool_t pool = nullptr;
    cudaStream_t st = nullptr;
    uint64_t used = 0;  // bytes of the blocks in use
};

std::mutex g_pool_mutex;
device_pool g_pools[kMaxDevices];  // the pools live as long as the process

// `more` bytes come into use (or go out of it).
void use_bytes(device_pool& p, int64_t more)
{
    p.used += (uint64_t)more;
    uint64_t threshold = p.used + kPoolKept;
    cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &threshold);
}

// The current device's pool (null where it has none).  Under g_pool_mutex.
device_pool& pool_of(int dev)
{
    device_pool& p = g_pools[dev];
    if (!p.tried) {
        p.tried = true;
        int supported = 0;
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        cudaStream_t st = nullptr;
        if (cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, dev) == cudaSuccess && supported &&
            cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess &&
            cudaMemPoolCreate(&pool, &props) == cudaSuccess) {
            p.pool = pool;
            p.st = st;
            use_bytes(p, 0);
        } else {
            cudaGetLastError();  // no pool: cudaMalloc serves
        }
    }
    return p;
}

}  // namespace

void* device_alloc(size_t bytes, device_block& block)
{
    block = {};
    int dev = 0;
    ABHSF_CUDA(cudaGetDevice(&dev));
    void* ptr = nullptr;
    std::lock_guard<std::mutex> lock(g_pool_mutex);
    device_pool none;
    device_pool& p = dev >= 0 && dev < kMaxDevices ? pool_of(dev) : none;
    if (p.pool && bytes <= kPoolBlock) {
        use_bytes(p, (int64_t)bytes);
        if (cudaMallocFromPoolAsync(&ptr, bytes, p.pool, p.st) == cudaSuccess &&
            cudaStreamSynchronize(p.st) == cudaSuccess) {
            block.dev = dev;
            block.bytes = bytes;
            return ptr;
        }
        use_bytes(p, -(int64_t)bytes);
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

void device_free(void* ptr, const device_block& block) noexcept
{
    if (block.dev < 0) {
        cudaFree(ptr);
        return;
    }
    int dev = block.dev;
    cudaGetDevice(&dev);
    if (dev != block.dev)
        cudaSetDevice(block.dev);
    cudaDeviceSynchronize();
    {
        std::lock_guard<std::mutex> lock(g_pool_mutex);
        device_pool& p = g_pools[block.dev];
        cudaFreeAsync(ptr, p.st);
        use_bytes(p, -(int64_t)block.bytes);
    }
    if (dev != block.dev)
        cudaSetDevice(dev);
}

}  // namespace abhsf
