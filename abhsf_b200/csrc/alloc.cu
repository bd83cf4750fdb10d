// alloc.cu -- device memory behind dbuf and scratch.
//
// A build makes 70 to 100 allocations.  A cudaMalloc with its cudaFree takes 0.6
// to 0.8 ms (16 MB and 256 MB alike, measured on a B200: 36 of the 48 ms of a
// build of 1M elements), a block of a memory pool that already holds its pages 2
// us.  So blocks of up to kPoolBlock come from a pool of the library's own, one
// per device.
//
// The pool keeps at most kPoolKept bytes that nobody uses: its release threshold
// (CUDA gives back what the pool holds above it at the next synchronisation) is
// moved along with the bytes in use.  The driver takes unused memory out of the
// pool where another allocation of the process finds no other (a torch.empty of
// 256 MB more than what is free, 1.7 GB unused here: it succeeds).  What it does
// not take is given back when an allocation of the library fails, and all of it
// when the caller asks (abhsf_trim_device_memory): other processes cannot have it
// otherwise.
//
// Both limits from a build with one product of 60M elements, which needs 2 GB of
// scratch (ms, in a new process and then again and again, B200):
//   blocks to  kept      first         later
//   (none)     0         64 to 1,016   43 to 72, up to 1,114 (a large cudaFree waits)
//   32 MB      256 MB    45 to 73      18 to 55, up to 129
//   256 MB     2 GB      49 to 98      18 to 39, up to 869
//   1 GB       256 MB    66 to 67      38 to 44 (the pool grows by 6.4 ms a GB and
//   1 GB       1 GB      58 to 247     26 to 50     gives back at the same rate)
//   1 GB       2 GB      48 to 50      12.2 to 12.8
// A build of 1M elements takes 2.6 ms with any of them, 47 to 60 without a pool.
//
// Nobody's work may still be using a block that is handed out again:
//
// * The scratch of a call is used on the call's stream alone.  It is allocated
//   and freed in that stream's order, so nothing has to be waited for.
// * A handle's blocks may be used on any stream, by kernels queued by any thread
//   and by graphs the library knows nothing of.  They are allocated on a stream of
//   the library's, which is waited for, and freed blocks are set aside until all
//   work of the device has been waited for once (settle_released, when the handle
//   goes).  That wait is the one inside cudaFree, of a small block made for it: a
//   cudaDeviceSynchronize fails while any stream of the device is being captured,
//   in whatever mode and by whatever thread, and the capture is lost (a CG solve
//   captures its iterations), where cudaFree is allowed while another thread
//   captures in thread-local or relaxed mode.  Where the wait fails (a capture in
//   global mode) the blocks stay aside until one succeeds.
#include <mutex>
#include <vector>

#include "abhsf/abhsf_test.h"
#include "common.cuh"

namespace abhsf {

namespace {

constexpr size_t kPoolBlock = size_t(1) << 30;
constexpr uint64_t kPoolKept = uint64_t(2) << 30;
constexpr int kMaxDevices = 64;

struct released_block {
    void* ptr;
    size_t bytes;
};

struct device_pool {
    bool tried = false;
    cudaMemPool_t pool = nullptr;
    cudaStream_t st = nullptr;
    uint64_t used = 0;                   // bytes of the blocks in use
    std::vector<released_block> aside;  // released, the device not waited for yet
    void* anchor = nullptr;              // see device_waited_for
};

// The pools live as long as the process (handles may be released after the
// static destructors have run).
struct pools {
    std::mutex mutex;
    device_pool of[kMaxDevices];
};
pools& all()
{
    static pools* p = new pools;
    return *p;
}

// Makes dev current for a scope.
class on_device {
  public:
    explicit on_device(int dev) : dev_(dev)
    {
        cudaGetDevice(&before_);
        if (before_ != dev_)
            cudaSetDevice(dev_);
    }
    ~on_device()
    {
        if (before_ != dev_)
            cudaSetDevice(before_);
    }
    on_device(const on_device&) = delete;
    on_device& operator=(const on_device&) = delete;

  private:
    int dev_, before_ = 0;
};

// `more` bytes come into use (or go out of it).  Under the mutex.
void use_bytes(device_pool& p, int64_t more)
{
    p.used += (uint64_t)more;
    uint64_t threshold = p.used + kPoolKept;
    cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &threshold);
}

// The current device's pool (null where it has none).
device_pool* pool_of(int dev)
{
    if (dev < 0 || dev >= kMaxDevices)
        return nullptr;
    std::lock_guard<std::mutex> lock(all().mutex);
    device_pool& p = all().of[dev];
    if (!p.tried) {
        p.tried = true;
        int supported = 0;
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        cudaStream_t st = nullptr;
        // an allocation never waits for another stream's work: what is not free yet is not taken
        int wait = 0;
        if (cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, dev) == cudaSuccess && supported &&
            cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) == cudaSuccess &&
            cudaMemPoolCreate(&pool, &props) == cudaSuccess &&
            cudaMemPoolSetAttribute(pool, cudaMemPoolReuseAllowInternalDependencies, &wait) == cudaSuccess) {
            p.pool = pool;
            p.st = st;
            use_bytes(p, 0);
        } else {
            cudaGetLastError();  // no pool: cudaMalloc serves
        }
    }
    return p.pool ? &p : nullptr;
}

// Waits for all work queued on the current device; false where that is not
// allowed now.  (The anchor keeps the allocator's chunk for small blocks open: a
// cudaMalloc and cudaFree inside it take 1.3 and 3 us, 600 us where they make and
// drop the chunk.)
bool device_waited_for(device_pool& p)
{
    void* fence = nullptr;
    bool ok = cudaMalloc(&fence, 256) == cudaSuccess;
    if (ok) {
        std::lock_guard<std::mutex> lock(all().mutex);
        if (!p.anchor)
            std::swap(p.anchor, fence);
    }
    if (ok && !fence)
        ok = cudaMalloc(&fence, 256) == cudaSuccess;
    ok = ok && cudaFree(fence) == cudaSuccess;
    if (!ok)
        cudaGetLastError();
    return ok;
}

void settle(int dev) noexcept
{
    device_pool& p = all().of[dev];
    std::vector<released_block> mine;
    {
        std::lock_guard<std::mutex> lock(all().mutex);
        mine.swap(p.aside);
    }
    if (mine.empty())
        return;
    const on_device guard(dev);
    const bool ok = device_waited_for(p);
    {
        std::lock_guard<std::mutex> lock(all().mutex);
        for (const released_block& b : mine) {
            if (ok && cudaFreeAsync(b.ptr, p.st) == cudaSuccess) {
                use_bytes(p, -(int64_t)b.bytes);
                continue;
            }
            cudaGetLastError();
            try {
                p.aside.push_back(b);
            } catch (...) {  // no host memory: the block is lost
            }
        }
    }
    if (ok && cudaStreamSynchronize(p.st) != cudaSuccess)  // free for every stream from here on
        cudaGetLastError();
}

// Everything the pool holds that nobody uses goes back to the device.
void trim(device_pool& p, int dev)
{
    settle(dev);
    const on_device guard(dev);
    device_waited_for(p);  // scratch freed behind work that still runs
    cudaMemPoolTrimTo(p.pool, 0);
    cudaGetLastError();
}

}  // namespace

void* device_alloc(size_t bytes, device_block& block)
{
    int dev = 0;
    ABHSF_CUDA(cudaGetDevice(&dev));
    void* ptr = nullptr;
    device_pool* p = pool_of(dev);
    if (p && bytes <= kPoolBlock) {
        const cudaStream_t st = block.scratch ? block.st : p->st;
        {
            std::lock_guard<std::mutex> lock(all().mutex);
            use_bytes(*p, (int64_t)bytes);  // first: the wait below must not give back what is about to be used
        }
        bool ok = cudaMallocFromPoolAsync(&ptr, bytes, p->pool, st) == cudaSuccess;
        if (ok && !block.scratch && cudaStreamSynchronize(st) != cudaSuccess) {
            cudaFreeAsync(ptr, st);
            ok = false;
        }
        if (ok) {
            block.dev = dev;
            block.bytes = bytes;
            return ptr;
        }
        cudaGetLastError();
        std::lock_guard<std::mutex> lock(all().mutex);
        use_bytes(*p, -(int64_t)bytes);
    }
    block.dev = -1;
    cudaError_t e = cudaMalloc(&ptr, bytes);
    if (e == cudaErrorMemoryAllocation && p) {
        cudaGetLastError();
        trim(*p, dev);
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
    device_pool& p = all().of[block.dev];
    if (block.scratch) {
        const on_device guard(block.dev);
        const bool ok = cudaFreeAsync(ptr, block.st) == cudaSuccess;
        if (!ok)
            cudaGetLastError();
        std::lock_guard<std::mutex> lock(all().mutex);
        if (ok) {
            use_bytes(p, -(int64_t)block.bytes);
            return;
        }
    }
    std::lock_guard<std::mutex> lock(all().mutex);
    try {
        p.aside.push_back({ptr, block.bytes});
    } catch (...) {  // no host memory: the block is lost
    }
}

void settle_released() noexcept
{
    for (int dev = 0; dev < kMaxDevices; ++dev) {
        bool any = false;
        {
            std::lock_guard<std::mutex> lock(all().mutex);
            any = !all().of[dev].aside.empty();
        }
        if (any)
            settle(dev);
    }
}

}  // namespace abhsf

extern "C" abhsf_status abhsf_trim_device_memory(int64_t* bytes)
{
    using namespace abhsf;
    return guarded([&] {
        uint64_t back = 0;
        for (int dev = 0; dev < kMaxDevices; ++dev) {
            device_pool& p = all().of[dev];
            {
                std::lock_guard<std::mutex> lock(all().mutex);
                if (!p.pool)
                    continue;
            }
            uint64_t before = 0, after = 0;
            ABHSF_CUDA(cudaMemPoolGetAttribute(p.pool, cudaMemPoolAttrReservedMemCurrent, &before));
            trim(p, dev);
            ABHSF_CUDA(cudaMemPoolGetAttribute(p.pool, cudaMemPoolAttrReservedMemCurrent, &after));
            back += before > after ? before - after : 0;
        }
        if (bytes)
            *bytes = (int64_t)back;
    });
}

extern "C" int64_t abhsf_test_blocks_set_aside(void)
{
    using namespace abhsf;
    std::lock_guard<std::mutex> lock(all().mutex);
    int64_t n = 0;
    for (const device_pool& p : all().of)
        n += (int64_t)p.aside.size();
    return n;
}
