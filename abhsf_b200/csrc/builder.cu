// builder.cu -- GPU construction of the ABHSF format and GPU block histograms.
//
// The reference builds nothing on a device: it partitions elements into
// blocks by sorting on the block key (block_statistics/block_stats.cpp:69-100,
// preprocessing/test.cpp:237-368) and evaluates the per-block cost model
// (include/abhsf/msmf.h:9-63).  Here the same partition is one radix sort of a
// 64-bit key on the device (CUB), and every other step -- key build, tile
// segmentation, per-tile scheme, offsets, payload scatter -- is a kernel of
// this file.  Results are deterministic: the only atomics are integer ORs /
// adds whose result does not depend on their order.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_select.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "internal.cuh"

namespace abhsf {
namespace {

constexpr int kThreads = 256;

inline unsigned grid_for(int64_t n)
{
    int64_t b = (n + kThreads - 1) / kThreads;
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>(b, 148 * 32));
}

#define GRID_STRIDE(i, n) for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (n); i += (int64_t)gridDim.x * blockDim.x)

enum : int { kErrRange = 1, kErrDuplicate = 2, kErrCsrTooLong = 4, kErrHistOverflow = 8, kUnordered = 16 };

// key = ((I * N + J) << 2 lg) | (lrow << lg) | lcol: tiles in (block row,
// block column) order, elements of a tile in row-major order; and the
// element's place in the input.  kUnordered: the input is not in row-major
// order.
__global__ void k_make_keys(const int64_t* __restrict__ rows, const int64_t* __restrict__ cols, int64_t nnz, int64_t m,
                            int64_t n, int lg, uint64_t N, uint64_t* __restrict__ keys, uint32_t* __restrict__ place,
                            int* __restrict__ err)
{
    const uint64_t lmask = (uint64_t(1) << lg) - 1;
    int e = 0;
    GRID_STRIDE(i, nnz)
    {
        const int64_t r = rows[i], c = cols[i];
        if (i > 0) {
            const int64_t pr = rows[i - 1];
            if (pr > r || (pr == r && cols[i - 1] > c))
                e |= kUnordered;
        }
        place[i] = (uint32_t)i;
        if (r < 0 || r >= m || c < 0 || c >= n) {
            e |= kErrRange;
            keys[i] = 0;
            continue;
        }
        const uint64_t I = uint64_t(r) >> lg, J = uint64_t(c) >> lg;
        keys[i] = ((I * N + J) << (2 * lg)) | ((uint64_t(r) & lmask) << lg) | (uint64_t(c) & lmask);
    }
    e = __reduce_or_sync(0xffffffffu, e);
    // (one lane, and only for a bit that is not set yet: every warp may have the same news)
    if ((threadIdx.x & 31) == 0 && (*(volatile int*)err & e) != e)
        atomicOr(err, e);
}

// Element i starts a tile (keys sorted); flags duplicate (row, col) pairs.
struct new_tile {
    const uint64_t* keys;
    int shift;
    int* err;
    __device__ bool operator()(int64_t i) const
    {
        if (i == 0)
            return true;
        const uint64_t p = keys[i - 1], k = keys[i];
        if (p == k)
            atomicOr(err, kErrDuplicate);
        return (p >> shift) != (k >> shift);
    }
};

// head[i] = 1 where a new block starts (the sorted key changes).
__global__ void k_heads(const uint64_t* __restrict__ keys, int64_t nnz, int64_t* __restrict__ head)
{
    GRID_STRIDE(i, nnz)
    head[i] = i == 0 || keys[i - 1] != keys[i] ? 1 : 0;
}

// After an inclusive scan of the head flags, run_of[i] is 1 + the run of i.
__global__ void k_run_starts(const int64_t* __restrict__ run_of, int64_t nnz, int64_t* __restrict__ start)
{
    GRID_STRIDE(i, nnz)
    {
        const int64_t t = run_of[i] - 1;
        if (i == 0 || run_of[i - 1] != run_of[i])
            start[t] = i;
        if (i == nnz - 1)
            start[t + 1] = nnz;
    }
}

struct scheme_params {
    int64_t s;
    uint64_t bits;
    int is_binary, allow_csr, forced;
};

__global__ void k_tile_meta(int64_t T, int64_t nnz, const int64_t* __restrict__ tile_start,
                            const uint64_t* __restrict__ keys, int shift, uint64_t N, scheme_params sp,
                            int64_t* __restrict__ tile_row,
                            uint32_t* __restrict__ tile_col, uint32_t* __restrict__ tile_nnz,
                            uint8_t* __restrict__ tile_scheme, int64_t* __restrict__ stored,
                            int64_t* __restrict__ pay, int* __restrict__ err)
{
    GRID_STRIDE(t, T + 1)
    {
        if (t == T) {  // the scans run over T + 1 entries; the last yields the totals
            stored[T] = 0;
            pay[T] = 0;
            continue;
        }
        const int64_t s0 = tile_start[t], z = (t + 1 < T ? tile_start[t + 1] : nnz) - s0;
        const uint64_t tk = keys[s0] >> shift;
        int sch = sp.forced;
        if (sch < 0)
            sch = abhsf_select_scheme(sp.s, sp.s, (uint64_t)z, sp.bits, sp.is_binary, sp.allow_csr, nullptr);
        if (sch == ABHSF_SCHEME_CSR && z > 65535)
            atomicOr(err, kErrCsrTooLong);
        tile_row[t] = (int64_t)(tk / N);
        tile_col[t] = (uint32_t)(tk % N);
        tile_nnz[t] = (uint32_t)z;
        tile_scheme[t] = (uint8_t)sch;
        stored[t] = (sch == ABHSF_SCHEME_DENSE) ? sp.s * sp.s : z;
        pay[t] = tile_payload_bytes(sch, sp.s, z);
    }
}

// brow_ptr[i] = first tile whose block row is >= i.
__global__ void k_brow_ptr(int64_t M, int64_t T, const int64_t* __restrict__ tile_row, int64_t* __restrict__ brow_ptr)
{
    GRID_STRIDE(i, M + 1)
    {
        int64_t lo = 0, hi = T;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if (tile_row[mid] < i)
                lo = mid + 1;
            else
                hi = mid;
        }
        brow_ptr[i] = lo;
    }
}

__device__ __forceinline__ uint16_t f64_to_bf16_bits(double v)
{
    const float f = __double2float_rn(v);
    uint32_t u = __float_as_uint(f);
    if ((u & 0x7F800000u) == 0x7F800000u && (u & 0x007FFFFFu))
        return (uint16_t)((u >> 16) | 0x0040u);
    u += 0x7FFFu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}

// Every element to its tile's payload and values.  A CTA takes kScatter
// consecutive sorted elements: the first one's tile by a search (32 probes a
// step), the others' by counting the tile starts among them.  The value comes
// from the element's place in the input.  A bitmap word's bits are put together
// in the warp first: its elements are neighbours.
constexpr int kScatter = 2048;
__global__ void __launch_bounds__(kThreads) k_scatter(const uint64_t* __restrict__ keys,
                                                      const uint32_t* __restrict__ place,
                                                      const double* __restrict__ vals, int64_t nnz, int64_t T, int lg,
                                                      const int64_t* __restrict__ tile_start,
                                                      const uint8_t* __restrict__ tile_scheme,
                                                      const int64_t* __restrict__ tile_val_off,
                                                      const int64_t* __restrict__ tile_idx_off, int value_type,
                                                      uint8_t* __restrict__ payload, void* __restrict__ values)
{
    constexpr int PER = kScatter / kThreads;
    __shared__ uint64_t sk[kScatter + 2];  // the key before the chunk, the chunk's, the key after it
    __shared__ uint16_t rank[kScatter];    // tile starts up to and with the element
    __shared__ int wsum[kThreads / 32];
    __shared__ int64_t first;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, shift = 2 * lg;
    const int64_t s = int64_t(1) << lg;
    const uint64_t lmask = (uint64_t(1) << shift) - 1;
    for (int64_t base = blockIdx.x * (int64_t)kScatter; base < nnz; base += (int64_t)gridDim.x * kScatter) {
        const int n = (int)min((int64_t)kScatter, nnz - base);
        __syncthreads();
        for (int e = tid; e < n + 2; e += kThreads) {
            const int64_t i = base + e - 1;
            sk[e] = i >= 0 && i < nnz ? keys[i] : ~uint64_t(0);
        }
        if (warp == 0) {  // the last tile that starts at or before base
            int64_t lo = 0, hi = T;  // tile_start[lo] <= base, tile_start[hi] > base (tile_start[T] = nnz)
            while (hi - lo > 1) {
                const int64_t step = (hi - lo + 31) / 32, at = lo + step * (lane + 1);
                const bool le = at < hi && tile_start[at] <= base;
                const int k = __popc(__ballot_sync(0xffffffffu, le));  // starts ascend: the first k lanes
                const int64_t nlo = lo + step * k;
                hi = min(hi, nlo + step);
                lo = nlo;
            }
            if (lane == 0)
                first = lo;
        }
        __syncthreads();
        int starts[PER], sum = 0;  // thread: PER consecutive elements
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int e = tid * PER + j;
            // the first element's tile is `first`, whether it starts there or not
            sum += e > 0 && e < n && (sk[e] >> shift) != (sk[e + 1] >> shift);
            starts[j] = sum;
        }
        int inc = sum;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const int v = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= d)
                inc += v;
        }
        if (lane == 31)
            wsum[warp] = inc;
        __syncthreads();
        int before = inc - sum;
        for (int w = 0; w < warp; ++w)
            before += wsum[w];
#pragma unroll
        for (int j = 0; j < PER; ++j)
            rank[tid * PER + j] = (uint16_t)(before + starts[j]);
        __syncthreads();
        for (int e0 = 0; e0 < n; e0 += kThreads) {
            const int e = e0 + tid;
            const bool have = e < n;
            const int64_t i = base + e;
            const uint64_t key = sk[min(e, n - 1) + 1], local = key & lmask;
            const int64_t t = first + rank[min(e, n - 1)];
            const int64_t ts = tile_start[t], p = i - ts;
            const int sch = tile_scheme[t];
            uint8_t* pay = payload + tile_idx_off[t];
            const uint32_t lr = (uint32_t)(local >> lg), lc = (uint32_t)(local & (s - 1));
            if (have) {
                const int64_t vpos = tile_val_off[t] + (sch == ABHSF_SCHEME_DENSE ? (int64_t)local : p);
                const double v = vals ? vals[place[i]] : 1.0;
                if (value_type == ABHSF_VALUE_F64)
                    static_cast<double*>(values)[vpos] = v;
                else if (value_type == ABHSF_VALUE_F32)
                    static_cast<float*>(values)[vpos] = __double2float_rn(v);
                else
                    static_cast<uint16_t*>(values)[vpos] = f64_to_bf16_bits(v);
                if (sch == ABHSF_SCHEME_COO) {
                    reinterpret_cast<uint16_t*>(pay)[p] = (uint16_t)((lr << lg) | lc);
                } else if (sch == ABHSF_SCHEME_CSR) {
                    pay[2 * s + p] = (uint8_t)lc;
                    // The last element of each row writes row_end for its row and the
                    // empty rows that follow it (rows before the first element stay 0).
                    const uint64_t nk = sk[e + 2];
                    const bool last = i + 1 >= nnz || (nk >> shift) != (key >> shift);
                    const uint32_t next_lr = last ? (uint32_t)s : (uint32_t)((nk & lmask) >> lg);
                    uint16_t* row_end = reinterpret_cast<uint16_t*>(pay);
                    for (uint32_t r = lr; r < next_lr; ++r)
                        row_end[r] = (uint16_t)(p + 1);
                }
            }
            const unsigned bm = __ballot_sync(0xffffffffu, have && sch == ABHSF_SCHEME_BITMAP);
            if (have && sch == ABHSF_SCHEME_BITMAP) {
                const unsigned same = __match_any_sync(bm, key >> 6);  // one word of one tile
                uint64_t bits = uint64_t(1) << (local & 63);
                const int top = 31 - __clz(same);
                // the lanes of a word are neighbours: an inclusive OR towards its last lane
#pragma unroll
                for (int d = 1; d < 32; d *= 2) {
                    const uint64_t o = __shfl_up_sync(bm, bits, d);
                    if (lane >= d && ((same >> (lane - d)) & 1u))
                        bits |= o;
                }
                if (lane == top)
                    atomicOr(reinterpret_cast<unsigned long long*>(pay) + (local >> 6), (unsigned long long)bits);
            }
        }
    }
}

// Duplicate elements are counted like distinct ones (as block_stats.cpp does),
// so a run may exceed r * s: such runs are reported, never written past hist.
__global__ void k_len_hist(int64_t B, const int64_t* __restrict__ start, unsigned long long* __restrict__ hist,
                           int64_t hist_len, int* __restrict__ err)
{
    GRID_STRIDE(b, B)
    {
        const int64_t len = start[b + 1] - start[b];
        if (len < hist_len)
            atomicAdd(hist + len, 1ull);
        else
            atomicOr(err, kErrHistOverflow);
    }
}

__global__ void k_block_keys(const int64_t* __restrict__ rows, const int64_t* __restrict__ cols, int64_t nnz,
                             int64_t m, int64_t n, int k, int l, uint64_t* __restrict__ keys, int* __restrict__ err)
{
    GRID_STRIDE(i, nnz)
    {
        const int64_t r = rows[i], c = cols[i];
        if (r < 0 || r >= m || c < 0 || c >= n) {
            atomicOr(err, kErrRange);
            keys[i] = 0;
            continue;
        }
        // block_statistics/block_stats.cpp:69-74
        keys[i] = ((uint64_t(r) >> k) << 32) + (uint64_t(c) >> l);
    }
}

// Block lengths into a histogram held in shared memory (hist_len <= 8192),
// then added to the global one.
__global__ void k_len_hist_shared(int64_t B, const int64_t* __restrict__ start, int64_t nnz,
                                  unsigned long long* __restrict__ hist, int hist_len, int* __restrict__ err)
{
    extern __shared__ unsigned int sh[];
    for (int i = threadIdx.x; i < hist_len; i += blockDim.x)
        sh[i] = 0;
    __syncthreads();
    GRID_STRIDE(b, B)
    {
        const int64_t len = (b + 1 < B ? start[b + 1] : nnz) - start[b];
        if (len < hist_len)
            atomicAdd(&sh[len], 1u);
        else
            atomicOr(err, kErrHistOverflow);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < hist_len; i += blockDim.x)
        if (sh[i])
            atomicAdd(hist + i, (unsigned long long)sh[i]);
}

// Histogram of the tiles' nonzeros over many counters: tiles of few in shared
// memory first.
__global__ void k_nnz_hist(int64_t T, const uint32_t* __restrict__ nnz, unsigned long long* __restrict__ hist)
{
    constexpr int N = 4096;
    __shared__ unsigned int sh[N];
    for (int i = threadIdx.x; i < N; i += blockDim.x)
        sh[i] = 0;
    __syncthreads();
    GRID_STRIDE(t, T)
    {
        const uint32_t z = nnz[t];
        if (z < N)
            atomicAdd(&sh[z], 1u);
        else
            atomicAdd(hist + z, 1ull);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < N; i += blockDim.x)
        if (sh[i])
            atomicAdd(hist + i, (unsigned long long)sh[i]);
}

void check_launch(const char* what) { ABHSF_CUDA(cudaGetLastError()); (void)what; }

template <typename T>
T read_scalar(const T* dptr, cudaStream_t st)
{
    T v{};
    ABHSF_CUDA(cudaMemcpyAsync(&v, dptr, sizeof(T), cudaMemcpyDeviceToHost, st));
    ABHSF_CUDA(cudaStreamSynchronize(st));
    return v;
}

// Copies host inputs to the device (or wraps device inputs).
struct coo_inputs {
    scratch<int64_t> rows_d, cols_d;
    scratch<double> vals_d;
    const int64_t* rows = nullptr;
    const int64_t* cols = nullptr;
    const double* vals = nullptr;

    coo_inputs(const int64_t* r, const int64_t* c, const double* v, int64_t nnz, bool on_device, cudaStream_t st)
        : rows_d(st), cols_d(st), vals_d(st)
    {
        if (on_device) {
            rows = r; cols = c; vals = v;
            return;
        }
        rows_d.alloc(nnz);
        cols_d.alloc(nnz);
        ABHSF_CUDA(cudaMemcpyAsync(rows_d.get(), r, nnz * sizeof(int64_t), cudaMemcpyHostToDevice, st));
        ABHSF_CUDA(cudaMemcpyAsync(cols_d.get(), c, nnz * sizeof(int64_t), cudaMemcpyHostToDevice, st));
        rows = rows_d.get();
        cols = cols_d.get();
        if (v) {
            vals_d.alloc(nnz);
            ABHSF_CUDA(cudaMemcpyAsync(vals_d.get(), v, nnz * sizeof(double), cudaMemcpyHostToDevice, st));
            vals = vals_d.get();
        }
    }
};

// Segments sorted keys into runs of equal keys; returns the run count and fills
// start[0..runs] (start[runs] = nnz).
int64_t segment_runs(const uint64_t* keys, int64_t nnz, cudaStream_t st, scratch<int64_t>& start)
{
    scratch<int64_t> head(nnz, st), run_of(nnz, st);
    k_heads<<<grid_for(nnz), kThreads, 0, st>>>(keys, nnz, head.get());
    check_launch("k_heads");
    size_t tmp_bytes = 0;
    ABHSF_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tmp_bytes, head.get(), run_of.get(), nnz, st));
    scratch<uint8_t> tmp(tmp_bytes, st);
    ABHSF_CUDA(cub::DeviceScan::InclusiveSum(tmp.get(), tmp_bytes, head.get(), run_of.get(), nnz, st));
    const int64_t runs = read_scalar(run_of.get() + nnz - 1, st);
    start.alloc(runs + 1);
    k_run_starts<<<grid_for(nnz), kThreads, 0, st>>>(run_of.get(), nnz, start.get());
    check_launch("k_run_starts");
    return runs;
}

void exclusive_scan(int64_t* in, int64_t* out, int64_t count, cudaStream_t st)
{
    size_t tmp_bytes = 0;
    ABHSF_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, in, out, count, st));
    scratch<uint8_t> tmp(tmp_bytes, st);
    ABHSF_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), tmp_bytes, in, out, count, st));
}

void raise_err(int e)
{
    if (e & kErrRange)
        fail(ABHSF_ERROR_INDEX_OUT_OF_RANGE, "an element lies outside the m x n matrix");
    if (e & kErrDuplicate)
        fail(ABHSF_ERROR_DUPLICATE_ENTRY, "two elements share one (row, col) position");
    if (e & kErrCsrTooLong)
        fail(ABHSF_ERROR_UNSUPPORTED, "forced CSR tile with more than 65535 nonzeros (uint16 row_end)");
    if (e & kErrHistOverflow)
        fail(ABHSF_ERROR_INVALID_VALUE, "a block holds more elements than hist_len - 1 (duplicate elements)");
}

}  // namespace

void exclusive_scan_i64(const int64_t* in, int64_t* out, int64_t count, cudaStream_t st)
{
    size_t tmp_bytes = 0;
    ABHSF_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, in, out, count, st));
    scratch<uint8_t> tmp(tmp_bytes, st);
    ABHSF_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), tmp_bytes, in, out, count, st));
}

void inclusive_scan_i64(const int64_t* in, int64_t* out, int64_t count, cudaStream_t st)
{
    size_t tmp_bytes = 0;
    ABHSF_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tmp_bytes, in, out, count, st));
    scratch<uint8_t> tmp(tmp_bytes, st);
    ABHSF_CUDA(cub::DeviceScan::InclusiveSum(tmp.get(), tmp_bytes, in, out, count, st));
}

// Host computation of one mmf line (block_statistics/mmf.cpp:53-138) for a
// given single-precision element width bits1 (32 for INTEGER / REAL, 64 for
// COMPLEX, 0 for BINARY: mmf.cpp:34-47); the double line uses 2 * bits1.
void mmf_line_from_hist(int64_t m, int64_t n, int64_t nnz, int type, int64_t r, int64_t s,
                        const std::map<uint64_t, uint64_t>& hist, uint64_t bits1, uint64_t o1[8], uint64_t o2[8])
{
    const bool is_binary = (type == ABHSF_MATRIX_BINARY);
    const uint64_t M = (uint64_t)((m + r - 1) / r), N = (uint64_t)((n + s - 1) / s);
    uint64_t blocks = 0;
    for (const auto& kv : hist)
        blocks += kv.second;
    const uint64_t csr0 = M * abhsf_ceil_log2(N + 1) + blocks * abhsf_ceil_log2(N);
    uint64_t coo = csr0, csr = csr0, bmp = csr0, d1 = csr0, d2 = csr0, a1 = csr0, a2 = csr0, w1 = csr0, w2 = csr0;
    if (is_binary)
        d1 = d2 = UINT64_MAX;
    const uint64_t R = (uint64_t)r, S = (uint64_t)s;
    for (const auto& kv : hist) {
        const uint64_t z = kv.first, c = kv.second;
        if (!c)
            continue;
        coo += abhsf_coo_bits(R, S, z) * c;
        csr += abhsf_csr_bits(R, S, z) * c;
        bmp += abhsf_bitmap_bits(R, S) * c;
        if (!is_binary) {
            d1 += abhsf_dense_bits(R, S, z, bits1) * c;
            d2 += abhsf_dense_bits(R, S, z, 2 * bits1) * c;
        }
        uint64_t b;
        abhsf_select_scheme(R, S, z, bits1, is_binary, 1, &b);
        a1 += (b + 2) * c;
        abhsf_select_scheme(R, S, z, 2 * bits1, is_binary, 1, &b);
        a2 += (b + 2) * c;
        abhsf_select_scheme(R, S, z, bits1, is_binary, 0, &b);
        w1 += (b + 2) * c;
        abhsf_select_scheme(R, S, z, 2 * bits1, is_binary, 0, &b);
        w2 += (b + 2) * c;
    }
    const uint64_t coo32 = (uint64_t)nnz * 64, csr32 = ((uint64_t)m + 1 + (uint64_t)nnz) * 32;
    const uint64_t v1 = (uint64_t)nnz * bits1, v2 = 2 * v1;
    const uint64_t s1[8] = {coo32 + v1, csr32 + v1, coo + v1, csr + v1, bmp + v1, d1 + v1, a1 + v1, w1 + v1};
    const uint64_t s2[8] = {coo32 + v2, csr32 + v2, coo + v2, csr + v2, bmp + v2, d2 + v2, a2 + v2, w2 + v2};
    std::copy(s1, s1 + 8, o1);
    std::copy(s2, s2 + 8, o2);
}

namespace {

// The scheme follows from a tile's nonzeros (or is the forced one), so the
// histogram of the tiles' nonzeros gives every total.
void finish_stats(abhsf_matrix& a, const scheme_params& sp, const int64_t* tile_start, cudaStream_t st)
{
    const int64_t hl = (int64_t)a.s * a.s + 1;
    std::vector<uint64_t> h(hl, 0);
    if (a.T) {
        scratch<unsigned long long> dh(hl, st);
        scratch<int> err(1, st);
        ABHSF_CUDA(cudaMemsetAsync(dh.get(), 0, hl * sizeof(unsigned long long), st));
        if (hl <= 8192)
            k_len_hist_shared<<<std::min(grid_for(a.T), 148u * 4), kThreads, hl * sizeof(unsigned int), st>>>(
                a.T, tile_start, a.nnz, dh.get(), (int)hl, err.get());
        else
            k_nnz_hist<<<std::min(grid_for(a.T), 148u * 4), kThreads, 0, st>>>(a.T, a.tile_nnz.get(), dh.get());
        check_launch("k_len_hist_shared");
        ABHSF_CUDA(cudaMemcpyAsync(h.data(), dh.get(), hl * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
        ABHSF_CUDA(cudaStreamSynchronize(st));
    }
    abhsf_stats& s = a.stats;
    s = abhsf_stats{};
    s.m = a.m; s.n = a.n; s.nnz = a.nnz;
    s.block_size = a.s; s.value_type = a.value_type;
    s.block_rows = a.M; s.block_cols = a.N; s.tiles = a.T;
    std::map<uint64_t, uint64_t> hist;
    for (int64_t z = 1; z < hl; ++z)
        if (h[z]) {
            const int sch = sp.forced >= 0 ? sp.forced
                                           : abhsf_select_scheme(sp.s, sp.s, (uint64_t)z, sp.bits, sp.is_binary,
                                                                 sp.allow_csr, nullptr);
            s.tiles_per_scheme[sch] += h[z];
            s.nnz_per_scheme[sch] += z * h[z];
            hist.emplace_hint(hist.end(), z, h[z]);
        }
    s.stored_values = a.n_values;
    s.payload_bytes = a.payload_bytes;
    s.format_bytes = (a.M + 1) * 8 + a.T * (4 + 4 + 1) + (a.T + 1) * 16 + a.payload_bytes +
                     a.n_values * (int64_t)value_size(a.value_type);
    s.spmv_bytes = s.format_bytes;  // the row slices, where prepared, replace their block rows' part
    // mmf line at this block size whose "double" column has the dense-cost
    // width; binary matrices carry no value bits (mmf.cpp:45-46).
    uint64_t o1[8], o2[8];
    const uint64_t bits1 = (a.matrix_type == ABHSF_MATRIX_BINARY) ? 0 : sp.bits / 2;
    mmf_line_from_hist(a.m, a.n, a.nnz, a.matrix_type, a.s, a.s, hist, bits1, o1, o2);
    std::copy(o2, o2 + 8, s.msmf_bits);
}

}  // namespace

void build_matrix(const int64_t* rows, const int64_t* cols, const double* vals, int64_t nnz, int64_t m, int64_t n,
                  const abhsf_build_opts& o, cudaStream_t st, abhsf_matrix& a)
{
    const int lg = log2_exact(o.block_size);
    if (lg < 4 || lg > 8)
        fail(ABHSF_ERROR_INVALID_VALUE, "block_size must be 16, 32, 64, 128 or 256");
    if (o.value_type < 0 || o.value_type > 2)
        fail(ABHSF_ERROR_INVALID_VALUE, "value_type out of range");
    if (o.matrix_type < 0 || o.matrix_type > 3)
        fail(ABHSF_ERROR_INVALID_VALUE, "matrix_type out of range");
    if (o.matrix_type == ABHSF_MATRIX_COMPLEX)
        fail(ABHSF_ERROR_UNSUPPORTED, "complex values are not stored by this build");
    if (o.forced_scheme < -1 || o.forced_scheme > 3)
        fail(ABHSF_ERROR_INVALID_VALUE, "forced_scheme must be -1 or 0..3");
    if (o.sum_order != ABHSF_SUM_REFERENCE && o.sum_order != ABHSF_SUM_TREE)
        fail(ABHSF_ERROR_INVALID_VALUE, "sum_order must be ABHSF_SUM_REFERENCE or ABHSF_SUM_TREE");
    if (o.slice_tile_nnz < -1)
        fail(ABHSF_ERROR_INVALID_VALUE, "slice_tile_nnz must be -1, 0 or positive");
    const bool binary = (o.matrix_type == ABHSF_MATRIX_BINARY);
    if (binary && o.forced_scheme == ABHSF_SCHEME_DENSE)
        fail(ABHSF_ERROR_INVALID_VALUE, "dense scheme is never used for binary matrices");
    if (m <= 0 || n <= 0 || nnz < 0)
        fail(ABHSF_ERROR_INVALID_VALUE, "m and n must be positive and nnz non-negative");
    if (nnz > 0 && (!rows || !cols))
        fail(ABHSF_ERROR_INVALID_VALUE, "rows and cols must be non-NULL");
    if (!vals && !binary && nnz > 0)
        fail(ABHSF_ERROR_INVALID_VALUE, "vals may be NULL only for binary matrices");
    const int64_t s = o.block_size;
    const int64_t M = (m + s - 1) / s, N = (n + s - 1) / s;
    if (M > int64_t(UINT32_MAX) || N > int64_t(UINT32_MAX))
        fail(ABHSF_ERROR_UNSUPPORTED, "more than 2^32 block rows or columns");
    const int key_bits = bit_length((uint64_t)(M * N - 1)) + 2 * lg;
    if (key_bits > 64)
        fail(ABHSF_ERROR_UNSUPPORTED, "matrix too large for a 64-bit block key");
    const uint64_t dense_bits = o.bits_per_value > 0 ? (uint64_t)o.bits_per_value : 8 * value_size(o.value_type);

    a.m = m; a.n = n; a.nnz = nnz; a.s = (int32_t)s; a.lg = lg;
    a.value_type = o.value_type; a.matrix_type = o.matrix_type;
    a.sum_order = o.sum_order;
    a.dc_avg = o.slice_tile_nnz < 0 ? 0.f : o.slice_tile_nnz == 0 ? kSliceTileNnzDefault : (float)o.slice_tile_nnz;
    a.M = M; a.N = N;
    ABHSF_CUDA(cudaGetDevice(&a.device));

    if (nnz > int64_t(UINT32_MAX))  // (the inputs and the sort's buffers would not fit a GPU)
        fail(ABHSF_ERROR_OUT_OF_MEMORY, "more than 2^32 elements");

    // totals the host reads, together: error bits, tiles, stored values, payload bytes
    scratch<int64_t> totals(4, st);
    ABHSF_CUDA(cudaMemsetAsync(totals.get(), 0, 4 * sizeof(int64_t), st));
    int* err = reinterpret_cast<int*>(totals.get());
    int64_t tot[4] = {0, 0, 0, 0};
    auto read_totals = [&] {
        ABHSF_CUDA(cudaMemcpyAsync(tot, totals.get(), sizeof(tot), cudaMemcpyDeviceToHost, st));
        ABHSF_CUDA(cudaStreamSynchronize(st));
        raise_err((int)tot[0]);
    };
    scratch<int64_t> tile_row(st), stored(st), pay(st);
    scratch<uint64_t> keys_in(st), keys(st);
    scratch<uint32_t> place_in(st), place(st);
    int64_t* tile_start = nullptr;
    std::unique_ptr<coo_inputs> in;
    const int shift = 2 * lg;
    if (nnz > 0) {
        in = std::make_unique<coo_inputs>(rows, cols, binary ? nullptr : vals, nnz, o.inputs_on_device != 0, st);
        keys_in.alloc(nnz);
        place_in.alloc(nnz);
        keys.alloc(nnz);
        place.alloc(nnz);
        k_make_keys<<<grid_for(nnz), kThreads, 0, st>>>(in->rows, in->cols, nnz, m, n, lg, (uint64_t)N, keys_in.get(),
                                                         place_in.get(), err);
        check_launch("k_make_keys");
        read_totals();
        // Elements given row by row, columns ascending (CSR order, most files):
        // those of a tile are in its order already, and a stable sort by tile
        // leaves them so -- 4 passes instead of 6 for a 4M x 4M matrix.
        const int begin_bit = (tot[0] & kUnordered) ? 0 : std::min(shift, key_bits - 1);
        size_t b1 = 0, b2 = 0;
        const thrust::counting_iterator<int64_t> all(0);
        const new_tile head{keys.get(), shift, err};
        ABHSF_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b1, keys_in.get(), keys.get(), place_in.get(), place.get(),
                                                   nnz, begin_bit, key_bits, st));
        tile_start = reinterpret_cast<int64_t*>(keys_in.get());  // the unsorted keys' memory, once they are sorted
        ABHSF_CUDA(cub::DeviceSelect::If(nullptr, b2, all, tile_start, totals.get() + 1, nnz, head, st));
        scratch<uint8_t> tmp(std::max(b1, b2), st);
        ABHSF_CUDA(cub::DeviceRadixSort::SortPairs(tmp.get(), b1, keys_in.get(), keys.get(), place_in.get(),
                                                   place.get(), nnz, begin_bit, key_bits, st));
        ABHSF_CUDA(cub::DeviceSelect::If(tmp.get(), b2, all, tile_start, totals.get() + 1, nnz, head, st));
        read_totals();
    }
    const int64_t T = tot[1];
    a.T = T;
    a.brow_ptr.alloc(M + 1);
    a.tile_col.alloc(T);
    a.tile_nnz.alloc(T);
    a.tile_scheme.alloc(T);
    a.tile_val_off.alloc(T + 1);
    a.tile_idx_off.alloc(T + 1);
    tile_row.alloc(T);
    stored.alloc(T + 1);
    pay.alloc(T + 1);
    scheme_params sp{s, dense_bits, binary ? 1 : 0, o.allow_csr ? 1 : 0, o.forced_scheme};
    k_tile_meta<<<grid_for(T + 1), kThreads, 0, st>>>(T, nnz, tile_start, keys.get(), shift, (uint64_t)N, sp,
                                                       tile_row.get(), a.tile_col.get(), a.tile_nnz.get(),
                                                       a.tile_scheme.get(), stored.get(), pay.get(), err);
    check_launch("k_tile_meta");
    exclusive_scan(stored.get(), a.tile_val_off.get(), T + 1, st);
    exclusive_scan(pay.get(), a.tile_idx_off.get(), T + 1, st);
    k_brow_ptr<<<grid_for(M + 1), kThreads, 0, st>>>(M, T, tile_row.get(), a.brow_ptr.get());
    check_launch("k_brow_ptr");
    ABHSF_CUDA(cudaMemcpyAsync(totals.get() + 2, a.tile_val_off.get() + T, sizeof(int64_t), cudaMemcpyDeviceToDevice,
                               st));
    ABHSF_CUDA(cudaMemcpyAsync(totals.get() + 3, a.tile_idx_off.get() + T, sizeof(int64_t), cudaMemcpyDeviceToDevice,
                               st));
    read_totals();
    a.n_values = tot[2];
    a.payload_bytes = tot[3];
    a.payload.alloc(a.payload_bytes);
    // 16 bytes of padding: pipelined kernels copy 16-byte-aligned supersets of value ranges
    const size_t vs = value_size(a.value_type);
    a.values.alloc(a.n_values * vs + 16);
    ABHSF_CUDA(cudaMemsetAsync(a.payload.get(), 0, a.payload.size(), st));
    if (a.n_values == nnz)  // no dense tile: every value is written
        ABHSF_CUDA(cudaMemsetAsync(a.values.get() + a.n_values * vs, 0, 16, st));
    else
        ABHSF_CUDA(cudaMemsetAsync(a.values.get(), 0, a.values.size(), st));
    if (nnz > 0) {
        const unsigned g = (unsigned)std::min<int64_t>((nnz + kScatter - 1) / kScatter, 148 * 8);
        k_scatter<<<g, kThreads, 0, st>>>(keys.get(), place.get(), in->vals, nnz, T, lg, tile_start,
                                          a.tile_scheme.get(), a.tile_val_off.get(), a.tile_idx_off.get(),
                                          a.value_type, a.payload.get(), a.values.get());
        check_launch("k_scatter");
    }
    a.dev_status.alloc(1);
    ABHSF_CUDA(cudaMemsetAsync(a.dev_status.get(), 0, sizeof(int), st));
    finish_stats(a, sp, tile_start, st);
    in.reset();  // the sort's memory is not needed any more
    keys_in.reset();
    keys.reset();
    place_in.reset();
    place.reset();
    prepare_tree(a, st);
    prepare_ring(a, st);
    ABHSF_CUDA(cudaStreamSynchronize(st));  // the handle may be used on any stream from here on
}

void block_histogram(const int64_t* rows, const int64_t* cols, int64_t nnz, int64_t m, int64_t n, int r, int s,
                     bool on_device, cudaStream_t st, uint64_t* hist, int64_t hist_len, int64_t* blocks)
{
    const int k = log2_exact(r), l = log2_exact(s);
    if (k < 1 || k > 8 || l < 1 || l > 8)
        fail(ABHSF_ERROR_INVALID_VALUE, "r and s must be powers of two in 2..256");
    if (m <= 0 || n <= 0 || nnz < 0)
        fail(ABHSF_ERROR_INVALID_VALUE, "m and n must be positive and nnz non-negative");
    if (!hist || hist_len < (int64_t)r * s + 1)
        fail(ABHSF_ERROR_INVALID_VALUE, "hist must hold r*s + 1 counters");
    if (((uint64_t)(m - 1) >> k) >= (uint64_t(1) << 32) || ((uint64_t)(n - 1) >> l) >= (uint64_t(1) << 32))
        fail(ABHSF_ERROR_UNSUPPORTED, "block row or column index beyond 32 bits");
    std::fill(hist, hist + hist_len, 0);
    if (blocks)
        *blocks = 0;
    if (nnz == 0)
        return;
    if (!rows || !cols)
        fail(ABHSF_ERROR_INVALID_VALUE, "rows and cols must be non-NULL");
    coo_inputs in(rows, cols, nullptr, nnz, on_device, st);
    scratch<int> err(1, st);
    ABHSF_CUDA(cudaMemsetAsync(err.get(), 0, sizeof(int), st));
    scratch<uint64_t> keys(nnz, st), keys_out(nnz, st);
    k_block_keys<<<grid_for(nnz), kThreads, 0, st>>>(in.rows, in.cols, nnz, m, n, k, l, keys.get(), err.get());
    check_launch("k_block_keys");
    raise_err(read_scalar(err.get(), st));
    const int end_bit = 32 + bit_length((uint64_t)(m - 1) >> k);
    size_t tmp_bytes = 0;
    ABHSF_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, tmp_bytes, keys.get(), keys_out.get(), nnz, 0, end_bit, st));
    {
        scratch<uint8_t> tmp(tmp_bytes, st);
        ABHSF_CUDA(cub::DeviceRadixSort::SortKeys(tmp.get(), tmp_bytes, keys.get(), keys_out.get(), nnz, 0, end_bit,
                                                  st));
    }
    scratch<int64_t> start(st);
    const int64_t B = segment_runs(keys_out.get(), nnz, st, start);
    scratch<unsigned long long> dh(hist_len, st);
    ABHSF_CUDA(cudaMemsetAsync(dh.get(), 0, hist_len * sizeof(unsigned long long), st));
    // few counters: added up in shared memory first (most blocks hold one of a
    // few counts, and 32,768 threads adding to one address wait on each other)
    if (hist_len <= 8192)
        k_len_hist_shared<<<std::min(grid_for(B), 148u * 8), kThreads, hist_len * sizeof(unsigned int), st>>>(
            B, start.get(), nnz, dh.get(), (int)hist_len, err.get());
    else
        k_len_hist<<<grid_for(B), kThreads, 0, st>>>(B, start.get(), dh.get(), hist_len, err.get());
    check_launch("k_len_hist");
    ABHSF_CUDA(cudaMemcpyAsync(hist, dh.get(), hist_len * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    ABHSF_CUDA(cudaStreamSynchronize(st));
    raise_err(read_scalar(err.get(), st));
    if (blocks)
        *blocks = B;
}

// ---------------------------------------------------------------------------
// Block histogram that allocates nothing (abhsf_block_histogram_noalloc).
//
// For callers that may not call cudaMalloc: processes whose device memory is
// handed out by their own allocator or pool, paths where a cudaMalloc (which
// can synchronise the device) is not acceptable, and processes already at
// their device-memory limit.  All scratch lives in the array below, which is
// part of the library's device image: every GPU that loads the library holds
// it until the process exits.  Every call reuses it; a call clears what must
// start at zero, and calls that overlap on the GPU race on it.
namespace {

constexpr size_t kNoAllocScratchBytes = size_t(64) << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mutex;
unsigned char* g_noalloc_ptr[kNoAllocMaxDevices] = {};

// Device address of the scratch array on the current device.  Looked up once
// per device with that device current; host code may not use the symbol
// itself as an address.
unsigned char* noalloc_scratch()
{
    int dev = 0;
    ABHSF_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices)
        fail(ABHSF_ERROR_UNSUPPORTED, "device index beyond the no-allocation table");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        ABHSF_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
    }
    return g_noalloc_ptr[dev];
}

// Hands out 256-byte-aligned pieces of the scratch array.
struct scratch_arena {
    unsigned char* base;
    size_t cap, used = 0;
    template <typename T>
    T* take(size_t count)
    {
        const size_t bytes = (count * sizeof(T) + 255) & ~size_t(255);
        if (used + bytes > cap)
            fail(ABHSF_ERROR_INVALID_VALUE, "input too large for the no-allocation scratch");
        T* p = reinterpret_cast<T*>(base + used);
        used += bytes;
        return p;
    }
};

}  // namespace

void block_histogram_noalloc(const int64_t* rows, const int64_t* cols, int64_t nnz, int64_t m, int64_t n, int r,
                             int s, cudaStream_t st, uint64_t* hist, int64_t hist_len, int64_t* blocks)
{
    const int k = log2_exact(r), l = log2_exact(s);
    if (k < 1 || k > 8 || l < 1 || l > 8)
        fail(ABHSF_ERROR_INVALID_VALUE, "r and s must be powers of two in 2..256");
    if (m <= 0 || n <= 0 || nnz < 0)
        fail(ABHSF_ERROR_INVALID_VALUE, "m and n must be positive and nnz non-negative");
    if (nnz > ABHSF_NOALLOC_MAX_NNZ)
        fail(ABHSF_ERROR_INVALID_VALUE, "nnz exceeds ABHSF_NOALLOC_MAX_NNZ, the no-allocation limit");
    if (!hist || hist_len < (int64_t)r * s + 1)
        fail(ABHSF_ERROR_INVALID_VALUE, "hist must hold r*s + 1 counters");
    if (((uint64_t)(m - 1) >> k) >= (uint64_t(1) << 32) || ((uint64_t)(n - 1) >> l) >= (uint64_t(1) << 32))
        fail(ABHSF_ERROR_UNSUPPORTED, "block row or column index beyond 32 bits");
    if (nnz > 0 && (!rows || !cols))
        fail(ABHSF_ERROR_INVALID_VALUE, "rows and cols must be non-NULL device pointers");
    unsigned char* base = noalloc_scratch();  // before any early return: the set-up is per device
    std::fill(hist, hist + hist_len, 0);
    if (blocks)
        *blocks = 0;
    if (nnz == 0)
        return;
    const int64_t hl = (int64_t)r * s + 1;  // counters the device fills
    scratch_arena ar{base, kNoAllocScratchBytes};
    int* err = ar.take<int>(1);
    uint64_t* keys = ar.take<uint64_t>(nnz);
    uint64_t* keys_out = ar.take<uint64_t>(nnz);
    int64_t* head = ar.take<int64_t>(nnz);
    int64_t* run_of = ar.take<int64_t>(nnz);
    int64_t* start = ar.take<int64_t>(nnz + 1);
    unsigned long long* dh = ar.take<unsigned long long>(hl);
    const int end_bit = 32 + bit_length((uint64_t)(m - 1) >> k);
    size_t sort_bytes = 0, scan_bytes = 0;
    ABHSF_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, sort_bytes, keys, keys_out, nnz, 0, end_bit, st));
    ABHSF_CUDA(cub::DeviceScan::InclusiveSum(nullptr, scan_bytes, head, run_of, nnz, st));
    unsigned char* sort_tmp = ar.take<unsigned char>(sort_bytes);
    unsigned char* scan_tmp = ar.take<unsigned char>(scan_bytes);
    // the scratch keeps the previous call's contents: clear what must start at zero
    ABHSF_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    ABHSF_CUDA(cudaMemsetAsync(dh, 0, hl * sizeof(unsigned long long), st));
    k_block_keys<<<grid_for(nnz), kThreads, 0, st>>>(rows, cols, nnz, m, n, k, l, keys, err);
    check_launch("k_block_keys");
    raise_err(read_scalar(err, st));
    ABHSF_CUDA(cub::DeviceRadixSort::SortKeys(sort_tmp, sort_bytes, keys, keys_out, nnz, 0, end_bit, st));
    k_heads<<<grid_for(nnz), kThreads, 0, st>>>(keys_out, nnz, head);
    check_launch("k_heads");
    ABHSF_CUDA(cub::DeviceScan::InclusiveSum(scan_tmp, scan_bytes, head, run_of, nnz, st));
    const int64_t B = read_scalar(run_of + nnz - 1, st);
    k_run_starts<<<grid_for(nnz), kThreads, 0, st>>>(run_of, nnz, start);
    check_launch("k_run_starts");
    k_len_hist<<<grid_for(B), kThreads, 0, st>>>(B, start, dh, hl, err);
    check_launch("k_len_hist");
    ABHSF_CUDA(cudaMemcpyAsync(hist, dh, hl * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    ABHSF_CUDA(cudaStreamSynchronize(st));
    raise_err(read_scalar(err, st));
    if (blocks)
        *blocks = B;
}

}  // namespace abhsf
