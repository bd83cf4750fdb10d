// block_stats.cu -- block nonzero histograms for many block sizes from one
// sort, sm_100a.
//
// The reference's block_stats counts, for each of 64 block sizes 2^k x 2^l
// (k, l = 1..8), how many blocks hold 1, 2, ... nonzeros, sorting the elements
// anew for every size (block_statistics/block_stats.cpp:69-100,144-170).  Every
// such block lies inside one 256 x 256 tile, so the elements are sorted once, by
// tile (radix sort of the tile bits only; the key's low bits keep the position
// in the tile), and each tile is counted for all sizes at a time:
//
// * a tile of one or two elements by one lane: one element is one block of one
//   at every size, and two share a block exactly from the bit length of their
//   row and column differences on;
// * up to 32 elements by a warp, an element a lane: the lanes in the same 2^k
//   rows (a match of r >> k) and in the same 2^l columns, and a block's count is
//   the population of the two masks' intersection -- 16 matches for 64 sizes;
// * more by a CTA: counters of the 128 x 128 finest blocks in shared memory,
//   summed pairwise along the columns and then, in registers, along the rows.
//
// The square sizes 16 .. 256 of the min-bss choice go the same way from 16 x 16
// cells.  Counts are added up in shared memory per CTA where they are small.
// Bound by the sort: of the 60M elements of a tiled mixture, four passes over 8
// bytes an element.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>
#include <thrust/iterator/counting_iterator.h>

#include <algorithm>
#include <map>
#include <vector>

#include "common.cuh"
#include "internal.cuh"

namespace abhsf {
namespace {

constexpr int kThreads = 256;
constexpr unsigned kFull = 0xffffffffu;
constexpr int kFew = 32;    // elements a warp counts, one a lane
constexpr int kSmall = 128;  // counts below this are added up in shared memory (CTA path)

enum : int { kErrRange = 1, kErrOverflow = 2 };

// The block sizes of a run: all 64 (k = p / 8 + 1, l = p % 8 + 1, cells of 2 x
// 2), or the squares 16 .. 256 (cells of 16 x 16).  Size p's counters start at
// off[p].
template <bool ALL>
struct sizes {
    static constexpr int BITS = ALL ? 7 : 4;  // bits of a cell's row (and column) in the tile
    static constexpr int N = ALL ? 64 : 5;
    static constexpr int LEVELS = ALL ? 8 : 5;
    static constexpr int CELL = ALL ? 4 : 256;  // elements a cell can hold
    int off[N];
    int64_t total;
    sizes()
    {
        int o = 0;
        for (int p = 0; p < N; ++p) {
            off[p] = o;
            o += ALL ? (2 << (p / 8)) * (2 << (p % 8)) + 1 : (16 << p) * (16 << p) + 1;
        }
        total = o;
    }
};

// key = tile (256 x 256, row-major) << 2 BITS | cell row << BITS | cell column
template <bool ALL>
__global__ void k_tile_keys(const int64_t* __restrict__ rows, const int64_t* __restrict__ cols, int64_t nnz, int64_t m,
                            int64_t n, uint64_t NJ, uint64_t* __restrict__ keys, int* __restrict__ err)
{
    constexpr int B = sizes<ALL>::BITS;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = __ldcs(rows + i), c = __ldcs(cols + i);
        if (r < 0 || r >= m || c < 0 || c >= n) {
            atomicOr(err, kErrRange);
            keys[i] = 0;
            continue;
        }
        keys[i] = ((uint64_t(r >> 8) * NJ + uint64_t(c >> 8)) << (2 * B)) | (uint64_t(r & 255) >> (8 - B)) << B |
                  uint64_t(c & 255) >> (8 - B);
    }
}

struct new_tile {
    const uint64_t* keys;
    int shift;
    __device__ bool operator()(int64_t i) const { return i == 0 || (keys[i - 1] >> shift) != (keys[i] >> shift); }
};

// Tiles of up to kFew elements; the others are listed in many.
template <bool ALL>
__global__ void __launch_bounds__(kThreads) k_tiles_few(const int64_t* __restrict__ tiles,
                                                        const int64_t* __restrict__ start, int64_t nnz,
                                                        const uint64_t* __restrict__ keys, sizes<ALL> sz,
                                                        unsigned long long* __restrict__ hist,
                                                        int64_t* __restrict__ many, unsigned long long* __restrict__ nmany,
                                                        int* __restrict__ err)
{
    using Z = sizes<ALL>;
    constexpr int B = Z::BITS, L = Z::LEVELS, H = kFew + 1;
    constexpr uint32_t M = (1u << B) - 1u;
    __shared__ unsigned int h[Z::N * H];
    __shared__ unsigned int pairs[L * L];  // two-element tiles by the level from which they share rows, and columns
    __shared__ unsigned int singles;
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < Z::N * H; i += kThreads)
        h[i] = 0;
    for (int i = threadIdx.x; i < L * L; i += kThreads)
        pairs[i] = 0;
    if (threadIdx.x == 0)
        singles = 0;
    __syncthreads();
    const int64_t T = *tiles;
    unsigned int n1 = 0;
    bool over = false;
    const int64_t warps = (int64_t)gridDim.x * (kThreads / 32);
    for (int64_t t0 = 32 * (blockIdx.x * (int64_t)(kThreads / 32) + threadIdx.x / 32); t0 < T; t0 += 32 * warps) {
        const int64_t t = t0 + lane;
        int64_t s = 0, z = 0;
        if (t < T) {
            s = start[t];
            z = (t + 1 < T ? start[t + 1] : nnz) - s;
        }
        if (z == 1)
            ++n1;
        if (z == 2) {
            const uint32_t d = (uint32_t)(keys[s] ^ keys[s + 1]);
            const int kr = 32 - __clz((d >> B) & M), kc = 32 - __clz(d & M);
            atomicAdd(&pairs[kr * L + kc], 1u);
        }
        const unsigned big = __ballot_sync(kFull, z > kFew);
        if (big) {
            unsigned long long at = 0;
            if (lane == 0)
                at = atomicAdd(nmany, (unsigned long long)__popc(big));
            at = __shfl_sync(kFull, at, 0);
            if (z > kFew)
                many[at + __popc(big & ((1u << lane) - 1u))] = t;
        }
        for (unsigned mid = __ballot_sync(kFull, z > 2 && z <= kFew); mid; mid &= mid - 1) {
            const int src = __ffs(mid) - 1;
            const int64_t s0 = __shfl_sync(kFull, s, src);
            const int n = (int)__shfl_sync(kFull, z, src);
            const unsigned act = n == 32 ? kFull : (1u << n) - 1u;
            if (lane < n) {
                const uint32_t key = (uint32_t)keys[s0 + lane];
                unsigned rm[L], cm[L];
#pragma unroll
                for (int k = 0; k < L; ++k) {
                    rm[k] = __match_any_sync(act, ((key >> B) & M) >> k);
                    cm[k] = __match_any_sync(act, (key & M) >> k);
                }
#pragma unroll
                for (int p = 0; p < Z::N; ++p) {
                    const int k = ALL ? p / 8 : p, l = ALL ? p % 8 : p;
                    const unsigned same = rm[k] & cm[l];
                    const int cnt = __popc(same);
                    const bool lead = (same & ((1u << lane) - 1u)) == 0;
                    const unsigned ones = __ballot_sync(act, cnt == 1);
                    if (lane == 0 && ones)
                        atomicAdd(&h[p * H + 1], (unsigned)__popc(ones));
                    if (lead && cnt > 1)
                        atomicAdd(&h[p * H + cnt], 1u);
                    if (p == 0)
                        over = over || cnt > Z::CELL;
                }
            }
            __syncwarp();
        }
    }
    if (over)
        atomicOr(err, kErrOverflow);
#pragma unroll
    for (int d = 16; d > 0; d /= 2)
        n1 += __shfl_down_sync(kFull, n1, d);
    if (lane == 0 && n1)
        atomicAdd(&singles, n1);
    __syncthreads();
    // (a count above what a block holds only with over set: nothing is written past the counters)
    for (int i = threadIdx.x; i < Z::N * H; i += kThreads) {
        const int p = i / H, len = i % H;
        const int most = ALL ? (4 << (p / 8 + p % 8)) : (256 << (2 * p));
        if (h[i] && len <= most)
            atomicAdd(hist + sz.off[p] + len, (unsigned long long)h[i]);
    }
    for (int p = threadIdx.x; p < Z::N; p += kThreads) {
        const int k = ALL ? p / 8 : p, l = ALL ? p % 8 : p;
        unsigned long long two = 0, apart = 0;
        for (int c = 0; c < L * L; ++c)
            (c / L <= k && c % L <= l ? two : apart) += pairs[c];
        atomicAdd(hist + sz.off[p] + 1, (unsigned long long)singles + 2 * apart);
        atomicAdd(hist + sz.off[p] + 2, two);
    }
}

// A tile a CTA, all 64 sizes.  Counters in bytes: a cell of 2 x 2 holds at most
// four (a fifth element is a duplicate and stops the tile).
struct full_smem {
    uint8_t c1[128 * 128];       // counts of 2 x 2 cells: cell row * 128 + cell column
    uint8_t c[128 * 124];        // 2 x 2^l for l = 2 .. 6, level after level
    uint16_t c78[128 * 3];       // l = 7 (two columns), 8 (one)
    uint16_t s[16 * 255];        // 16 x 2^l: level after level, 16 rows of 256 >> l
    unsigned int h[64 * kSmall];
    int over;
};

__global__ void __launch_bounds__(kThreads) k_tiles_full(const int64_t* __restrict__ tiles,
                                                         const int64_t* __restrict__ start, int64_t nnz,
                                                         const uint64_t* __restrict__ keys, sizes<true> sz,
                                                         unsigned long long* __restrict__ hist,
                                                         const int64_t* __restrict__ many,
                                                         const unsigned long long* __restrict__ nmany,
                                                         int* __restrict__ err)
{
    extern __shared__ __align__(16) uint8_t full_raw[];
    full_smem& sm = *reinterpret_cast<full_smem*>(full_raw);
    const int tid = threadIdx.x;
    const int64_t T = *tiles, n = (int64_t)*nmany;
    uint32_t* c32 = reinterpret_cast<uint32_t*>(sm.c1);
    for (int i = tid; i < 64 * kSmall; i += kThreads)
        sm.h[i] = 0;
    if (tid == 0)
        sm.over = 0;
    auto count = [&](int k, int l, unsigned v) {  // a block of 2^k x 2^l with v elements
        if (v == 0)
            return;
        const int p = (k - 1) * 8 + l - 1;
        if (v < (unsigned)kSmall)
            atomicAdd(&sm.h[p * kSmall + v], 1u);
        else
            atomicAdd(hist + sz.off[p] + v, 1ull);
    };
    for (int64_t q = blockIdx.x; q < n; q += gridDim.x) {
        const int64_t t = many[q], s0 = start[t], s1 = t + 1 < T ? start[t + 1] : nnz;
        __syncthreads();
        for (int i = tid; i < 128 * 128 / 4; i += kThreads)
            c32[i] = 0;
        __syncthreads();
        for (int64_t i = s0 + tid; i < s1; i += kThreads) {
            const uint32_t cell = (uint32_t)keys[i] & 16383u;
            const int sh = 8 * (int)(cell & 3u);
            const uint32_t old = atomicAdd(c32 + (cell >> 2), 1u << sh);
            if (((old >> sh) & 255u) >= 4u)
                sm.over = 1;
        }
        __syncthreads();
        if (sm.over)
            break;
        // along the columns: 2 x 2^l from 2 x 2^(l - 1)
        for (int l = 2; l <= 8; ++l) {
            const int w = 256 >> l;
            const uint8_t* in = l == 2 ? sm.c1 : sm.c + 128 * (128 - (512 >> (l - 1)));
            uint8_t* out = sm.c + 128 * (128 - (512 >> l));
            for (int i = tid; i < 128 * w; i += kThreads) {
                if (l <= 6)
                    out[i] = (uint8_t)(in[2 * i] + in[2 * i + 1]);
                else if (l == 7)
                    sm.c78[i] = (uint16_t)(in[2 * i] + in[2 * i + 1]);
                else
                    sm.c78[256 + i] = (uint16_t)(sm.c78[2 * i] + sm.c78[2 * i + 1]);
            }
            __syncthreads();
        }
        // along the rows: eight cells of a column, heights 2 .. 16
        for (int idx = tid; idx < 4080; idx += kThreads) {
            const int l = __clz(4095 - idx) - 19, w = 256 >> l;
            const int j = idx - (4096 - (8192 >> l)), c = j & (w - 1), rb = j >> (8 - l);
            unsigned v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int at = (8 * rb + i) * w + c;
                v[i] = l == 1 ? sm.c1[at]
                       : l <= 6 ? sm.c[128 * (128 - (512 >> l)) + at]
                                : sm.c78[(l == 8 ? 256 : 0) + at];
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                count(1, l, v[i]);
#pragma unroll
            for (int k = 2, m = 4; k <= 4; ++k, m /= 2)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (i < m) {
                        v[i] = v[2 * i] + v[2 * i + 1];
                        count(k, l, v[i]);
                    }
            sm.s[16 * (256 - (512 >> l)) + rb * w + c] = (uint16_t)v[0];
        }
        __syncthreads();
        if (tid < 255) {  // heights 32 .. 256
            const int l = __clz(255 - tid) - 23, w = 256 >> l, c = tid - (256 - (512 >> l));
            unsigned v[16];
#pragma unroll
            for (int i = 0; i < 16; ++i)
                v[i] = sm.s[16 * (256 - (512 >> l)) + i * w + c];
#pragma unroll
            for (int k = 5, m = 8; k <= 8; ++k, m /= 2)
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i < m) {
                        v[i] = v[2 * i] + v[2 * i + 1];
                        count(k, l, v[i]);
                    }
        }
    }
    __syncthreads();
    if (tid == 0 && sm.over)
        atomicOr(err, kErrOverflow);
    for (int i = tid; i < 64 * kSmall; i += kThreads) {
        const int p = i / kSmall, len = i % kSmall;
        if (sm.h[i] && len <= (4 << (p / 8 + p % 8)))
            atomicAdd(hist + sz.off[p] + len, (unsigned long long)sm.h[i]);
    }
}

// A tile a warp, the square sizes.
__global__ void __launch_bounds__(kThreads) k_tiles_square(const int64_t* __restrict__ tiles,
                                                           const int64_t* __restrict__ start, int64_t nnz,
                                                           const uint64_t* __restrict__ keys, sizes<false> sz,
                                                           unsigned long long* __restrict__ hist,
                                                           const int64_t* __restrict__ many,
                                                           const unsigned long long* __restrict__ nmany,
                                                           int* __restrict__ err)
{
    __shared__ unsigned int cells[kThreads / 32][256];
    __shared__ unsigned int h[5 * kSmall];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t T = *tiles, n = (int64_t)*nmany;
    unsigned int* c = cells[warp];
    for (int i = threadIdx.x; i < 5 * kSmall; i += kThreads)
        h[i] = 0;
    __syncthreads();
    bool over = false;
    auto count = [&](int p, unsigned v) {
        if (v == 0)
            return;
        if (v < (unsigned)kSmall)
            atomicAdd(&h[p * kSmall + v], 1u);
        else if (v <= (256u << (2 * p)))
            atomicAdd(hist + sz.off[p] + v, 1ull);
        else
            over = true;
    };
    for (int64_t q = blockIdx.x * (int64_t)(kThreads / 32) + warp; q < n; q += (int64_t)gridDim.x * (kThreads / 32)) {
        const int64_t t = many[q], s0 = start[t], s1 = t + 1 < T ? start[t + 1] : nnz;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            c[lane + 32 * i] = 0;
        __syncwarp();
        for (int64_t i = s0 + lane; i < s1; i += 32)
            atomicAdd(c + ((uint32_t)keys[i] & 255u), 1u);
        __syncwarp();
        // size 16 << p: (16 >> p) x (16 >> p) blocks, summed in place (a lane writes what it alone reads)
#pragma unroll
        for (int i = 0; i < 8; ++i)
            count(0, c[lane + 32 * i]);
#pragma unroll
        for (int p = 1; p < 5; ++p) {
            const int w = 16 >> p;  // the finer grid has 2 w columns
            unsigned v[2] = {0, 0};
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int b = lane + 32 * i;
                if (b < w * w) {
                    const unsigned* f = c + (b / w) * 4 * w + (b % w) * 2;
                    v[i] = f[0] + f[1] + f[2 * w] + f[2 * w + 1];
                    count(p, v[i]);
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 2; ++i)
                if (lane + 32 * i < w * w)
                    c[lane + 32 * i] = v[i];
            __syncwarp();
        }
    }
    if (over)
        atomicOr(err, kErrOverflow);
    __syncthreads();
    for (int i = threadIdx.x; i < 5 * kSmall; i += kThreads)
        if (h[i])
            atomicAdd(hist + sz.off[i / kSmall] + i % kSmall, (unsigned long long)h[i]);
}

// Every size's counters, one after another, into hist (host).
template <bool ALL>
void histograms(const int64_t* rows, const int64_t* cols, int64_t nnz, int64_t m, int64_t n, bool on_device,
                cudaStream_t st, uint64_t* hist)
{
    constexpr int shift = 2 * sizes<ALL>::BITS;
    const sizes<ALL> sz;
    int dev = 0, nsm = 0;
    ABHSF_CUDA(cudaGetDevice(&dev));
    ABHSF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const uint64_t NI = (uint64_t)((m + 255) >> 8), NJ = (uint64_t)((n + 255) >> 8);
    const int end_bit = shift + bit_length(NI * NJ - 1);
    // counters: the histograms, then the number of tiles of more than kFew
    // elements, the number of tiles, the error bits
    scratch<unsigned long long> dh(sz.total + 3, st);
    unsigned long long* nmany = dh.get() + sz.total;
    int64_t* tiles = reinterpret_cast<int64_t*>(nmany + 1);
    int* err = reinterpret_cast<int*>(nmany + 2);
    scratch<uint64_t> keys(nnz, st), sorted(nnz, st);
    scratch<int64_t> many(nnz / (kFew + 1) + 1, st);
    scratch<int64_t> rows_d(st), cols_d(st);  // host inputs
    if (!on_device) {
        rows_d.alloc(nnz);
        cols_d.alloc(nnz);
        ABHSF_CUDA(cudaMemcpyAsync(rows_d.get(), rows, nnz * sizeof(int64_t), cudaMemcpyHostToDevice, st));
        ABHSF_CUDA(cudaMemcpyAsync(cols_d.get(), cols, nnz * sizeof(int64_t), cudaMemcpyHostToDevice, st));
        rows = rows_d.get();
        cols = cols_d.get();
    }
    ABHSF_CUDA(cudaMemsetAsync(dh.get(), 0, dh.size() * sizeof(unsigned long long), st));
    const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((nnz + kThreads - 1) / kThreads, nsm * 32));
    k_tile_keys<ALL><<<g, kThreads, 0, st>>>(rows, cols, nnz, m, n, NJ, keys.get(), err);
    ABHSF_CUDA(cudaGetLastError());
    const new_tile head{sorted.get(), shift};
    const thrust::counting_iterator<int64_t> all(0);
    int64_t* start = reinterpret_cast<int64_t*>(keys.get());  // the unsorted keys' memory, once they are sorted
    size_t b1 = 0, b2 = 0;
    ABHSF_CUDA(cub::DeviceRadixSort::SortKeys(nullptr, b1, keys.get(), sorted.get(), nnz, shift,
                                              std::max(end_bit, shift + 1), st));
    ABHSF_CUDA(cub::DeviceSelect::If(nullptr, b2, all, start, tiles, nnz, head, st));
    scratch<uint8_t> tmp(std::max(b1, b2), st);
    ABHSF_CUDA(cub::DeviceRadixSort::SortKeys(tmp.get(), b1, keys.get(), sorted.get(), nnz, shift,
                                              std::max(end_bit, shift + 1), st));
    ABHSF_CUDA(cub::DeviceSelect::If(tmp.get(), b2, all, start, tiles, nnz, head, st));
    const unsigned gf = (unsigned)std::max<int64_t>(1, std::min<int64_t>((nnz + 1023) / 1024, nsm * 8));
    k_tiles_few<ALL><<<gf, kThreads, 0, st>>>(tiles, start, nnz, sorted.get(), sz, dh.get(), many.get(), nmany, err);
    ABHSF_CUDA(cudaGetLastError());
    const int64_t most = nnz / (kFew + 1);  // tiles of more than kFew elements
    if constexpr (ALL) {
        ABHSF_CUDA(cudaFuncSetAttribute(k_tiles_full, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)sizeof(full_smem)));
        const unsigned gt = (unsigned)std::max<int64_t>(1, std::min<int64_t>(most, nsm * 3));
        k_tiles_full<<<gt, kThreads, sizeof(full_smem), st>>>(tiles, start, nnz, sorted.get(), sz, dh.get(), many.get(),
                                                              nmany, err);
    } else {
        const unsigned gt = (unsigned)std::max<int64_t>(1, std::min<int64_t>((most + 7) / 8, nsm * 8));
        k_tiles_square<<<gt, kThreads, 0, st>>>(tiles, start, nnz, sorted.get(), sz, dh.get(), many.get(), nmany, err);
    }
    ABHSF_CUDA(cudaGetLastError());
    uint64_t tail[3];
    ABHSF_CUDA(cudaMemcpyAsync(hist, dh.get(), sz.total * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
    ABHSF_CUDA(cudaMemcpyAsync(tail, nmany, sizeof(tail), cudaMemcpyDeviceToHost, st));
    ABHSF_CUDA(cudaStreamSynchronize(st));
    const int e = (int)(uint32_t)tail[2];
    if (e & kErrRange)
        fail(ABHSF_ERROR_INDEX_OUT_OF_RANGE, "an element lies outside the m x n matrix");
    if (e & kErrOverflow)
        fail(ABHSF_ERROR_INVALID_VALUE, "a block holds more elements than hist_len - 1 (duplicate elements)");
}

}  // namespace

void block_histogram_all(const int64_t* rows, const int64_t* cols, int64_t nnz, int64_t m, int64_t n, bool on_device,
                         cudaStream_t st, uint64_t* hist, int64_t* blocks)
{
    if (m <= 0 || n <= 0 || nnz < 0)
        fail(ABHSF_ERROR_INVALID_VALUE, "m and n must be positive and nnz non-negative");
    if (!hist)
        fail(ABHSF_ERROR_INVALID_VALUE, "hist must hold ABHSF_BSTATS_ALL_LEN counters");
    if ((uint64_t)(m - 1) >= (uint64_t(1) << 32) || ((uint64_t)(n - 1) >> 1) >= (uint64_t(1) << 32))
        fail(ABHSF_ERROR_UNSUPPORTED, "row index or block column index beyond 32 bits");
    std::fill(hist, hist + ABHSF_BSTATS_ALL_LEN, 0);
    if (blocks)
        std::fill(blocks, blocks + 64, 0);
    if (nnz == 0)
        return;
    if (!rows || !cols)
        fail(ABHSF_ERROR_INVALID_VALUE, "rows and cols must be non-NULL");
    histograms<true>(rows, cols, nnz, m, n, on_device, st, hist);
    if (blocks) {
        const sizes<true> sz;
        for (int p = 0; p < 64; ++p) {
            const int64_t end = p + 1 < 64 ? sz.off[p + 1] : sz.total;
            for (int64_t i = sz.off[p]; i < end; ++i)
                blocks[p] += (int64_t)hist[i];
        }
    }
}

// ABHSF storage (bits, the mmf line's abhsf column at the stored value width,
// CSR as the options allow) of square block sizes 16, 32, 64, 128, 256: the
// quantity the reference's min-bss tool minimises (block_statistics/min-bss.cpp:14-58).
void block_size_storage(const int64_t* rows, const int64_t* cols, int64_t nnz, int64_t m, int64_t n,
                        const abhsf_build_opts& o, cudaStream_t st, uint64_t bits[kNumBlockSizes])
{
    if (o.value_type < 0 || o.value_type > 2)
        fail(ABHSF_ERROR_INVALID_VALUE, "value_type out of range");
    if (o.matrix_type < 0 || o.matrix_type > 3)
        fail(ABHSF_ERROR_INVALID_VALUE, "matrix_type out of range");
    const uint64_t dense_bits = o.bits_per_value > 0 ? (uint64_t)o.bits_per_value : 8 * value_size(o.value_type);
    const uint64_t bits1 = (o.matrix_type == ABHSF_MATRIX_BINARY) ? 0 : dense_bits / 2;
    if (nnz > 0 && (!rows || !cols))
        fail(ABHSF_ERROR_INVALID_VALUE, "rows and cols must be non-NULL");
    if (m <= 0 || n <= 0 || nnz < 0)
        fail(ABHSF_ERROR_INVALID_VALUE, "m and n must be positive and nnz non-negative");
    if (((uint64_t)(m - 1) >> 4) >= (uint64_t(1) << 32) || ((uint64_t)(n - 1) >> 4) >= (uint64_t(1) << 32))
        fail(ABHSF_ERROR_UNSUPPORTED, "block row or column index beyond 32 bits");
    const sizes<false> sz;
    std::vector<uint64_t> h((size_t)sz.total, 0);
    if (nnz > 0)
        histograms<false>(rows, cols, nnz, m, n, o.inputs_on_device != 0, st, h.data());
    for (int k = 0; k < kNumBlockSizes; ++k) {
        const int s = 16 << k;
        std::map<uint64_t, uint64_t> hist;
        for (int z = 1; z <= s * s; ++z)
            if (h[sz.off[k] + z])
                hist[z] = h[sz.off[k] + z];
        uint64_t o1[8], o2[8];
        mmf_line_from_hist(m, n, nnz, o.matrix_type, s, s, hist, bits1, o1, o2);
        bits[k] = o.allow_csr ? o2[6] : o2[7];
    }
}

int select_block_size(const uint64_t bits[kNumBlockSizes])
{
    int best = 0;
    for (int k = 1; k < kNumBlockSizes; ++k)
        if (bits[k] < bits[best])
            best = k;
    return 16 << best;
}

}  // namespace abhsf
