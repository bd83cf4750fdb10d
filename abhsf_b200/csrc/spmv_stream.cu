// spmv_stream.cu -- y += A x over hypersparse block rows through delta-coded
// row slices, in the reference's summation order, sm_100a.
//
// A block row whose tiles hold one or a few elements each costs the ring
// kernel (spmv_ring.cu) a descriptor, an x block and a tile walk per tile for
// a few multiply-adds.  Such block rows are re-encoded once, when the matrix
// is prepared, the way the reference's delta COO keeps a matrix
// (spmv/orig/delta.cpp:118-219, spmv/unified/spmv.cpp:815-1032: elements row
// by row, columns ascending, each column stored as the difference to the
// previous one), laid out for a warp:
//
// * The non-empty rows of a range of block rows (slice_segments) are ordered
//   by length (longest first, then ascending row) and dealt to slices of up
//   to 32 rows, one row per lane, so that a slice's rows end together.  A
//   slice stores its rows' elements column-major -- element k of lane l at
//   slot base + 32 k + l -- as one 32-bit word each, the column minus the
//   row's previous column (the first one absolute), and a copy of the value.
//   A lane record (offset << 8 | length - 1, the offset from the range's
//   first row) says which row a lane sums.
// * A row longer than kChainMin is a slice of its own (a chain): its elements
//   stored in order, each word the absolute column.
//
// A warp sums one slice at a time.  Sliced rows: every lane walks its row,
// kUnroll elements per step -- coalesced word and value loads (the active
// lanes are always a prefix, rows being ordered by length), the column by a
// running sum of the deltas, x gathered through L2 -- and adds each product
// onto its row's sum in column order, starting from y: the order of the
// reference CSR's spmv_naive (spmv/bottlenecks/spmv.cpp:58-64), so y is
// bitwise the same.  A chain (its own kernel, beside the others): 512 products
// at a time, in turn or a segment a lane by the rule of chain_sum.cuh, which
// gives the same bits.  For one matrix the chains are queued first (the longest
// bounds the product), in a batch behind the ring kernel, whose CTAs they would
// keep from an SM.  Slices and chains are dealt to warps at preparation time,
// longest first.  Nothing here stalls on another warp.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <queue>
#include <vector>

#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>

#include "chain_sum.cuh"
#include "common.cuh"
#include "internal.cuh"

namespace abhsf {

namespace {

constexpr int kWarpsPerCta = 8;
constexpr int kCtasPerSm = 4;     // CTAs per SM in the grid (64 registers a thread)
constexpr int kUnroll = 4;        // elements a lane loads per step of a sliced row
constexpr int kChainWarps = 4;    // warps per CTA of the chain kernel
constexpr int kChainCtasPerSm = 4;  // register bound of the chain kernel (128 a thread)
constexpr int kChainGridPerSm = 1;  // chain CTAs per SM in the grid: the rest of the SM is left to the others
constexpr int kSliceGridPerSm = 3;  // sliced-row CTAs per SM beside chains
constexpr int kChainGroup = 512;  // chain: elements a warp sums at a time, 16 a lane
constexpr int kMmCols = 4;        // columns a warp of the SpMM kernels serves
constexpr int kMmWide = 16;       // ... and of the sliced-row one where there are as many and no chains
constexpr int kMmWarps = 2;       // sliced-row SpMM: warps a CTA (small ones fit beside the chains)
constexpr int64_t kMmManySteps = 40;  // ... steps a warp from which on warps count for four columns
constexpr int kMmCtas = 16, kMmLateCtas = 10;  // ... and CTAs an SM where warps count, and where latency does
constexpr uint32_t kChain = 1u;   // dc_slice::geo: a one-row chain
constexpr int kMidShift = 20;     // dc_slice::geo: matrix index of a batch
constexpr int kLenBits = 8;       // lane record: row offset << kLenBits | (length - 1)
constexpr uint32_t kLenMask = (1u << kLenBits) - 1u;
constexpr int kChainMin = 256;   // rows longer than this are summed alone, as a chain
static_assert(kChainMin <= (1 << kLenBits), "a sliced row's length - 1 fits the lane record");
constexpr int kRingTilesMax = 256;  // block rows of more tiles go to the slices whatever their density

// What the kernel needs of one slice (32 bytes, in schedule order).
struct __align__(16) dc_slice {
    int64_t base;    // first slot of its words and values
    int64_t meta;    // sliced: first of its 32 lane records; chain: the row within the block row
    uint32_t brow;   // block row
    uint32_t steps;  // sliced: elements of its longest row; chain: the row's elements
    uint32_t lanes;  // rows (1 for a chain)
    uint32_t geo;    // kChain | matrix index << kMidShift
};
static_assert(sizeof(dc_slice) == 32, "dc_slice is 32 bytes");

template <int VT>
struct vt_of {
    using V = double;
    using T = double;
};
template <>
struct vt_of<ABHSF_VALUE_F32> {
    using V = float;
    using T = float;
};
template <>
struct vt_of<ABHSF_VALUE_BF16> {
    using V = uint16_t;
    using T = float;
};

__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float dmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float dadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double wide(double v) { return v; }
__device__ __forceinline__ float wide(float v) { return v; }
__device__ __forceinline__ float wide(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }

// Shared memory of one warp of the chain kernel: two halves of a group's x and
// values, each lane's 16 padded by 16 bytes.
template <typename T, typename V>
__host__ __device__ constexpr int chain_smem_warp()
{
    return 2 * 32 * (16 * (int)(sizeof(T) + sizeof(V)) + 32);
}

// Streamed once: loaded with the evict-first hint so that x stays in L2.
__device__ __forceinline__ uint32_t ld_stream(const uint32_t* p) { return __ldcs(p); }
__device__ __forceinline__ double ld_stream(const double* p) { return __ldcs(p); }
__device__ __forceinline__ float ld_stream(const float* p) { return __ldcs(p); }
__device__ __forceinline__ uint16_t ld_stream(const uint16_t* p)
{
    return __ldcs(reinterpret_cast<const unsigned short*>(p));
}

// One matrix of a launch.
struct dc_mat {
    const uint32_t* words;
    const void* vals;        // values in slot order
    const uint32_t* lane;    // lane records
    int64_t m;
};

struct dc_args {
    const dc_slice* slices;  // every warp's slices, warp after warp
    const int64_t* wbeg;     // [warps + 1]
    int warps;
    dc_mat A;                // the matrix (B = false)
    const void* x;
    void* y;
    int64_t ldx, ldy;        // SpMM: x[i * ldx + column], y[i * ldy + column]
    int cols;                // SpMM: columns
    int fresh;               // SpMV: y = A x (y starts from zero)
    int wait;                // waits for the kernel before it at its start
    const int* skip;         // nothing is done where *skip is set
    const dc_mat* mats;      // a batch (B = true): matrix i's arrays, x and y
    const void* const* xs;
    void* const* ys;
};

// The start of an SpMV kernel: lets the next kernel start -- after the kernel
// before is complete, for the first kernel of a product that was queued while
// that one ran (spmv_set_y).  True where there is nothing to do.  (x, which that
// kernel wrote, is read by plain loads: the read-only path promises nothing
// about data written during the kernel's life.)
__device__ __forceinline__ bool begin(const dc_args& P)
{
    if (P.wait)
        asm volatile("griddepcontrol.wait;" ::: "memory");
    beside_begin();
    return P.skip && *reinterpret_cast<const volatile int*>(P.skip) != 0;
}

// Sliced rows.  A warp sums its dealt slices one after another, each lane
// one row.  The next slice's descriptor and lane record, and the next step's
// words and values, are loaded while the current ones are summed, so that a
// step waits only on its x gathers.
template <int S, int VT, bool B>
__global__ void __launch_bounds__(32 * kWarpsPerCta, kCtasPerSm) k_spmv_slices(dc_args P)
{
    using T = typename vt_of<VT>::T;
    using V = typename vt_of<VT>::V;
    // f32 / bf16 values leave room in 64 registers for twice the steps in flight
    // (bf16 one fewer: 213 us against 241 on the 3D Laplacian 256^3, 227 with 4;
    // rows of 21 or of power-law lengths the same)
    constexpr int U = VT == ABHSF_VALUE_F64 ? kUnroll : VT == ABHSF_VALUE_BF16 ? 2 * kUnroll - 1 : 2 * kUnroll;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gw = blockIdx.x * kWarpsPerCta + warp;
    const bool nothing = begin(P);
    if (gw >= P.warps)
        return;
    int64_t si = P.wbeg[gw];
    const int64_t s1 = nothing ? si : P.wbeg[gw + 1];
    // (one way out: with a second return here the loop took 4% longer in FP64)
    if (si < s1) {
        auto mat = [&](const dc_slice& q) -> const dc_mat& { return B ? P.mats[q.geo >> kMidShift] : P.A; };
        auto record = [&](const dc_slice& q) -> uint32_t {
            return lane < (int)q.lanes ? mat(q).lane[q.meta + lane] : 0u;
        };
        dc_slice sl = P.slices[si];
        dc_slice nx = si + 1 < s1 ? P.slices[si + 1] : sl;
        uint32_t rec = record(sl);
#pragma unroll 1
        for (; si < s1; ++si) {
            const bool more = si + 1 < s1;
            const dc_slice nn = si + 2 < s1 ? P.slices[si + 2] : nx;
            const uint32_t rec_n = more ? record(nx) : 0u;
            const int mid = (int)(sl.geo >> kMidShift);
            const dc_mat& M = mat(sl);
            const T* X = static_cast<const T*>(B ? P.xs[mid] : P.x);
            T* Y = static_cast<T*>(B ? P.ys[mid] : P.y);
            const uint32_t* W = M.words + sl.base + lane;
            const V* Vv = static_cast<const V*>(M.vals) + sl.base + lane;
            // one row per lane, element k of the lane's row at slot 32 k + lane
            const int len = lane < (int)sl.lanes ? (int)(rec & kLenMask) + 1 : 0;
            const int64_t row = (int64_t)sl.brow * S + (int64_t)(rec >> kLenBits);
            T acc = len && !P.fresh ? Y[row] : T(0);
            uint32_t col = 0;
            // values stay in their stored type until their product: a widening
            // at the load would wait for the prefetch it belongs to
            uint32_t w[U];
            V v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                w[u] = u < len ? ld_stream(W + 32 * u) : 0u;
                v[u] = u < len ? ld_stream(Vv + 32 * u) : V(0);
            }
#pragma unroll 1
            for (int k0 = 0; k0 < (int)sl.steps; k0 += U) {
                uint32_t wn[U];
                V vn[U];
                T x[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {  // the next step's words and values
                    const int k = k0 + U + u;
                    wn[u] = k < len ? ld_stream(W + 32 * k) : 0u;
                    vn[u] = k < len ? ld_stream(Vv + 32 * k) : V(0);
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    col += w[u];
                    x[u] = k0 + u < len ? X[col] : T(0);
                }
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (k0 + u < len)
                        acc = dadd(acc, dmul(wide(v[u]), x[u]));
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    w[u] = wn[u];
                    v[u] = vn[u];
                }
            }
            if (len)
                Y[row] = acc;
            sl = nx;
            nx = nn;
            rec = rec_n;
        }
    }
    beside_end();
}

// Asynchronous 4- or 8-byte copy of one element to shared memory.
template <typename T>
__device__ __forceinline__ void cp_async(T* dst, const T* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(sizeof(T))
                 : "memory");
}

// The 16 values of a lane's segment (16-byte aligned in shared memory).
template <typename V>
__device__ __forceinline__ void load16(const V* q, V (&t)[16])
{
    constexpr int N = 16 / (int)sizeof(V);  // values of one 16-byte read
#pragma unroll
    for (int k = 0; k < 16 / N; ++k) {
        union {
            uint4 u;
            V v[N];
        } c;
        c.u = reinterpret_cast<const uint4*>(q)[k];
#pragma unroll
        for (int i = 0; i < N; ++i)
            t[N * k + i] = c.v[i];
    }
}

// ... and back.
template <typename V>
__device__ __forceinline__ void store16(V* q, const V (&t)[16])
{
    constexpr int N = 16 / (int)sizeof(V);
#pragma unroll
    for (int k = 0; k < 16 / N; ++k) {
        union {
            uint4 u;
            V v[N];
        } c;
#pragma unroll
        for (int i = 0; i < N; ++i)
            c.v[i] = t[N * k + i];
        reinterpret_cast<uint4*>(q)[k] = c.u;
    }
}

// Eight consecutive values from shared memory (16-byte aligned), in two or
// four 16-byte loads.
__device__ __forceinline__ void load8(const double* q, double (&t)[8])
{
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double2 u = reinterpret_cast<const double2*>(q)[k];
        t[2 * k] = u.x;
        t[2 * k + 1] = u.y;
    }
}
__device__ __forceinline__ void load8(const float* q, float (&t)[8])
{
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float4 u = reinterpret_cast<const float4*>(q)[k];
        t[4 * k] = u.x;
        t[4 * k + 1] = u.y;
        t[4 * k + 2] = u.z;
        t[4 * k + 3] = u.w;
    }
}

// Adds nseg runs of 16 products, `stride` values apart in shared memory, onto
// run one after another (every lane the same: broadcast loads).  Eight
// products are loaded while the eight before them are added, so that nothing
// but the adds lies on the chain; eight runs at a time (one at a time a lone row
// of 60,000 took 152 us in f32, 137 so).
template <typename T>
__device__ __forceinline__ T add_in_turn(T run, const T* q, int stride, int nseg)
{
    T t[8], u[8];
    load8(q, t);
    auto add_run = [&](bool more) {
        load8(q + 8, u);
#pragma unroll
        for (int k = 0; k < 8; ++k)
            run = dadd(run, t[k]);
        q += stride;
        if (more)
            load8(q, t);
#pragma unroll
        for (int k = 0; k < 8; ++k)
            run = dadd(run, u[k]);
    };
    int b = nseg;
#pragma unroll 1
    for (; b > 8; b -= 8)
#pragma unroll
        for (int k = 0; k < 8; ++k)
            add_run(true);
#pragma unroll 1
    for (; b > 0; --b)
        add_run(b > 1);
    return run;
}

// A chain as a warp walks it, kChainGroup elements at a time.
template <typename T, typename V>
struct chain_pos {
    int64_t si;   // its place in the schedule
    int b0, len;  // first element of the group; the row's elements
    const uint32_t* W;
    const V* Vv;
    const T* X;
    T* y;
};

template <int S, bool B, typename T, typename V>
__device__ __forceinline__ void chain_at(const dc_args& P, const dc_slice& sl, chain_pos<T, V>& c)
{
    const int mid = (int)(sl.geo >> kMidShift);
    const dc_mat& M = B ? P.mats[mid] : P.A;
    c.b0 = 0;
    c.len = (int)sl.steps;
    c.W = M.words + sl.base;
    c.Vv = static_cast<const V*>(M.vals) + sl.base;
    c.X = static_cast<const T*>(B ? P.xs[mid] : P.x);
    c.y = static_cast<T*>(B ? P.ys[mid] : P.y) + (int64_t)sl.brow * S + sl.meta;
}

// The chains: one warp per row, the row's elements in order (each word the
// absolute column), 512 at a time.  Lane l holds elements 16 l .. 16 l + 15 of
// a group: its segment of chain::sum_group, which adds the group in order
// without a chain of 512 additions (8.2 cycles each in FP64, 4 in f32).  Where
// that would not pay -- few segments, or a sum near zero that keeps crossing
// binades (chain::calm) -- or gives up, every lane adds the products in turn
// from shared memory.  A warp's rows form one stream of
// groups: while one is summed, the values and gathered x of the next are on
// their way into the other half of the warp's shared buffer (cp.async: they
// take no registers), and so are the words of the one after, whichever rows
// they belong to.  The places of a group past its row's end hold -0, which
// leaves any sum as it is.
// Bound by latency: one warp issues 408 instructions a group, 4.8 cycles each,
// and some 500 cycles more for a segment run again.  So the time depends on the
// values.  R-MAT scale 22 (chains and sliced rows together; us, against additions
// in turn): N(0,1) x U[-1,1] products onto a y that has grown 570 -> 370, onto
// y = 0 583 -> 580 to 627, all products positive onto y = 0 581 -> 415; f32 442 ->
// 310 to 340, 456 -> 402, 457 -> 368.  A lone row of 60,000: FP64 229 -> 90, onto 0
// 241 -> 183; f32 136 -> 81, 149 -> 162.  200 rows of 20,000: FP64 118 -> 87, onto 0
// 131 -> 139; f32 63 -> 66, 75 -> 88.  Rows of 260 to 600: 20 to 40% off either way.
// Without the two rules (segments, calm) a y = 0 took 604 to 635 on R-MAT scale
// 22 and 153 (f32 111) on the 200 rows.  Two CTAs an SM, or the sliced rows two,
// were slower on the 256-matrix batch (0.87 ms against 0.79).
template <int S, int VT, bool B>
__global__ void __launch_bounds__(32 * kChainWarps, kChainCtasPerSm) k_spmv_chains(dc_args P)
{
    using T = typename vt_of<VT>::T;
    using V = typename vt_of<VT>::V;
    constexpr int L = 16, G = kChainGroup;
    static_assert(G == 32 * L, "a segment a lane");
    // A group goes in turn at once where that is faster: up to kTurn segments (in
    // f32 an addition takes half as long), or where the sum is not kAbove binades
    // above the products (2 fewer: 200 rows of 20,000 onto 0 146 -> 152 us; 1 more:
    // onto a y that has grown 85 -> 92) unless the row's group before was settled
    // without a segment run again.
    constexpr int kTurn = sizeof(T) == 8 ? 12 : 19, kAbove = sizeof(T) == 8 ? 4 : 5;
    // segments 16 bytes apart, so that the lanes' 16-byte reads meet no bank twice
    constexpr int STX = L + 16 / (int)sizeof(T), STV = L + 16 / (int)sizeof(V);
    extern __shared__ __align__(16) uint8_t chain_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gw = blockIdx.x * kChainWarps + warp;
    const bool nothing = begin(P);
    if (gw >= P.warps)
        return;
    T* xb = reinterpret_cast<T*>(chain_smem + warp * chain_smem_warp<T, V>());
    V* vb = reinterpret_cast<V*>(xb + 2 * 32 * STX);
    const int64_t s1 = P.wbeg[gw + 1];
    chain_pos<T, V> cur{}, nxt{}, ahead;  // summed; copied; its words loaded
    ahead.si = P.wbeg[gw];
    if (nothing || ahead.si >= s1) {
        beside_end();
        return;
    }
    chain_at<S, B>(P, P.slices[ahead.si], ahead);
    dc_slice after = ahead.si + 1 < s1 ? P.slices[ahead.si + 1] : P.slices[ahead.si];
    uint32_t w[L];
    V vq[sizeof(V) < 4 ? L : 1];  // 2-byte values cannot be copied asynchronously
    auto load_words = [&] {
        const uint32_t* W = ahead.W + ahead.b0 + lane;
        const int left = ahead.len - ahead.b0 - lane;  // elements of the row from this lane's first on
        if (ahead.len - ahead.b0 >= G) {
#pragma unroll
            for (int j = 0; j < L; ++j)
                w[j] = ld_stream(W + 32 * j);
        } else {
#pragma unroll
            for (int j = 0; j < L; ++j)
                w[j] = 32 * j < left ? ld_stream(W + 32 * j) : 0u;
        }
    };
    auto advance = [&] {  // ahead: the next group (si = s1 at the end)
        ahead.b0 += G;
        if (ahead.b0 >= ahead.len && ++ahead.si < s1) {
            chain_at<S, B>(P, after, ahead);
            if (ahead.si + 1 < s1)
                after = P.slices[ahead.si + 1];
        }
    };
    // element 32 j + lane of a group is value lane % 16 of segment 2 j + lane / 16
    T* const x_to = xb + (lane / L) * STX + lane % L;
    V* const v_to = vb + (lane / L) * STV + lane % L;
    auto copy_one = [&](int half, int j, const V* Vv) {
        cp_async(x_to + half * 32 * STX + 2 * j * STX, nxt.X + w[j]);
        if constexpr (sizeof(V) >= 4)
            cp_async(v_to + half * 32 * STV + 2 * j * STV, Vv + 32 * j);
        else
            vq[j] = ld_stream(Vv + 32 * j);
    };
    auto copy = [&](int half) {  // nxt's values and x
        const V* Vv = nxt.Vv + nxt.b0 + lane;
        const int left = nxt.len - nxt.b0 - lane;
        if (nxt.len - nxt.b0 >= G) {
#pragma unroll
            for (int j = 0; j < L; ++j)
                copy_one(half, j, Vv);
        } else {
#pragma unroll
            for (int j = 0; j < L; ++j)
                if (32 * j < left)
                    copy_one(half, j, Vv);
        }
    };
    load_words();
    nxt = ahead;
    T y_nxt = P.fresh ? T(0) : *nxt.y;
    advance();
    copy(0);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (ahead.si < s1)
        load_words();
    T run = T(0);
    int half = 0, again = -1;  // again: segments run again in the row's group before (-1: added in turn)
#pragma unroll 1
    for (;;) {
        cur = nxt;
        if (cur.b0 == 0)
            run = y_nxt;
        if constexpr (sizeof(V) < 4) {
#pragma unroll
            for (int j = 0; j < L; ++j)
                v_to[half * 32 * STV + 2 * j * STV] = vq[j];
        }
        const bool more = ahead.si < s1;
        if (more) {
            nxt = ahead;
            if (nxt.b0 == 0)
                y_nxt = P.fresh ? T(0) : *nxt.y;
            advance();
            copy(half ^ 1);
            if (ahead.si < s1)
                load_words();
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;\n" ::: "memory");
        __syncwarp();  // every lane's copies of the current group have landed
        T p[L];
        T* xs = xb + half * 32 * STX + lane * STX;
        {
            V v[L];
            load16(xs, p);
            load16(vb + half * 32 * STV + lane * STV, v);
#pragma unroll
            for (int i = 0; i < L; ++i)
                p[i] = dmul(wide(v[i]), p[i]);
        }
        const int have = cur.len - cur.b0 - L * lane;  // of the lane's segment
        if (cur.len - cur.b0 < G) {
#pragma unroll
            for (int i = 0; i < L; ++i)
                p[i] = i < have ? p[i] : T(-0.0);
        }
        const int nseg = min(32, (cur.len - cur.b0 + L - 1) / L);
        if (cur.b0 == 0)
            again = -1;
        if (nseg <= kTurn || !(again == 0 || chain::calm<kAbove>(run, p)) ||
            (again = chain::sum_group<1, L>(run, p, lane)) < 0) {
            again = -1;
            store16(xs, p);
            __syncwarp();
            run = add_in_turn(run, xb + half * 32 * STX, STX, nseg);
        }
        if (cur.b0 + G >= cur.len && lane == 0)
            *cur.y = run;
        __syncwarp();  // this half is read before it is filled again
        if (!more)
            break;
        half ^= 1;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    beside_end();
}

// Y += A X over k > 1 columns (FP64).  A unit of blockIdx.x is C columns of G R
// of a slice's rows: 4 columns (one 32-byte sector of a row of X) of all 32, or
// 16 (a whole line) of a quarter.  Lane (g, h) = (lane / C, lane % C) keeps the
// sums of column h for rows g, g + G, g + 2 G, g + 3 G of them and reads those
// rows' words and values itself (C lanes the same address: a broadcast), so
// nothing is exchanged between lanes.  The next U steps' words and values are in
// flight while the gathers of the current ones return.  Every (row, column) sum
// adds its products in the row's column order from Y's value: column j of Y is
// bitwise the SpMV of column j of X.
// Beside chains, or where the longest slice takes longer than a warp's share of
// all, bound by the latency of the gathers: ten CTAs an SM and eight gathers a
// lane in flight.  R-MAT scale 18, 7 columns: passes of 4, 2
// and 1 columns, each with up to four gathers a lane in flight and column and
// value by shuffles, took 415 us of kernel time, this 78 us (with the chains:
// 1,305 -> 98 us; 88 with sixteen CTAs instead of 85); scale 10, no chains, 16
// columns 54 us against 87 the other way.
// Else bound by the lines a gather touches (4 columns a warp: eight a
// load, 16: two) and by the warps to hide them: sixteen CTAs (64 registers, 48 to
// 64 bytes spilled; with four columns a warp from kMmManySteps on: 3D Laplacian
// 60^3, 32 a warp at 8 columns, 34.5 us with ten and 38 with sixteen, 2D 700^2,
// 52, 56 and 46), and 16 columns a warp where there are as many, a step at a time.
// 3D Laplacian 120^3, 2 / 8 / 16 / 32 columns: 118 / 237 / 445 / 866 us with
// ten CTAs and 4 columns a warp, 93 / 183 / 335 / 653 so (113 / 256 / 353 / 1,527
// in passes of 2, 8, 16 and 32 columns before either).
template <int S, int C, int CTAS>
__global__ void __launch_bounds__(32 * kMmWarps, CTAS) k_spmm_slices(dc_args P)
{
    constexpr int R = kMmCols, U = C == kMmWide ? 1 : 2;  // rows a lane; steps a round
    constexpr int G = 32 / C, Q = C / R;                  // rows side by side; parts of a slice's 32 rows
    static_assert(G * R * Q == 32, "a unit of the grid is G R rows by C columns");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = G * R * (blockIdx.x % Q) + lane / C, h = blockIdx.x / Q * C + lane % C;
    const int gw = blockIdx.y * kMmWarps + warp;
    beside_begin();
    if (gw >= P.warps || h >= P.cols)
        return;
    const double* X = static_cast<const double*>(P.x) + h;
    double* Y = static_cast<double*>(P.y) + h;
    const int64_t s1 = P.wbeg[gw + 1];
#pragma unroll 1
    for (int64_t si = P.wbeg[gw]; si < s1; ++si) {
        const dc_slice sl = P.slices[si];
        const uint32_t* W = P.A.words + sl.base + g;
        const double* Vv = static_cast<const double*>(P.A.vals) + sl.base + g;
        int len[R];
        double* y[R];
        double acc[R];
        uint32_t col[R], w[U][R];
        double v[U][R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int r = g + G * i;
            const uint32_t rec = r < (int)sl.lanes ? P.A.lane[sl.meta + r] : 0u;
            len[i] = r < (int)sl.lanes ? (int)(rec & kLenMask) + 1 : 0;
            y[i] = Y + ((int64_t)sl.brow * S + (int64_t)(rec >> kLenBits)) * P.ldy;
            col[i] = 0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < R; ++i) {
                w[u][i] = u < len[i] ? __ldg(W + 32 * u + G * i) : 0u;
                v[u][i] = u < len[i] ? __ldg(Vv + 32 * u + G * i) : 0.0;
            }
#pragma unroll
        for (int i = 0; i < R; ++i)
            acc[i] = len[i] ? *y[i] : 0.0;
        // the longest of the warp's rows is its first (all 32 lanes are here where Q > 1)
        const int steps = Q > 1 ? __shfl_sync(0xffffffffu, len[0], 0) : (int)sl.steps;
#pragma unroll 1
        for (int k0 = 0; k0 < steps; k0 += U) {
            double x[U][R];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    col[i] += w[u][i];
                    x[u][i] = k0 + u < len[i] ? __ldg(X + (int64_t)col[i] * P.ldx) : 0.0;
                    w[u][i] = k0 + U + u < len[i] ? __ldg(W + 32 * (k0 + U + u) + G * i) : 0u;
                }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    if (k0 + u < len[i])
                        acc[i] = dadd(acc[i], dmul(v[u][i], x[u][i]));
                    v[u][i] = k0 + U + u < len[i] ? __ldg(Vv + 32 * (k0 + U + u) + G * i) : 0.0;
                }
        }
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (len[i])
                *y[i] = acc[i];
    }
    beside_end();
}

// Y += A X over k > 1 columns, the chains: one row and kMmCols = 4 columns a
// warp, 128 elements at a time.  Lane (g, h) holds elements 16 g .. 16 g + 15
// for column h: its segment of column h's chain in chain::sum_group (four
// chains of eight segments at once).  The words and values are loaded by the
// quad (lane (g, h) elements 16 g + 4 j + h) and handed round by shuffles, so
// that the 16 gathers of X a lane has in flight are one sector each for the
// quad.  Where sum_group gives up, the segments are added one after another.
// R-MAT scale 18, 7 columns: three passes with eight gathers in flight a warp
// step took 1,236 us of kernel time, this 88 us.
template <int S>
__global__ void __launch_bounds__(32 * kChainWarps, kChainCtasPerSm) k_spmm_chains(dc_args P)
{
    constexpr int L = 16, G = 8 * L, Q = L / kMmCols;
    constexpr unsigned full = 0xffffffffu;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane / kMmCols, q = lane % kMmCols, h = blockIdx.x * kMmCols + q;
    const int gw = blockIdx.y * kChainWarps + warp;
    beside_begin();
    if (gw >= P.warps)
        return;
    const bool live = h < P.cols;  // the last columns' warps may hold fewer than four
    const double* X = static_cast<const double*>(P.x) + (live ? h : 0);
    double* Y = static_cast<double*>(P.y) + (live ? h : 0);
    const int64_t s1 = P.wbeg[gw + 1];
#pragma unroll 1
    for (int64_t si = P.wbeg[gw]; si < s1; ++si) {
        const dc_slice sl = P.slices[si];
        const uint32_t* W = P.A.words + sl.base;
        const double* Vv = static_cast<const double*>(P.A.vals) + sl.base;
        const int len = (int)sl.steps, e0 = L * g + q;
        double* y = Y + ((int64_t)sl.brow * S + sl.meta) * P.ldy;
        uint32_t w[Q];
        double v[Q], x[L], run = *y;
#pragma unroll
        for (int j = 0; j < Q; ++j)
            w[j] = ld_stream(W + min(e0 + kMmCols * j, len - 1));
#pragma unroll
        for (int i = 0; i < L; ++i)
            x[i] = __ldg(X + (int64_t)__shfl_sync(full, w[i / kMmCols], kMmCols * g + i % kMmCols) * P.ldx);
#pragma unroll
        for (int j = 0; j < Q; ++j) {
            v[j] = ld_stream(Vv + min(e0 + kMmCols * j, len - 1));
            w[j] = ld_stream(W + min(e0 + G + kMmCols * j, len - 1));
        }
#pragma unroll 1
        for (int b0 = 0; b0 < len; b0 += G) {
            double p[L];
#pragma unroll
            for (int i = 0; i < L; ++i) {
                const double vi = __shfl_sync(full, v[i / kMmCols], kMmCols * g + i % kMmCols);
                p[i] = b0 + L * g + i < len ? dmul(vi, x[i]) : -0.0;
                x[i] = __ldg(X + (int64_t)__shfl_sync(full, w[i / kMmCols], kMmCols * g + i % kMmCols) * P.ldx);
            }
#pragma unroll
            for (int j = 0; j < Q; ++j) {
                v[j] = ld_stream(Vv + min(b0 + G + e0 + kMmCols * j, len - 1));
                w[j] = ld_stream(W + min(b0 + 2 * G + e0 + kMmCols * j, len - 1));
            }
            if (chain::sum_group<kMmCols, L>(run, p, lane) < 0) {
                const int nseg = min(8, (len - b0 + L - 1) / L);
#pragma unroll 1
                for (int s = 0; s < nseg; ++s) {
#pragma unroll
                    for (int i = 0; i < L; ++i)
                        run = g == s ? dadd(run, p[i]) : run;
                    run = __shfl_sync(full, run, kMmCols * s + q);
                }
            }
        }
        if (g == 0 && live)
            *y = run;
    }
    beside_end();
}

// --------------------------------------------------------------- preparation

// Block rows the slices serve: no dense tile (its stored zeros would need
// words too), and no bitmap tile (the ring kernel's bitmap walk reads a bit
// per position where a slice reads a word per element), at most `avg`
// elements per tile on average, or more than kRingTilesMax tiles (one CTA of
// the ring kernel sums a whole block row, so a block row of very many tiles
// would keep one SM busy long after the rest).
// fbytes[k]: the block row's share of the format bytes (its brow_ptr entry,
// its tiles' headers, payloads and values).
__global__ void k_dc_classify(int64_t nr, const uint32_t* __restrict__ rows, tiles_view A, float avg, int vsize,
                              uint8_t* __restrict__ ok, int64_t* __restrict__ elems, int64_t* __restrict__ fbytes)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < nr; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t I = rows[k], t0 = A.brow_ptr[I], t1 = A.brow_ptr[I + 1];
        bool sparse = true, bitmap = false;
        for (int64_t t = t0; t < t1 && sparse; ++t) {
            sparse = A.tile_scheme[t] != ABHSF_SCHEME_DENSE;
            bitmap = bitmap || A.tile_scheme[t] == ABHSF_SCHEME_BITMAP;
        }
        const int64_t e = A.tile_val_off[t1] - A.tile_val_off[t0];
        ok[k] = sparse && ((double)e <= (double)avg * (double)(t1 - t0) || t1 - t0 > kRingTilesMax || !bitmap) ? 1 : 0;
        elems[k] = e;
        fbytes[k] = 8 + (t1 - t0) * (4 + 4 + 1 + 8 + 8) + (A.tile_idx_off[t1] - A.tile_idx_off[t0]) + vsize * e;
    }
}

__device__ __forceinline__ int64_t brow_of_tile(const int64_t* brow_ptr, int64_t M, int64_t t)
{
    int64_t lo = 0, hi = M;  // largest I with brow_ptr[I] <= t
    while (hi - lo > 1) {
        const int64_t mid = (lo + hi) / 2;
        if (brow_ptr[mid] <= t)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// A warp's lanes over the z elements of one tile, in any order: f(e, row,
// column) for element e of the tile, its row and column in the tile.
template <typename F>
__device__ __forceinline__ void for_elements(const tiles_view& A, int64_t t, int64_t z, int s, int lg, int lane, F&& f)
{
    const uint8_t* pay = A.payload + A.tile_idx_off[t];
    const uint16_t* w16 = reinterpret_cast<const uint16_t*>(pay);
    const int sch = A.tile_scheme[t];
    if (sch == ABHSF_SCHEME_CSR) {
        for (int64_t e = lane; e < z; e += 32) {
            int lo = 0, hi = s - 1;  // the first row whose end is beyond e
            while (lo < hi) {
                const int mid = (lo + hi) / 2;
                if (w16[mid] > e)
                    hi = mid;
                else
                    lo = mid + 1;
            }
            f(e, lo, (int)pay[2 * s + e]);
        }
    } else if (sch == ABHSF_SCHEME_BITMAP) {
        const uint64_t* bm = reinterpret_cast<const uint64_t*>(pay);
        const int words = s * s / 64;
        int64_t done = 0;
        for (int w0 = 0; w0 < words; w0 += 32) {
            const int wi = w0 + lane;
            uint64_t bits = wi < words ? bm[wi] : 0;
            const int cnt = __popcll(bits);
            int inc = cnt;
#pragma unroll
            for (int d = 1; d < 32; d *= 2) {
                const int v = __shfl_up_sync(0xffffffffu, inc, d);
                if (lane >= d)
                    inc += v;
            }
            int64_t e = done + inc - cnt;
            for (; bits; bits &= bits - 1, ++e) {
                const int bit = wi * 64 + __ffsll((long long)bits) - 1;
                f(e, bit >> lg, bit & (s - 1));
            }
            done += __shfl_sync(0xffffffffu, inc, 31);
        }
    } else {
        for (int64_t e = lane; e < z; e += 32)
            f(e, w16[e] >> lg, w16[e] & (s - 1));
    }
}

// Elements per row of the slice block rows (sidx[I] >= 0): cnt[sidx * s + lrow].
// A tile a warp (a thread a tile took 0.7 ms to expand 1M elements in tiles of
// 256, whose elements it visited one after another).
__global__ void k_dc_row_counts(int64_t T, tiles_view A, int s, int lg, const int32_t* __restrict__ sidx,
                                unsigned int* __restrict__ cnt)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
    for (int64_t t = blockIdx.x * (int64_t)(blockDim.x / 32) + threadIdx.x / 32; t < T; t += warps) {
        const int k = sidx[brow_of_tile(A.brow_ptr, A.M, t)];
        if (k < 0)
            continue;
        unsigned int* c = cnt + (int64_t)k * s;
        const int64_t z = A.tile_val_off[t + 1] - A.tile_val_off[t];
        for_elements(A, t, z, s, lg, lane, [&](int64_t, int lr, int) { atomicAdd(c + lr, 1u); });
    }
}

// Every element of the slice block rows at its place in element order (the
// block rows ascending, each in format order): its key (slice block row * s
// + row), its column and its value index.
__global__ void k_dc_expand(int64_t T, tiles_view A, int s, int lg, const int32_t* __restrict__ sidx,
                            const int64_t* __restrict__ ebase, uint32_t* __restrict__ key, uint32_t* __restrict__ pos,
                            uint32_t* __restrict__ colv, int64_t* __restrict__ vidx)
{
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
    for (int64_t t = blockIdx.x * (int64_t)(blockDim.x / 32) + threadIdx.x / 32; t < T; t += warps) {
        const int64_t I = brow_of_tile(A.brow_ptr, A.M, t);
        const int k = sidx[I];
        if (k < 0)
            continue;
        const int64_t v0 = A.tile_val_off[t], z = A.tile_val_off[t + 1] - v0;
        const int64_t e0 = ebase[k] + (v0 - A.tile_val_off[A.brow_ptr[I]]);
        const uint64_t c0 = (uint64_t)A.tile_col[t] * (uint64_t)s;
        for_elements(A, t, z, s, lg, lane, [&](int64_t e, int lr, int lc) {
            const int64_t q = e0 + e;
            key[q] = (uint32_t)((int64_t)k * s + lr);
            pos[q] = (uint32_t)q;
            colv[q] = (uint32_t)(c0 + (uint64_t)lc);
            vidx[q] = v0 + e;
        });
    }
}

// The sliced rows (1 .. kChainMin elements), and the chains, among the ns * s
// rows.
struct is_sliced {
    const unsigned int* cnt;
    __device__ bool operator()(uint32_t q) const { return cnt[q] >= 1u && cnt[q] <= (unsigned)kChainMin; }
};
struct is_chain {
    const unsigned int* cnt;
    __device__ bool operator()(uint32_t q) const { return cnt[q] > (unsigned)kChainMin; }
};

// Index of the segment (seg[0 .. n]: block-row boundaries) block row I lies in.
__device__ __forceinline__ int segment_of(const int64_t* seg, int n, int64_t I)
{
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (seg[mid] <= I)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// Sort keys of the sliced rows: segment, then length, longest first.
__global__ void k_dc_row_keys(int64_t nS, const uint32_t* __restrict__ q, const unsigned int* __restrict__ cnt,
                              const uint32_t* __restrict__ sel, const int64_t* __restrict__ seg, int nseg, int lg,
                              uint32_t* __restrict__ key)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nS; i += (int64_t)gridDim.x * blockDim.x)
        key[i] = (uint32_t)segment_of(seg, nseg, sel[q[i] >> lg]) << kLenBits | ((unsigned)kChainMin - cnt[q[i]]);
}

// begin[g]: the first sorted row of segment g (g = 0 .. nseg).
__global__ void k_dc_segment_begin(int64_t nS, const uint32_t* __restrict__ key, int nseg, int64_t* __restrict__ begin)
{
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g <= nseg; g += gridDim.x * blockDim.x) {
        int64_t lo = 0, hi = nS;
        while (lo < hi) {
            const int64_t mid = (lo + hi) / 2;
            if ((int64_t)(key[mid] >> kLenBits) < g)
                lo = mid + 1;
            else
                hi = mid;
        }
        begin[g] = lo;
    }
}

// Steps of every slice: the length of its first row.  first[g]: the first
// slice of segment g.
__global__ void k_dc_steps(int64_t nS, const uint32_t* __restrict__ key, const int64_t* __restrict__ begin,
                           const int64_t* __restrict__ first, uint32_t* __restrict__ steps)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nS; i += (int64_t)gridDim.x * blockDim.x) {
        const int g = (int)(key[i] >> kLenBits);
        const int64_t at = i - begin[g];
        if (at % 32 == 0)
            steps[first[g] + at / 32] = (uint32_t)kChainMin - (key[i] & kLenMask);
    }
}

// Lane record and first slot of every sliced row.
__global__ void k_dc_lanes(int64_t nS, const uint32_t* __restrict__ key, const uint32_t* __restrict__ q,
                           const uint32_t* __restrict__ sel, const int64_t* __restrict__ seg,
                           const int64_t* __restrict__ begin, const int64_t* __restrict__ first,
                           const int64_t* __restrict__ base, int lg, uint32_t* __restrict__ lane,
                           int64_t* __restrict__ slot0)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nS; i += (int64_t)gridDim.x * blockDim.x) {
        const int g = (int)(key[i] >> kLenBits);
        const int64_t at = i - begin[g], j = first[g] + at / 32;
        const uint32_t len = (uint32_t)kChainMin - (key[i] & kLenMask), r = q[i];
        const int64_t off = (((int64_t)sel[r >> lg] - seg[g]) << lg) + (r & ((1u << lg) - 1u));
        lane[32 * j + at % 32] = (uint32_t)off << kLenBits | (len - 1u);
        slot0[r] = base[j] + at % 32;
    }
}

__global__ void k_dc_gather(int64_t n, const uint32_t* __restrict__ q, const unsigned int* __restrict__ cnt,
                            unsigned int* __restrict__ out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = cnt[q[i]];
}

__global__ void k_dc_chain_slots(int64_t n, const uint32_t* __restrict__ q, const int64_t* __restrict__ slot,
                                 int64_t* __restrict__ slot0)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        slot0[q[i]] = slot[i];
}

// Words and values at their slots, from the elements sorted row by row (each
// row's elements in column order): the q-th sorted element is element
// q - rstart[key] of its row.
template <typename V>
__global__ void k_dc_emit(int64_t E, const uint32_t* __restrict__ key, const uint32_t* __restrict__ pos,
                          const uint32_t* __restrict__ colv, const int64_t* __restrict__ vidx,
                          const int64_t* __restrict__ rstart, const int64_t* __restrict__ slot0,
                          const unsigned int* __restrict__ cnt, const V* __restrict__ values,
                          uint32_t* __restrict__ words, V* __restrict__ vals)
{
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < E; q += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t kr = key[q];
        const int64_t rank = q - rstart[kr];
        const uint32_t c = colv[pos[q]];
        const bool ch = cnt[kr] > (unsigned)kChainMin;
        const int64_t slot = slot0[kr] + (ch ? rank : 32 * rank);
        words[slot] = (ch || rank == 0) ? c : c - colv[pos[q - 1]];
        vals[slot] = values[vidx[pos[q]]];
    }
}

inline unsigned grid_of(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 8192)); }

// Warps of a launch: the chains one CTA per SM; the sliced rows every
// resident CTA, less one per SM when chains run beside them (their CTA needs
// the registers), or one CTA per SM when they run beside the ring kernel
// (which leaves an SM the registers and warps of one such CTA).
int stream_grid_warps(int64_t items, bool chains, bool beside_chains, bool beside_ring)
{
    int dev = 0, nsm = 0;
    ABHSF_CUDA(cudaGetDevice(&dev));
    ABHSF_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
    const int ctas = beside_ring ? 1 : beside_chains ? kSliceGridPerSm : kCtasPerSm;
    const int64_t full = chains ? (int64_t)nsm * kChainGridPerSm * kChainWarps : (int64_t)nsm * ctas * kWarpsPerCta;
    return (int)std::max<int64_t>(1, std::min<int64_t>(full, items));
}

// Time a slice takes, for the deal: a sliced one walks its longest row, a
// chain takes about 2,400 cycles a group while its sum is near zero (where
// groups are added in turn more often) and 1,700 later, and its first loads.
inline uint64_t slice_weight(const abhsf_matrix::dc_slice_host& p)
{
    if (!p.chain)
        return 32ull * p.steps + 64u;
    const uint64_t groups = (p.steps + kChainGroup - 1) / kChainGroup;
    return 1700u * groups + 700u * std::min<uint64_t>(groups, 8) + 500u;
}

}  // namespace

// Longest-processing-time deal of the sliced rows (or the chains) of several
// matrices (block rows in [brow_lo, brow_hi) only) over the warps of one
// launch.
void deal_slices(const std::vector<const abhsf_matrix*>& mats, dbuf<uint8_t>& sched, dbuf<int64_t>& wbeg_d,
                 int& warps_out, cudaStream_t st, int64_t brow_lo, int64_t brow_hi, int kind, bool beside_ring)
{
    const bool chains = kind != kDealSliced;
    struct item {
        uint64_t w;
        uint32_t mid;
        uint32_t k;
    };
    std::vector<item> items;
    bool other = false;  // a slice of the other kind in the range
    for (size_t i = 0; i < mats.size(); ++i) {
        const auto& ps = mats[i]->dc_host;
        for (size_t k = 0; k < ps.size(); ++k)
            if ((int64_t)ps[k].brow >= brow_lo && (int64_t)ps[k].brow < brow_hi) {
                if (ps[k].chain != chains)
                    other = true;
                else
                    items.push_back(item{slice_weight(ps[k]), (uint32_t)i, (uint32_t)k});
            }
    }
    warps_out = 0;
    if (items.empty())
        return;
    const int W = stream_grid_warps((int64_t)items.size(), chains, !chains && other, beside_ring);
    std::stable_sort(items.begin(), items.end(), [](const item& a, const item& b) { return a.w > b.w; });
    using load_t = std::pair<uint64_t, int>;
    std::priority_queue<load_t, std::vector<load_t>, std::greater<load_t>> heap;
    for (int w = 0; w < W; ++w)
        heap.push({0, w});
    std::vector<std::vector<uint32_t>> per(W);
    for (uint32_t j = 0; j < items.size(); ++j) {
        load_t top = heap.top();
        heap.pop();
        per[top.second].push_back(j);
        heap.push({top.first + items[j].w, top.second});
    }
    std::vector<dc_slice> out;
    out.reserve(items.size());
    std::vector<int64_t> wbeg(W + 1, 0);
    for (int w = 0; w < W; ++w) {
        wbeg[w] = (int64_t)out.size();
        for (uint32_t j : per[w]) {  // heaviest first within the warp, too
            const auto& h = mats[items[j].mid]->dc_host[items[j].k];
            dc_slice p;
            p.base = h.base;
            p.meta = h.meta;
            p.brow = h.brow;
            p.steps = h.steps;
            p.lanes = h.lanes;
            p.geo = (h.chain ? kChain : 0u) | items[j].mid << kMidShift;
            out.push_back(p);
        }
    }
    wbeg[W] = (int64_t)out.size();
    // (a second deal of the same slices fits the first one's memory)
    if (sched.size() < out.size() * sizeof(dc_slice))
        sched.alloc(out.size() * sizeof(dc_slice));
    if (wbeg_d.size() < (size_t)W + 1)
        wbeg_d.alloc(W + 1);
    ABHSF_CUDA(cudaMemcpyAsync(sched.get(), out.data(), out.size() * sizeof(dc_slice), cudaMemcpyHostToDevice, st));
    ABHSF_CUDA(cudaMemcpyAsync(wbeg_d.get(), wbeg.data(), (W + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    ABHSF_CUDA(cudaStreamSynchronize(st));
    warps_out = W;
}

// Block-row boundaries of the ranges whose sliced rows may share a slice:
// the kHostChunks parts the host-memory SpMV copies and sums one after
// another (a part's slices must not reach into the next), each cut into
// pieces of at most 2^24 rows (the row offset a lane record holds).
std::vector<int64_t> slice_segments(int64_t M, int s)
{
    const int64_t piece = std::max<int64_t>(1, (int64_t(1) << (32 - kLenBits)) / s);
    std::vector<int64_t> b{0};
    for (int c = 1; c <= kHostChunks; ++c) {
        const int64_t e = M * c / kHostChunks;
        while (e - b.back() > piece)
            b.push_back(b.back() + piece);
        if (e > b.back())
            b.push_back(e);
    }
    return b;
}

// The slices of a prepared matrix: which non-empty block rows they serve
// (dc_tree_flag, by tree-row position), their words, values and lane
// records, and the matrix's own schedule.  avg <= 0 leaves every block row
// to the ring.
void prepare_stream(abhsf_matrix& a, float avg, cudaStream_t st)
{
    a.dc_host.clear();
    a.dc_tree_flag.assign((size_t)a.tree_nrows, 0);
    a.dc_warps = a.dc_cwarps = 0;
    a.dc_every_row = false;
    a.dc_elements = a.dc_rows = a.dc_slots = a.dc_lane_records = a.dc_steps = a.dc_longest = 0;
    const int s = a.s, lg = a.lg;
    if (avg <= 0.f || a.tree_nrows == 0 || a.sum_order != ABHSF_SUM_REFERENCE || (uint64_t)a.n > (uint64_t(1) << 32))
        return;
    const int64_t nr = a.tree_nrows;
    scratch<uint8_t> ok(nr, st);
    scratch<int64_t> elems(nr, st), fbytes(nr, st);
    const int vsize = (int)value_size(a.value_type);
    k_dc_classify<<<grid_of(nr), 256, 0, st>>>(nr, a.tree_rows.get(), a.view(), avg, vsize, ok.get(), elems.get(),
                                                fbytes.get());
    ABHSF_CUDA(cudaGetLastError());
    std::vector<uint8_t> okh(nr);
    std::vector<int64_t> eh(nr), fh(nr);
    std::vector<uint32_t> rows(nr);
    ABHSF_CUDA(cudaMemcpyAsync(okh.data(), ok.get(), nr, cudaMemcpyDeviceToHost, st));
    ABHSF_CUDA(cudaMemcpyAsync(eh.data(), elems.get(), nr * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    ABHSF_CUDA(cudaMemcpyAsync(fh.data(), fbytes.get(), nr * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    ABHSF_CUDA(cudaMemcpyAsync(rows.data(), a.tree_rows.get(), nr * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    ABHSF_CUDA(cudaStreamSynchronize(st));
    // slice block rows in ascending block-row order
    std::vector<int64_t> tree_at(a.M, -1);
    for (int64_t k = 0; k < nr; ++k)
        if (okh[k])
            tree_at[rows[k]] = k;
    std::vector<std::pair<uint32_t, int64_t>> sel;  // (block row, tree position)
    for (int64_t I = 0; I < a.M; ++I)
        if (tree_at[I] >= 0)
            sel.push_back({(uint32_t)I, tree_at[I]});
    const int64_t ns = (int64_t)sel.size();
    int64_t E = 0;
    for (auto& p : sel)
        E += eh[p.second];
    if (ns == 0 || E == 0 || E >= (int64_t(1) << 31) || ns * s >= (int64_t(1) << 32))
        return;
    std::vector<int32_t> sidx_h(a.M, -1);
    std::vector<int64_t> ebase(ns + 1, 0);
    for (int64_t k = 0; k < ns; ++k) {
        sidx_h[sel[k].first] = (int32_t)k;
        ebase[k + 1] = ebase[k] + eh[sel[k].second];
    }
    scratch<int32_t> sidx(a.M, st);
    scratch<unsigned int> cnt(ns * s, st);
    ABHSF_CUDA(cudaMemcpyAsync(sidx.get(), sidx_h.data(), a.M * sizeof(int32_t), cudaMemcpyHostToDevice, st));
    ABHSF_CUDA(cudaMemsetAsync(cnt.get(), 0, ns * s * sizeof(unsigned int), st));
    k_dc_row_counts<<<grid_of(8 * a.T), 256, 0, st>>>(a.T, a.view(), s, lg, sidx.get(), cnt.get());
    ABHSF_CUDA(cudaGetLastError());
    // Sliced rows: per segment (slice_segments), the rows of up to kChainMin
    // elements by length, longest first, then ascending row, in groups of 32 --
    // rows of one length class share a slice whatever their block row, so that
    // its lanes run out together.  Longer rows are chains, per block row, longest
    // first, then ascending row; a segment's chains come before its slices.
    // The rows are ordered on the device (871k rows of the tiled mixture took 8
    // ms on the host); the host adds up the slots, one step a slice.
    const int64_t R = ns * s;
    const std::vector<int64_t> seg = slice_segments(a.M, s);
    const int nseg = (int)seg.size() - 1;
    std::vector<uint32_t> selrow_h(ns);
    for (int64_t k = 0; k < ns; ++k)
        selrow_h[k] = sel[k].first;
    const int64_t L = std::min(R, E);  // rows with elements, at most: far fewer than R where block rows hold a few
    scratch<uint32_t> selrow(ns, st), sq(L, st), sq2(L, st), cq(E / kChainMin + 1, st), skey(L, st), skey2(L, st);
    scratch<int64_t> seg_d(nseg + 1, st), begin_d(nseg + 1, st), first_d(nseg + 1, st), found(2, st), rstart(R + 1, st),
        slot0(R, st);
    ABHSF_CUDA(cudaMemcpyAsync(selrow.get(), selrow_h.data(), ns * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    ABHSF_CUDA(cudaMemcpyAsync(seg_d.get(), seg.data(), (nseg + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    std::vector<int64_t> begin(nseg + 1, 0), first(nseg + 1, 0);
    std::vector<uint32_t> chain_q;
    std::vector<unsigned int> chain_len;
    int64_t nS = 0;
    {
        const thrust::counting_iterator<uint32_t> all(0);
        size_t b1 = 0, b2 = 0, b3 = 0, b4 = 0;
        int kb = kLenBits;
        while ((int64_t(1) << (kb - kLenBits)) < nseg)
            ++kb;
        ABHSF_CUDA(cub::DeviceSelect::If(nullptr, b1, all, sq.get(), found.get(), R, is_sliced{cnt.get()}, st));
        ABHSF_CUDA(cub::DeviceSelect::If(nullptr, b2, all, cq.get(), found.get() + 1, R, is_chain{cnt.get()}, st));
        ABHSF_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b3, skey.get(), skey2.get(), sq.get(), sq2.get(), L, 0, kb,
                                                   st));
        ABHSF_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, b4, cnt.get(), rstart.get(), R, st));
        scratch<uint8_t> tmp(std::max(std::max(b1, b2), std::max(b3, b4)), st);
        ABHSF_CUDA(cub::DeviceSelect::If(tmp.get(), b1, all, sq.get(), found.get(), R, is_sliced{cnt.get()}, st));
        ABHSF_CUDA(cub::DeviceSelect::If(tmp.get(), b2, all, cq.get(), found.get() + 1, R, is_chain{cnt.get()}, st));
        ABHSF_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), b4, cnt.get(), rstart.get(), R, st));
        int64_t n2[2] = {0, 0};
        ABHSF_CUDA(cudaMemcpyAsync(n2, found.get(), sizeof(n2), cudaMemcpyDeviceToHost, st));
        ABHSF_CUDA(cudaStreamSynchronize(st));
        nS = n2[0];
        if (nS) {
            k_dc_row_keys<<<grid_of(nS), 256, 0, st>>>(nS, sq.get(), cnt.get(), selrow.get(), seg_d.get(), nseg, lg,
                                                       skey.get());
            ABHSF_CUDA(cudaGetLastError());
            ABHSF_CUDA(cub::DeviceRadixSort::SortPairs(tmp.get(), b3, skey.get(), skey2.get(), sq.get(), sq2.get(), nS,
                                                       0, kb, st));
            k_dc_segment_begin<<<1, 256, 0, st>>>(nS, skey2.get(), nseg, begin_d.get());
            ABHSF_CUDA(cudaGetLastError());
            ABHSF_CUDA(cudaMemcpyAsync(begin.data(), begin_d.get(), (nseg + 1) * sizeof(int64_t),
                                       cudaMemcpyDeviceToHost, st));
        }
        if (n2[1]) {
            chain_q.resize(n2[1]);
            ABHSF_CUDA(cudaMemcpyAsync(chain_q.data(), cq.get(), n2[1] * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
            scratch<unsigned int> cl(n2[1], st);
            k_dc_gather<<<grid_of(n2[1]), 256, 0, st>>>(n2[1], cq.get(), cnt.get(), cl.get());
            ABHSF_CUDA(cudaGetLastError());
            chain_len.resize(n2[1]);
            ABHSF_CUDA(cudaMemcpyAsync(chain_len.data(), cl.get(), n2[1] * sizeof(unsigned int),
                                       cudaMemcpyDeviceToHost, st));
            ABHSF_CUDA(cudaStreamSynchronize(st));
        }
        ABHSF_CUDA(cudaStreamSynchronize(st));
    }
    int64_t nslices = 0;
    for (int g = 0; g < nseg; ++g) {
        first[g] = nslices;
        nslices += (begin[g + 1] - begin[g] + 31) / 32;
    }
    first[nseg] = nslices;
    std::vector<uint32_t> steps(nslices);
    if (nS) {
        scratch<uint32_t> steps_d(nslices, st);
        ABHSF_CUDA(cudaMemcpyAsync(first_d.get(), first.data(), (nseg + 1) * sizeof(int64_t), cudaMemcpyHostToDevice,
                                   st));
        k_dc_steps<<<grid_of(nS), 256, 0, st>>>(nS, skey2.get(), begin_d.get(), first_d.get(), steps_d.get());
        ABHSF_CUDA(cudaGetLastError());
        ABHSF_CUDA(cudaMemcpyAsync(steps.data(), steps_d.get(), nslices * sizeof(uint32_t), cudaMemcpyDeviceToHost,
                                   st));
        ABHSF_CUDA(cudaStreamSynchronize(st));
    }
    std::vector<size_t> corder(chain_q.size());  // chains by block row, then length (longest first), then row
    for (size_t i = 0; i < corder.size(); ++i)
        corder[i] = i;
    std::stable_sort(corder.begin(), corder.end(), [&](size_t x, size_t y) {
        const uint32_t kx = chain_q[x] >> lg, ky = chain_q[y] >> lg;
        return kx != ky ? kx < ky : chain_len[x] > chain_len[y];
    });
    auto& SL = a.dc_host;
    SL.reserve(nslices + chain_q.size());
    std::vector<int64_t> base(nslices), chain_slot(chain_q.size());
    int64_t slots = 0;
    size_t c = 0;
    for (int g = 0; g < nseg; ++g) {
        for (; c < corder.size(); ++c) {
            const uint32_t q = chain_q[corder[c]];
            if ((int64_t)selrow_h[q >> lg] >= seg[g + 1])
                break;
            abhsf_matrix::dc_slice_host h;
            h.base = slots;
            h.meta = q & (uint32_t)(s - 1);
            h.brow = selrow_h[q >> lg];
            h.steps = chain_len[corder[c]];
            h.lanes = 1;
            h.chain = true;
            chain_slot[corder[c]] = slots;
            slots += h.steps;
            SL.push_back(h);
        }
        for (int64_t j = first[g]; j < first[g + 1]; ++j) {
            abhsf_matrix::dc_slice_host h;
            h.base = slots;
            h.meta = 32 * j;
            h.brow = (uint32_t)seg[g];
            h.steps = steps[j];
            h.lanes = (uint32_t)std::min<int64_t>(32, begin[g + 1] - begin[g] - 32 * (j - first[g]));
            h.chain = false;
            base[j] = slots;
            slots += 32 * (int64_t)h.steps;
            SL.push_back(h);
        }
    }
    a.dc_lane.alloc(std::max<int64_t>(32 * nslices, 1));
    if (nS) {
        scratch<int64_t> base_d(nslices, st);
        ABHSF_CUDA(cudaMemcpyAsync(base_d.get(), base.data(), nslices * sizeof(int64_t), cudaMemcpyHostToDevice, st));
        ABHSF_CUDA(cudaMemsetAsync(a.dc_lane.get(), 0, 32 * nslices * sizeof(uint32_t), st));
        k_dc_lanes<<<grid_of(nS), 256, 0, st>>>(nS, skey2.get(), sq2.get(), selrow.get(), seg_d.get(), begin_d.get(),
                                                first_d.get(), base_d.get(), lg, a.dc_lane.get(), slot0.get());
        ABHSF_CUDA(cudaGetLastError());
        ABHSF_CUDA(cudaStreamSynchronize(st));
    }
    if (!chain_q.empty()) {
        scratch<int64_t> slot_d(chain_q.size(), st);
        ABHSF_CUDA(cudaMemcpyAsync(slot_d.get(), chain_slot.data(), chain_q.size() * sizeof(int64_t),
                                   cudaMemcpyHostToDevice, st));
        k_dc_chain_slots<<<grid_of(chain_q.size()), 256, 0, st>>>((int64_t)chain_q.size(), cq.get(), slot_d.get(),
                                                                  slot0.get());
        ABHSF_CUDA(cudaGetLastError());
        ABHSF_CUDA(cudaStreamSynchronize(st));
    }
    // the elements row by row: sort by (block row, row), stable in format order
    scratch<uint32_t> key(E, st), pos(E, st), key2(E, st), pos2(E, st), colv(E, st);
    scratch<int64_t> vidx(E, st), ebase_d(ns + 1, st);
    ABHSF_CUDA(cudaMemcpyAsync(ebase_d.get(), ebase.data(), (ns + 1) * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    k_dc_expand<<<grid_of(8 * a.T), 256, 0, st>>>(a.T, a.view(), s, lg, sidx.get(), ebase_d.get(), key.get(), pos.get(),
                                              colv.get(), vidx.get());
    ABHSF_CUDA(cudaGetLastError());
    int bits = 1;
    while (bits < 32 && (int64_t(1) << bits) < ns * s)
        ++bits;
    size_t tb = 0;
    ABHSF_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, key.get(), key2.get(), pos.get(), pos2.get(), (int)E, 0,
                                               bits, st));
    {
        scratch<uint8_t> tmp(tb, st);
        ABHSF_CUDA(cub::DeviceRadixSort::SortPairs(tmp.get(), tb, key.get(), key2.get(), pos.get(), pos2.get(),
                                                   (int)E, 0, bits, st));
        ABHSF_CUDA(cudaStreamSynchronize(st));  // before tmp goes
    }
    const size_t vs = value_size(a.value_type);
    a.dc_words.alloc(slots);
    a.dc_vals.alloc(slots * vs);
    ABHSF_CUDA(cudaMemsetAsync(a.dc_words.get(), 0, slots * sizeof(uint32_t), st));
    ABHSF_CUDA(cudaMemsetAsync(a.dc_vals.get(), 0, slots * vs, st));
    auto emit = [&](auto tag) {
        using V = decltype(tag);
        k_dc_emit<V><<<grid_of(E), 256, 0, st>>>(E, key2.get(), pos2.get(), colv.get(), vidx.get(), rstart.get(),
                                                  slot0.get(), cnt.get(),
                                                  reinterpret_cast<const V*>(a.values.get()), a.dc_words.get(),
                                                  reinterpret_cast<V*>(a.dc_vals.get()));
    };
    if (vs == 8)
        emit(double{});
    else if (vs == 4)
        emit(float{});
    else
        emit(uint16_t{});
    ABHSF_CUDA(cudaGetLastError());
    ABHSF_CUDA(cudaStreamSynchronize(st));
    int64_t moved = 0;  // format bytes of the block rows the slices take over
    for (int64_t k = 0; k < ns; ++k) {
        a.dc_tree_flag[sel[k].second] = 1;
        moved += fh[sel[k].second];
    }
    a.stats.spmv_bytes = a.stats.format_bytes - moved + E * (int64_t)(sizeof(uint32_t) + vs) +
                         (int64_t)SL.size() * (int64_t)sizeof(dc_slice) + nS * (int64_t)sizeof(uint32_t);  // a lane record a sliced row
    a.dc_elements = E;
    a.dc_rows = ns;
    a.dc_every_row = ns == a.tree_nrows && nS + (int64_t)chain_q.size() == a.m;
    a.dc_slots = slots;
    a.dc_lane_records = 32 * nslices;
    for (uint32_t t : steps) {
        a.dc_steps += t;
        a.dc_longest = std::max<int64_t>(a.dc_longest, t);
    }
    deal_slices({&a}, a.dc_sched, a.dc_wbeg, a.dc_warps, st, 0, INT64_MAX, kDealSliced);
    deal_slices({&a}, a.dc_csched, a.dc_cwbeg, a.dc_cwarps, st, 0, INT64_MAX, kDealChains);
}

namespace {

// The chain kernel keeps its products in shared memory, the sliced-row
// kernels use none.  An SM set up for a kernel without shared memory (all of
// it L1) takes no CTA that needs some until it drains, so the chains would
// wait for the sliced rows instead of running beside them: every kernel here
// asks for the same split of L1 and shared memory.
constexpr int kCarveoutPct = 40;  // a chain CTA takes 73 KB

// Sets the split for kernel Kern once per device (the attribute belongs to
// the device's context).
template <auto Kern>
void same_carveout(int smem = 0)
{
    static std::atomic<uint64_t> done{0};
    int dev = 0;
    ABHSF_CUDA(cudaGetDevice(&dev));
    const uint64_t bit = uint64_t(1) << (dev & 63);
    if (done.load(std::memory_order_relaxed) & bit)
        return;
    ABHSF_CUDA(cudaFuncSetAttribute(Kern, cudaFuncAttributePreferredSharedMemoryCarveout, kCarveoutPct));
    if (smem > 48 * 1024)
        ABHSF_CUDA(cudaFuncSetAttribute(Kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    done.fetch_or(bit, std::memory_order_relaxed);
}

template <int S, int VT, bool B>
void launch_kind(beside& bs, bool chains, const dc_args& P, cudaStream_t st)
{
    if (chains) {
        constexpr int smem = kChainWarps * chain_smem_warp<typename vt_of<VT>::T, typename vt_of<VT>::V>();
        same_carveout<k_spmv_chains<S, VT, B>>(smem);
        const unsigned grid = (unsigned)((P.warps + kChainWarps - 1) / kChainWarps);
        launch_beside(bs, k_spmv_chains<S, VT, B>, grid, 32 * kChainWarps, smem, st, P);
    } else {
        same_carveout<k_spmv_slices<S, VT, B>>();
        const unsigned grid = (unsigned)((P.warps + kWarpsPerCta - 1) / kWarpsPerCta);
        launch_beside(bs, k_spmv_slices<S, VT, B>, grid, 32 * kWarpsPerCta, 0, st, P);
    }
}

template <int VT, bool B>
void launch_vt(beside& bs, int s, bool chains, const dc_args& P, cudaStream_t st)
{
    switch (s) {
    case 16: launch_kind<16, VT, B>(bs, chains, P, st); break;
    case 32: launch_kind<32, VT, B>(bs, chains, P, st); break;
    case 64: launch_kind<64, VT, B>(bs, chains, P, st); break;
    case 128: launch_kind<128, VT, B>(bs, chains, P, st); break;
    default: launch_kind<256, VT, B>(bs, chains, P, st); break;
    }
}

void launch(beside& bs, int s, int vt, bool batch, bool chains, const dc_args& P, cudaStream_t st)
{
    if (P.warps == 0)
        return;
    if (vt == ABHSF_VALUE_F64)
        batch ? launch_vt<ABHSF_VALUE_F64, true>(bs, s, chains, P, st) : launch_vt<ABHSF_VALUE_F64, false>(bs, s, chains, P, st);
    else if (vt == ABHSF_VALUE_F32)
        batch ? launch_vt<ABHSF_VALUE_F32, true>(bs, s, chains, P, st) : launch_vt<ABHSF_VALUE_F32, false>(bs, s, chains, P, st);
    else
        batch ? launch_vt<ABHSF_VALUE_BF16, true>(bs, s, chains, P, st)
              : launch_vt<ABHSF_VALUE_BF16, false>(bs, s, chains, P, st);
}

dc_mat mat_of(const abhsf_matrix& a) { return dc_mat{a.dc_words.get(), a.dc_vals.get(), a.dc_lane.get(), a.m}; }

dc_args args_of(const abhsf_matrix& a, const uint8_t* sched, const int64_t* wbeg, int warps, const void* x,
                int64_t ldx, void* y, int64_t ldy, int cols)
{
    dc_args P{};
    P.slices = reinterpret_cast<const dc_slice*>(sched);
    P.wbeg = wbeg;
    P.warps = warps;
    P.A = mat_of(a);
    P.x = x;
    P.y = y;
    P.ldx = ldx;
    P.ldy = ldy;
    P.cols = cols;
    return P;
}

dc_args batch_args(const abhsf_batch& b, const uint8_t* sched, const int64_t* wbeg, int warps,
                   const double* const* xs, double* const* ys)
{
    dc_args P{};
    P.slices = reinterpret_cast<const dc_slice*>(sched);
    P.wbeg = wbeg;
    P.warps = warps;
    P.mats = reinterpret_cast<const dc_mat*>(b.dc_table.get());
    P.xs = reinterpret_cast<const void* const*>(xs);
    P.ys = reinterpret_cast<void* const*>(ys);
    P.ldx = P.ldy = 1;
    P.cols = 1;
    return P;
}

// Column groups first in the grid: the groups of one slice run side by side
// and share its words and values in L2.
template <int S>
void launch_mm(beside& bs, bool chains, bool late, bool many, const dc_args& P, cudaStream_t st)
{
    same_carveout<k_spmm_chains<S>>();
    same_carveout<k_spmm_slices<S, kMmCols, kMmLateCtas>>();
    const int per = chains ? kChainWarps : kMmWarps;
    auto grid = [&](int cols) {
        return dim3((unsigned)((cols + kMmCols - 1) / kMmCols), (unsigned)((P.warps + per - 1) / per));
    };
    if (chains) {
        launch_beside(bs, k_spmm_chains<S>, grid(P.cols), 32u * per, 0, st, P);
        return;
    }
    if (late) {  // (k_spmm_slices)
        launch_beside(bs, k_spmm_slices<S, kMmCols, kMmLateCtas>, grid(P.cols), 32u * per, 0, st, P);
        return;
    }
    dc_args R = P;
    R.cols = P.cols / kMmWide * kMmWide;
    if (R.cols > 0)
        launch_beside(bs, k_spmm_slices<S, kMmWide, kMmCtas>, grid(R.cols), 32u * per, 0, st, R);
    if (R.cols == P.cols)
        return;
    R.x = static_cast<const double*>(P.x) + R.cols;
    R.y = static_cast<double*>(P.y) + R.cols;
    R.cols = P.cols - R.cols;
    launch_beside(bs, many ? k_spmm_slices<S, kMmCols, kMmCtas> : k_spmm_slices<S, kMmCols, kMmLateCtas>, grid(R.cols),
                  32u * per, 0, st, R);
}

// P.cols columns: the SpMV kernels for one, the SpMM ones (FP64) for more and
// for one that is a column of a wider X or Y.
void launch_cols(beside& bs, int s, int vt, bool chains, bool late, bool many, const dc_args& P, cudaStream_t st)
{
    if (P.warps == 0)
        return;
    if (P.cols == 1 && P.ldx == 1 && P.ldy == 1) {
        launch(bs, s, vt, false, chains, P, st);
        return;
    }
    switch (s) {
    case 16: launch_mm<16>(bs, chains, late, many, P, st); break;
    case 32: launch_mm<32>(bs, chains, late, many, P, st); break;
    case 64: launch_mm<64>(bs, chains, late, many, P, st); break;
    case 128: launch_mm<128>(bs, chains, late, many, P, st); break;
    default: launch_mm<256>(bs, chains, late, many, P, st); break;
    }
}

}  // namespace

dc_plan plan_of(const abhsf_matrix& a)
{
    dc_plan p;
    p.sched = a.dc_sched.get();
    p.wbeg = a.dc_wbeg.get();
    p.warps = a.dc_warps;
    p.csched = a.dc_csched.get();
    p.cwbeg = a.dc_cwbeg.get();
    p.cwarps = a.dc_cwarps;
    p.steps = a.dc_steps;
    p.longest = a.dc_longest;
    return p;
}

void slices_begin(beside& bs, const abhsf_matrix& a, const dc_plan& p, const void* x, int64_t ldx, void* y,
                  int64_t ldy, cudaStream_t st, int cols)
{
    if (p.cwarps)
        launch_cols(bs, a.s, a.value_type, true, false, false, args_of(a, p.csched, p.cwbeg, p.cwarps, x, ldx, y, ldy, cols), st);
}

void slices_end(beside& bs, const abhsf_matrix& a, const dc_plan& p, const void* x, int64_t ldx, void* y, int64_t ldy,
                cudaStream_t st, int cols)
{
    // SpMM: 148 x 10 x 2 warps share the steps of every four columns
    const int64_t warps = 148 * kMmLateCtas * kMmWarps, steps = p.steps * ((cols + 3) / 4);
    const bool late = p.cwarps > 0 || p.longest * warps > steps, many = steps >= kMmManySteps * warps;
    if (p.warps)
        launch_cols(bs, a.s, a.value_type, false, late, many,
                    args_of(a, p.sched, p.wbeg, p.warps, x, ldx, y, ldy, cols), st);
}

bool spmv_sets_y(const abhsf_matrix& a) { return a.dc_every_row; }

void spmv_set_y(const abhsf_matrix& a, const void* x, void* y, const int* skip, cudaStream_t st)
{
    beside bs;
    bs.any = true;  // its first kernel is queued while the kernel before runs, and waits for it at its start
    auto args = [&](const dbuf<uint8_t>& sched, const dbuf<int64_t>& wbeg, int warps, bool wait) {
        dc_args P = args_of(a, sched.get(), wbeg.get(), warps, x, 1, y, 1, 1);
        P.fresh = 1;
        P.wait = wait;
        P.skip = skip;
        return P;
    };
    if (a.dc_cwarps)
        launch(bs, a.s, a.value_type, false, true, args(a.dc_csched, a.dc_cwbeg, a.dc_cwarps, true), st);
    if (a.dc_warps)
        launch(bs, a.s, a.value_type, false, false, args(a.dc_sched, a.dc_wbeg, a.dc_warps, a.dc_cwarps == 0), st);
}

// The ring kernel serves some block rows: the sliced rows go beside it, dealt
// over one CTA an SM, for which the ring leaves registers and warps (they need no
// shared memory).  The ring is queued first: behind the sliced rows it began 5 us
// later (tiled mixture 104.4 against 109.2 us, f32 73.2 against 76.9).
void slices_beside_ring(abhsf_matrix& a, cudaStream_t st)
{
    if (a.dc_warps == 0)
        return;
    deal_slices({&a}, a.dc_sched, a.dc_wbeg, a.dc_warps, st, 0, INT64_MAX, kDealSliced, true);
}

// The slices of every matrix of a batch in one launch (and its chains in one more).
void prepare_batch_stream(abhsf_batch& b, cudaStream_t st)
{
    b.dc_warps = b.dc_cwarps = 0;
    std::vector<dc_mat> t;
    bool any = false;
    for (const abhsf_matrix* a : b.mats) {
        t.push_back(mat_of(*a));
        any = any || !a->dc_host.empty();
    }
    if (!any)
        return;
    b.dc_table.alloc(t.size() * sizeof(dc_mat));
    ABHSF_CUDA(cudaMemcpyAsync(b.dc_table.get(), t.data(), t.size() * sizeof(dc_mat), cudaMemcpyHostToDevice, st));
    deal_slices(b.mats, b.dc_sched, b.dc_wbeg, b.dc_warps, st, 0, INT64_MAX, kDealSliced);
    deal_slices(b.mats, b.dc_csched, b.dc_cwbeg, b.dc_cwarps, st, 0, INT64_MAX, kDealChains);
}

void batch_stream_begin(beside& bs, const abhsf_batch& b, const double* const* xs, double* const* ys, cudaStream_t st)
{
    if (b.dc_cwarps)
        launch(bs, b.s, ABHSF_VALUE_F64, true, true,
               batch_args(b, b.dc_csched.get(), b.dc_cwbeg.get(), b.dc_cwarps, xs, ys), st);
}

void batch_stream_end(beside& bs, const abhsf_batch& b, const double* const* xs, double* const* ys, cudaStream_t st)
{
    if (b.dc_warps)
        launch(bs, b.s, ABHSF_VALUE_F64, true, false,
               batch_args(b, b.dc_sched.get(), b.dc_wbeg.get(), b.dc_warps, xs, ys), st);
}

}  // namespace abhsf

extern "C" abhsf_status abhsf_slices_info(const abhsf_matrix* a, int64_t* slices, int64_t* slots,
                                          int64_t* lane_records, int64_t* elements, int64_t* block_rows)
{
    return abhsf::guarded([&] {
        if (!a)
            abhsf::fail(ABHSF_ERROR_INVALID_VALUE, "matrix handle is NULL");
        if (slices)
            *slices = (int64_t)a->dc_host.size();
        if (slots)
            *slots = a->dc_slots;
        if (lane_records)
            *lane_records = a->dc_lane_records;
        if (elements)
            *elements = a->dc_elements;
        if (block_rows)
            *block_rows = a->dc_rows;
    });
}

extern "C" abhsf_status abhsf_slices_export(const abhsf_matrix* a, int64_t* base, int64_t* meta, uint32_t* brow,
                                            uint32_t* steps, uint32_t* lanes, uint8_t* chain, uint32_t* lane_records,
                                            uint32_t* words, void* values)
{
    return abhsf::guarded([&] {
        if (!a)
            abhsf::fail(ABHSF_ERROR_INVALID_VALUE, "matrix handle is NULL");
        const auto& P = a->dc_host;
        for (size_t k = 0; k < P.size(); ++k) {
            if (base)
                base[k] = P[k].base;
            if (meta)
                meta[k] = P[k].meta;
            if (brow)
                brow[k] = P[k].brow;
            if (steps)
                steps[k] = P[k].steps;
            if (lanes)
                lanes[k] = P[k].lanes;
            if (chain)
                chain[k] = P[k].chain ? 1 : 0;
        }
        if (lane_records && a->dc_lane_records)
            ABHSF_CUDA(cudaMemcpy(lane_records, a->dc_lane.get(), a->dc_lane_records * sizeof(uint32_t),
                                  cudaMemcpyDeviceToHost));
        if (a->dc_slots > 0) {
            if (words)
                ABHSF_CUDA(cudaMemcpy(words, a->dc_words.get(), a->dc_slots * sizeof(uint32_t), cudaMemcpyDeviceToHost));
            if (values)
                ABHSF_CUDA(cudaMemcpy(values, a->dc_vals.get(), a->dc_slots * abhsf::value_size(a->value_type),
                                      cudaMemcpyDeviceToHost));
        }
    });
}
