// chain_sum.cuh -- a chain of rounded additions summed by a whole warp, to the
// bit.
//
// y = fl(... fl(fl(y + p_0) + p_1) ... + p_n): the reference's order fixes the
// result, and adding one product after another costs the latency of an
// addition each (8.2 cycles in FP64).  Rounded addition does not regroup, but
// inside one binade it moves rigidly: let every partial sum of a run of
// additions lie strictly inside one binade (2^e, 2^(e+1)) whose spacing is u.
// Each addition then rounds to a multiple of u, and started d spacings higher
// (still inside the binade) every partial sum is exactly d spacings higher --
// if d is even, or if no addition is a tie (round to even looks at the last
// bit of the sum).
//
// So the products are split into segments, one a lane.  Every lane guesses its
// segment's start (a scan of the segments' plain sums), runs its additions
// from there, and notes whether its partial sums stayed inside a binade with
// room at its ends, and whether one was a tie.  How far each segment's start
// was from its predecessor's end, in spacings (the difference of the bit
// patterns), is scanned too: that is the distance from the true start.  The
// first segment the rule does not cover is run again from its true start, now
// known, and the distances after it are set right.  Every segment is thus either run
// from its true start or covered by the rule: the result is the one of the
// additions in turn, whatever the values (infinities, NaN, subnormals and
// zeros fail the rule and are run again).
#pragma once

#include <climits>

#include "common.cuh"

namespace abhsf {
namespace chain {

// Bit patterns.  key: sign, exponent and kKeyMant mantissa bits; a partial sum
// whose key is not the first or last of its binade can move by kRoom spacings
// and stay inside.
struct f64_bits {
    using I = long long;
    static constexpr int kMant = 52, kExpMax = 0x7ff, kKeyMant = 20;
    static constexpr int kRoom = 0x7fffffff;
    __device__ static I bits(double v) { return __double_as_longlong(v); }
    __device__ static double value(I b) { return __longlong_as_double(b); }
    __device__ static uint32_t key(double v) { return (uint32_t)__double2hiint(v); }
    __device__ static double half_spacing(int ex) { return __hiloint2double((ex - kMant - 1) << 20, 0); }
    __device__ static double add(double a, double b) { return __dadd_rn(a, b); }
    __device__ static double mag(double a) { return fabs(a); }
};
struct f32_bits {
    using I = int;
    static constexpr int kMant = 23, kExpMax = 0xff, kKeyMant = 13;
    static constexpr int kRoom = (1 << (kMant - kKeyMant)) - 1;
    __device__ static I bits(float v) { return __float_as_int(v); }
    __device__ static float value(I b) { return __int_as_float(b); }
    __device__ static uint32_t key(float v) { return (uint32_t)__float_as_int(v) >> (kMant - kKeyMant); }
    __device__ static float half_spacing(int ex) { return __int_as_float((ex - kMant - 1) << kMant); }
    __device__ static float add(float a, float b) { return __fadd_rn(a, b); }
    __device__ static float mag(float a) { return fabsf(a); }
};
template <typename T>
struct bits_of {
    using B = f64_bits;
};
template <>
struct bits_of<float> {
    using B = f32_bits;
};

// Adds p[0 .. L-1] onto a in turn.  inside: every partial sum, a among them,
// lies inside one binade with room for kRoom spacings at both ends; tie: one
// of the additions was a tie (meaningful where inside).
template <int L, typename T>
__device__ __forceinline__ T run_segment(T a, const T (&p)[L], bool& inside, bool& tie)
{
    using B = typename bits_of<T>::B;
    constexpr uint32_t mm = (1u << B::kKeyMant) - 1u;
    uint32_t lo = B::key(a), hi = lo;
    const int ex = (int)((lo >> B::kKeyMant) & (uint32_t)B::kExpMax);
    // half a spacing of the binade; too small a binade fails the test below
    const T half = B::half_spacing(max(ex, B::kMant + 2));
    bool t = false;
#pragma unroll
    for (int i = 0; i < L; ++i) {
        const T s = B::add(a, p[i]);
        // inside a binade s - a is exact, and so is the rounding error p - (s - a)
        const T err = B::add(p[i], -B::add(s, -a));
        t = t || B::mag(err) == half;
        a = s;
        const uint32_t k = B::key(a);
        lo = min(lo, k);
        hi = max(hi, k);
    }
    inside = (lo >> B::kKeyMant) == (hi >> B::kKeyMant) && (lo & mm) != 0u && (hi & mm) != mm && ex > B::kMant + 1 &&
             ex != B::kExpMax;
    tie = t;
    return a;
}

// The exponent of v as an integer that compares like |v| (inf and NaN above all).
template <typename T>
__device__ __forceinline__ uint32_t exponent(T v)
{
    using B = typename bits_of<T>::B;
    return (B::key(v) >> B::kKeyMant) & (uint32_t)B::kExpMax;
}

// Whether few of a group's segments will cross a binade, by a sample of its
// products (a quarter of each lane's): they are of one sign (the sum doubles a few
// times at most), or y is 2^kAbove times as large.  Sums near zero of products of
// both signs would have most segments run again.
template <int kAbove, int L, typename T>
__device__ __forceinline__ bool calm(T y, const T (&p)[L])
{
    uint32_t most = 0, signs = 0;
#pragma unroll
    for (int i = 1; i < L; i += 4) {
        const uint32_t e = exponent(p[i]);
        most = max(most, e);
        signs |= e == 0 ? 0u : p[i] < T(0) ? 1u : 2u;
    }
    return __reduce_or_sync(0xffffffffu, signs) != 3u ||
           exponent(y) >= __reduce_max_sync(0xffffffffu, most) + (uint32_t)kAbove;
}

// p[0 .. L-1] added onto a in turn, and nothing else.
template <int L, typename T>
__device__ __forceinline__ T add_segment(T a, const T (&p)[L])
{
#pragma unroll
    for (int i = 0; i < L; ++i)
        a = bits_of<T>::B::add(a, p[i]);
    return a;
}

// Adds the products of 32 / STRIDE segments of L each onto y, in order: lane
// STRIDE g + h holds segment g of chain h in p (STRIDE chains at once, each
// lane of a chain holding its y).  Returns how many steps of running segments
// again it took; -1, y unchanged, where more than kAgain would have to be run one
// after another: the caller adds in turn.
template <int STRIDE, int L, typename T>
__device__ __forceinline__ int sum_group(T& y, const T (&p)[L], int lane)
{
    using B = typename bits_of<T>::B;
    using I = typename B::I;
    constexpr unsigned full = 0xffffffffu;
    // Segments run again at most.  Adding in turn takes as long as some 16
    // of 32 segments run again, but 4 of 8 (R-MAT scale 18, 7 columns: 121 us
    // with 2 or more of 8, 99 with 1).
    constexpr int kAgain = STRIDE == 1 ? 12 : 1;
    constexpr int kFar = 1 << 20;  // spacings between a start and the end before it
    const int g = lane / STRIDE, h = lane % STRIDE;
    const unsigned mine = (full / ((1u << STRIDE) - 1u)) << h;  // the lanes of this chain
    T part[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        part[i] = p[i];
#pragma unroll
    for (int i = 4; i < L; ++i)
        part[i % 4] = B::add(part[i % 4], p[i]);
    T sum = B::add(B::add(part[0], part[1]), B::add(part[2], part[3]));
#pragma unroll
    for (int d = STRIDE; d < 32; d *= 2) {
        const T t = __shfl_up_sync(full, sum, d);
        if (lane >= d)
            sum = B::add(sum, t);
    }
    sum = __shfl_up_sync(full, sum, STRIDE);
    const T start = g ? B::add(y, sum) : y;
    bool inside, tie;
    T end = run_segment<L>(start, p, inside, tie);
    const unsigned outside = __ballot_sync(full, !inside);
    if (__any_sync(full, __popc(outside & mine) > kAgain))
        return -1;
    const long long gap = (long long)B::bits(__shfl_up_sync(full, end, STRIDE)) - (long long)B::bits(start);
    const bool far = gap >= kFar || gap <= -kFar;
    int off = g > 0 && !far ? (int)gap : 0;  // spacings from the start to the true start
#pragma unroll
    for (int d = STRIDE; d < 32; d *= 2) {
        const int t = __shfl_up_sync(full, off, d);
        if (lane >= d)
            off += t;
    }
    int first = 0;  // segments up to this one are settled
#pragma unroll 1
    for (int again = 0;; ++again) {
        const bool good =
            g <= first ||
            (!far && (off == 0 || (inside && off <= B::kRoom && off >= -B::kRoom && !(tie && (off & 1)))));
        const unsigned bad = __ballot_sync(full, !good);
        const T moved = B::value(B::bits(end) + (I)off);  // the true end
        if (bad == 0) {
            y = __shfl_sync(full, moved, 32 - STRIDE + h);
            return again;
        }
        if (again == kAgain)
            return -1;
        // this chain's first segment that the rule does not cover, from its
        // true start; the later segments' distances move by as much as its end did
        const T again_end = add_segment<L>(__shfl_up_sync(full, moved, STRIDE), p);
        const long long shift = (long long)B::bits(again_end) - (long long)B::bits(end);
        const int b = bad & mine ? (__ffs(bad & mine) - 1) / STRIDE : g;
        const int more = __shfl_sync(full, shift < kFar && shift > -kFar ? (int)shift - off : INT_MIN, b * STRIDE + h);
        if (__any_sync(full, (bad & mine) && more == INT_MIN))
            return -1;
        if (bad & mine) {
            first = b;
            if (g == b) {
                end = again_end;
                off = 0;
            } else if (g > b) {
                off += more;
            }
        }
    }
}

}  // namespace chain
}  // namespace abhsf
