// cg.cu -- conjugate gradients on ABHSF matrices: plain FP64, and mixed
// precision (an f32 CG on an f32 or bf16 copy of the matrix whose solution
// accumulates in FP64 and whose residual is replaced by the FP64 residual of
// the f64 matrix each time it has fallen by a set factor: reliable updates).
//
// The reference has no solver; its SpMV is the kernel such a solver calls
// (spmv/bottlenecks/spmv.cpp:58-64).  Both solvers here keep every scalar
// (alpha, beta, r.r) on the device: a CG iteration is one SpMV and three vector
// kernels, and chunks of iterations are captured once into a CUDA graph and
// replayed.  A dot product is summed in FP64 over a fixed grid (deterministic);
// the kernel that needs the result adds up the grid's partial sums itself, every
// CTA the same way, instead of waiting for a kernel of one CTA.  Each kernel is
// launched while the one before it ends (programmatic dependent launch) and
// waits for it on the device.  Once the recurrence residual meets the tolerance,
// the state's `done` flag turns the rest of the chunk into no-ops; where the
// SpMV heeds the flag too, a chunk is queued before the state after the one
// before it has been read.
// Bound by memory for large systems and by the launches for small ones.  The
// vector kernels move ten vectors an iteration (dot 2, residual 3, direction 5),
// and the SpMV that sets y does not read it; where it adds, the residual kernel
// clears Ap too, eleven.  A kernel each for the dot, for x and r, and for p moved
// twelve.
#include <cmath>
#include <vector>

#include "common.cuh"
#include "internal.cuh"

namespace abhsf {
namespace {

constexpr int kRedBlocks = 592;  // 4 x 148 SMs
constexpr int kRedThreads = 256;
constexpr int kChunk = 8;  // CG iterations per captured graph

// rr and done: entry i for iterations whose number in the chunk is i modulo 2.
// A kernel reads this iteration's entry and writes the next one's.
struct cg_state {
    double rr[2];  // r . r of the residual the iteration starts from
    double alpha;  // step of this iteration
    double tol2;   // stop when r . r <= tol2
    int done[2];   // tolerance met, or iteration limit reached, before the iteration
    int iters;     // iterations performed
    int max_iters;
    int active;  // this iteration updates x, r and p (not a breakdown)
};
static_assert(kChunk % 2 == 0, "a chunk ends at entry 0 again");

// Waits for the kernel before, then lets the next one be launched (launches with
// the programmatic-serialization attribute).  What the kernel before wrote is
// read by plain loads: the read-only path (const __restrict__, __ldg) promises
// nothing about data written during the kernel's life, which begins before the
// wait.
__device__ __forceinline__ void wait_and_next()
{
    asm volatile("griddepcontrol.wait;\ngriddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ double block_sum(double v)
{
    __shared__ double part[kRedThreads / 32];
    for (int d = 16; d > 0; d >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, d);
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = v;
    __syncthreads();
    v = threadIdx.x < kRedThreads / 32 ? part[threadIdx.x] : 0.0;
    if (threadIdx.x < 32)
        for (int d = 16; d > 0; d >>= 1)
            v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;  // valid in thread 0
}

// 16 bytes of T: the unit the vector kernels below load and store when every
// array they touch is 16-byte aligned (VEC), so that an f32 pass moves as
// many bytes per instruction as an f64 one.
template <typename T>
struct __align__(16) pack {
    static constexpr int N = 16 / sizeof(T);
    T v[N];
};

template <typename T>
__device__ __forceinline__ pack<T> ld_pack(const T* p)
{
    return *reinterpret_cast<const pack<T>*>(p);
}

template <typename T>
__device__ __forceinline__ void st_pack(T* p, const pack<T>& v)
{
    *reinterpret_cast<pack<T>*>(p) = v;
}

constexpr int64_t kStride = (int64_t)kRedBlocks * kRedThreads;

// partial[blockIdx.x] = sum over this block's grid-stride share of a[i] b[i]
// (with VEC, packs of 16 bytes, then the tail past the last whole pack)
template <typename T, bool VEC>
__global__ void __launch_bounds__(kRedThreads) k_dot(int64_t n, const T* a, const T* b, double* partial,
                                                     const int* done)
{
    wait_and_next();
    if (done && *done)
        return;
    constexpr int N = pack<T>::N;
    const int64_t tid = blockIdx.x * (int64_t)kRedThreads + threadIdx.x;
    const int64_t nv = VEC ? n / N : 0;
    double s = 0.0;
    for (int64_t i = tid; i < nv; i += kStride) {
        const pack<T> va = ld_pack(a + i * N), vb = ld_pack(b + i * N);
#pragma unroll
        for (int k = 0; k < N; ++k)
            s += (double)va.v[k] * (double)vb.v[k];
    }
    for (int64_t i = nv * N + tid; i < n; i += kStride)
        s += (double)a[i] * (double)b[i];
    s = block_sum(s);
    if (threadIdx.x == 0)
        partial[blockIdx.x] = s;
}

__device__ __forceinline__ double sum_partials(const double* partial)
{
    double s = 0.0;
    for (int i = threadIdx.x; i < kRedBlocks; i += kRedThreads)
        s += partial[i];
    return block_sum(s);
}

// state from r . r (first partials), with tolerance tol2 = rtol^2 * bb
__global__ void __launch_bounds__(kRedThreads) k_cg_init(const double* __restrict__ partial, cg_state* st,
                                                         double tol2, int max_iters)
{
    const double rr = sum_partials(partial);
    if (threadIdx.x == 0) {
        st->rr[0] = rr;
        st->alpha = 0.0;
        st->tol2 = tol2;
        st->iters = 0;
        st->max_iters = max_iters;
        st->active = 0;
        st->done[0] = (rr <= tol2 || max_iters <= 0) ? 1 : 0;
    }
}

// restart the recurrence from a replaced residual: r . r from the partials,
// the tolerance factor2 * r . r, the search direction and iteration count kept
__global__ void __launch_bounds__(kRedThreads) k_cg_resume(const double* __restrict__ partial, cg_state* st,
                                                           double factor2)
{
    const double rr = sum_partials(partial);
    if (threadIdx.x == 0) {
        const double tol2 = factor2 * rr;
        st->rr[0] = rr;
        st->tol2 = tol2;
        st->done[0] = (rr <= tol2 || st->iters >= st->max_iters) ? 1 : 0;
    }
}

// alpha = r.r / p.Ap from the partial sums; r -= alpha Ap; partial r . r.
// ZERO: Ap = 0, ready for the next y += A p (else that SpMV starts from zero).
template <typename T, bool VEC, bool ZERO>
__global__ void __launch_bounds__(kRedThreads) k_cg_residual(int64_t n, T* r, T* ap, cg_state* st, int cur,
                                                             const double* pap_part, double* partial)
{
    wait_and_next();
    constexpr int N = pack<T>::N;
    __shared__ double step;
    const int64_t tid = blockIdx.x * (int64_t)kRedThreads + threadIdx.x;
    const int64_t nv = VEC ? n / N : 0;
    // the first packs are on their way while the partial sums are added up
    pack<T> nr{}, na{};
    if (tid < nv) {
        nr = ld_pack(r + tid * N);
        na = ld_pack(ap + tid * N);
    }
    if (st->done[cur])
        return;
    const double pap = sum_partials(pap_part);
    if (threadIdx.x == 0) {
        const bool go = pap > 0.0;  // else breakdown: p = 0 or A not positive definite on p
        step = go ? st->rr[cur] / pap : 0.0;
        if (blockIdx.x == 0) {
            st->alpha = step;
            st->active = go ? 1 : 0;
        }
    }
    __syncthreads();
    const T alpha = (T)step;
    double s = 0.0;
    for (int64_t i = tid; i < nv; i += kStride) {
        pack<T> vr = nr;
        const pack<T> va = na;
        if (i + kStride < nv) {
            nr = ld_pack(r + (i + kStride) * N);
            na = ld_pack(ap + (i + kStride) * N);
        }
        pack<T> zero;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            vr.v[k] = vr.v[k] - alpha * va.v[k];
            zero.v[k] = T(0);
            s += (double)vr.v[k] * (double)vr.v[k];
        }
        st_pack(r + i * N, vr);
        if (ZERO)
            st_pack(ap + i * N, zero);
    }
    for (int64_t i = nv * N + tid; i < n; i += kStride) {
        const T ri = r[i] - alpha * ap[i];
        r[i] = ri;
        if (ZERO)
            ap[i] = T(0);
        s += (double)ri * (double)ri;
    }
    s = block_sum(s);
    if (threadIdx.x == 0)
        partial[blockIdx.x] = s;
}

// beta = new r.r / r.r from the partial sums; x += alpha p; p = r + beta p, also
// in the iteration that met the tolerance, so that a recurrence resumed from a
// replaced residual continues from the right p; the next iteration's state.
template <typename T, bool VEC>
__global__ void __launch_bounds__(kRedThreads) k_cg_direction(int64_t n, T* x, T* p, const T* r, cg_state* st, int cur,
                                                              const double* rr_part)
{
    wait_and_next();
    constexpr int N = pack<T>::N;
    const int nxt = cur ^ 1;
    const int64_t tid = blockIdx.x * (int64_t)kRedThreads + threadIdx.x;
    const int64_t nv = VEC ? n / N : 0;
    pack<T> nx{}, np{}, nr{};  // the next pack of each vector
    if (tid < nv) {
        nx = ld_pack(x + tid * N);
        np = ld_pack(p + tid * N);
        nr = ld_pack(r + tid * N);
    }
    if (st->done[cur]) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            st->rr[nxt] = st->rr[cur];
            st->done[nxt] = 1;
        }
        return;
    }
    __shared__ double grow;
    const bool active = st->active != 0;
    const T alpha = (T)st->alpha;
    const double rr_new = sum_partials(rr_part);
    if (threadIdx.x == 0) {
        const double rr = st->rr[cur];
        grow = rr_new / rr;
        if (blockIdx.x == 0) {
            int done = 1;
            if (active) {
                const int iters = st->iters + 1;
                st->iters = iters;
                done = rr_new <= st->tol2 || iters >= st->max_iters ? 1 : 0;
            }
            st->rr[nxt] = active ? rr_new : rr;
            st->done[nxt] = done;
        }
    }
    __syncthreads();
    const T beta = (T)grow;
    for (int64_t i = tid; i < nv; i += kStride) {
        pack<T> vx = nx, vp = np;
        const pack<T> vr = nr;
        const int64_t j = i + kStride;
        if (j < nv) {
            nx = ld_pack(x + j * N);
            np = ld_pack(p + j * N);
            nr = ld_pack(r + j * N);
        }
#pragma unroll
        for (int k = 0; k < N; ++k) {
            vx.v[k] += alpha * vp.v[k];
            vp.v[k] = vr.v[k] + beta * vp.v[k];
        }
        st_pack(x + i * N, vx);
        if (active)
            st_pack(p + i * N, vp);
    }
    for (int64_t i = nv * N + tid; i < n; i += kStride) {
        const T pi = p[i];
        x[i] += alpha * pi;
        if (active)
            p[i] = r[i] + beta * pi;
    }
}

template <typename T>
__global__ void k_neg(int64_t n, const T* __restrict__ a, T* __restrict__ out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = -a[i];
}

// out = (float) r
__global__ void k_to_f32(int64_t n, const double* __restrict__ r, float* __restrict__ out)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = (float)r[i];
}

// x += d; d = 0 (the f32 correction folded into the FP64 solution)
__global__ void k_fold(int64_t n, double* __restrict__ x, float* __restrict__ d)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        x[i] += (double)d[i];
        d[i] = 0.0f;
    }
}

unsigned elem_grid(int64_t n) { return (unsigned)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16)); }

// y += A x in T (f64 or f32 kernels)
void spmv_t(const abhsf_matrix& a, const double* x, double* y, cudaStream_t st) { spmv_dispatch(a, x, y, st); }
void spmv_t(const abhsf_matrix& a, const float* x, float* y, cudaStream_t st) { spmv_f32_dispatch(a, x, y, st); }

template <typename T>
struct cg_work {
    scratch<T> r, p, ap;
    cg_work(int64_t n, cudaStream_t cs) : r(n, cs), p(n, cs), ap(n, cs) {}
};

// r = b - A x (xn: scratch)
template <typename T>
void residual(const abhsf_matrix& a, const T* b, const T* x, T* r, T* xn, int64_t n, cudaStream_t st)
{
    k_neg<T><<<elem_grid(n), 256, 0, st>>>(n, x, xn);
    ABHSF_CUDA(cudaMemcpyAsync(r, b, n * sizeof(T), cudaMemcpyDeviceToDevice, st));
    spmv_t(a, xn, r, st);
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// A vector kernel that waits on the device for the kernel before it in st.
template <typename... P, typename... A>
void launch_after(void (*kern)(P...), cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kRedBlocks);
    cfg.blockDim = dim3(kRedThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    ABHSF_CUDA(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
}

template <typename T>
void dot(const T* a, const T* b, int64_t n, double* partial, cudaStream_t st, const int* done = nullptr)
{
    launch_after(aligned16(a) && aligned16(b) ? k_dot<T, true> : k_dot<T, false>, st, n, a, b, partial, done);
}

// p = r and the state from r . r: the start of a CG recurrence.
template <typename T>
void cg_start(cg_work<T>& w, int64_t n, cg_state* st_d, double* partial, double tol2, int max_iters,
              cudaStream_t cs)
{
    ABHSF_CUDA(cudaMemcpyAsync(w.p.get(), w.r.get(), n * sizeof(T), cudaMemcpyDeviceToDevice, cs));
    dot<T>(w.r.get(), w.r.get(), n, partial, cs);
    k_cg_init<<<1, kRedThreads, 0, cs>>>(partial, st_d, tol2, max_iters);
    ABHSF_CUDA(cudaGetLastError());
}

// kChunk CG iterations on A x = b (x, w.r, w.p, w.ap and the state on the
// device), captured once into a graph and replayed until the state is done.
template <typename T>
class cg_graph {
  public:
    // partial: 2 kRedBlocks
    cg_graph(const abhsf_matrix& a, T* x, cg_work<T>& w, int64_t n, cg_state* st_d, double* partial, cudaStream_t cs)
        : heeds_(spmv_sets_y(a)), ap_(w.ap.get()), n_(n)
    {
        ABHSF_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&seen_), 2 * sizeof(cg_state), cudaHostAllocDefault));
        cudaGraph_t graph = nullptr;
        try {
            for (cudaEvent_t& e : ev_)
                ABHSF_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
            ABHSF_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
            try {
                record(a, x, w, n, st_d, partial, cs);
            } catch (...) {
                if (cudaStreamEndCapture(cs, &graph) == cudaSuccess && graph)
                    cudaGraphDestroy(graph);
                throw;
            }
            const cudaError_t cap = cudaStreamEndCapture(cs, &graph);
            if (cap != cudaSuccess || !graph)
                fail(ABHSF_ERROR_CUDA, std::string("CG graph capture: ") + cudaGetErrorString(cap));
            const cudaError_t ins = cudaGraphInstantiate(&exec_, graph, 0);
            cudaGraphDestroy(graph);
            if (ins != cudaSuccess)
                fail(ABHSF_ERROR_CUDA, std::string("CG graph instantiation: ") + cudaGetErrorString(ins));
        } catch (...) {
            release();
            throw;
        }
    }
    ~cg_graph() { release(); }
    cg_graph(const cg_graph&) = delete;
    cg_graph& operator=(const cg_graph&) = delete;

    // Replays chunks until the state says done; returns the iteration count.
    // Where a chunk after the last is a no-op throughout, it is queued before
    // the state is read, so that the GPU does not wait for the host.
    // An SpMV that adds finds Ap = 0, left by the residual kernel of the
    // iteration before -- but behind the last iteration of a recurrence the
    // chunk's remaining products still add onto it, and a recurrence that is
    // resumed (the mixed solver's) must not start from that.
    int run(const cg_state* st_d, cudaStream_t cs)
    {
        if (!heeds_)
            ABHSF_CUDA(cudaMemsetAsync(ap_, 0, n_ * sizeof(T), cs));
        for (int k = 0;; ++k) {
            if (heeds_ || k > 0)
                ABHSF_CUDA(cudaGraphLaunch(exec_, cs));
            ABHSF_CUDA(cudaMemcpyAsync(seen_ + (k & 1), st_d, sizeof(cg_state), cudaMemcpyDeviceToHost, cs));
            ABHSF_CUDA(cudaEventRecord(ev_[k & 1], cs));
            const int look = heeds_ ? k - 1 : k;  // the state to wait for
            if (look < 0)
                continue;
            ABHSF_CUDA(cudaEventSynchronize(ev_[look & 1]));
            if (seen_[look & 1].done[0])
                return seen_[look & 1].iters;
        }
    }

  private:
    void record(const abhsf_matrix& a, T* x, cg_work<T>& w, int64_t n, cg_state* st_d, double* partial, cudaStream_t cs)
    {
        T *r = w.r.get(), *p = w.p.get(), *ap = w.ap.get();
        const bool vec = aligned16(x) && aligned16(r) && aligned16(ap) && aligned16(p);
        double *pap = partial, *rr = partial + kRedBlocks;
        for (int it = 0; it < kChunk; ++it) {
            const int cur = it & 1;
            if (heeds_)
                spmv_set_y(a, p, ap, st_d->done + cur, cs);
            else
                spmv_t(a, p, ap, cs);
            dot<T>(p, ap, n, pap, cs, st_d->done + cur);
            launch_after(heeds_ ? (vec ? k_cg_residual<T, true, false> : k_cg_residual<T, false, false>)
                                : (vec ? k_cg_residual<T, true, true> : k_cg_residual<T, false, true>),
                         cs, n, r, ap, st_d, cur, pap, rr);
            launch_after(vec ? k_cg_direction<T, true> : k_cg_direction<T, false>, cs, n, x, p, r, st_d, cur, rr);
        }
    }
    void release()
    {
        if (exec_)
            cudaGraphExecDestroy(exec_);
        for (cudaEvent_t e : ev_)
            if (e)
                cudaEventDestroy(e);
        if (seen_)
            cudaFreeHost(seen_);
    }

    const bool heeds_;  // the SpMV sets y and heeds the done flag
    T* const ap_;
    const int64_t n_;
    cg_state* seen_ = nullptr;  // pinned: the state after the last two chunks
    cudaEvent_t ev_[2] = {nullptr, nullptr};
    cudaGraphExec_t exec_ = nullptr;
};

struct solve_stream {
    cudaStream_t user, cs = nullptr;
    cudaEvent_t ev = nullptr;
    explicit solve_stream(cudaStream_t u) : user(u)
    {
        ABHSF_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
        ABHSF_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        ABHSF_CUDA(cudaEventRecord(ev, user));  // the solve starts after the caller's queued work
        ABHSF_CUDA(cudaStreamWaitEvent(cs, ev, 0));
    }
    ~solve_stream()
    {
        cudaStreamSynchronize(cs);
        cudaEventDestroy(ev);
        cudaStreamDestroy(cs);
    }
};

double norm2(const double* a, int64_t n, double* partial, cg_state* st_d, cg_state* st_h, cudaStream_t cs)
{
    dot<double>(a, a, n, partial, cs);
    k_cg_init<<<1, kRedThreads, 0, cs>>>(partial, st_d, 0.0, 0);
    ABHSF_CUDA(cudaMemcpyAsync(st_h, st_d, sizeof(cg_state), cudaMemcpyDeviceToHost, cs));
    ABHSF_CUDA(cudaStreamSynchronize(cs));
    return st_h->rr[0];
}

void check_square(const abhsf_matrix& a)
{
    if (a.m != a.n)
        fail(ABHSF_ERROR_INVALID_VALUE, "CG needs a square matrix");
}

}  // namespace

void cg_solve(const abhsf_matrix& a, const double* b, double* x, double rtol, int max_iters, abhsf_cg_info* info,
              cudaStream_t user)
{
    check_square(a);
    const int64_t n = a.n;
    solve_stream ss(user);
    cudaStream_t cs = ss.cs;
    cg_work<double> w(n, cs);
    scratch<double> xn(n, cs), partial(2 * kRedBlocks, cs);
    scratch<cg_state> st_d(1, cs);
    cg_state st_h{};
    const double bb = norm2(b, n, partial.get(), st_d.get(), &st_h, cs);
    residual<double>(a, b, x, w.r.get(), xn.get(), n, cs);
    cg_start<double>(w, n, st_d.get(), partial.get(), rtol * rtol * bb, max_iters, cs);
    cg_graph<double> g(a, x, w, n, st_d.get(), partial.get(), cs);
    const int iters = g.run(st_d.get(), cs);
    residual<double>(a, b, x, w.r.get(), xn.get(), n, cs);
    const double rr = norm2(w.r.get(), n, partial.get(), st_d.get(), &st_h, cs);
    info->iterations = iters;
    info->outer_iterations = 1;
    info->rel_residual = bb > 0.0 ? std::sqrt(rr / bb) : std::sqrt(rr);
    info->converged = info->rel_residual <= rtol ? 1 : 0;
}

void cg_solve_mixed(const abhsf_matrix& a64, const abhsf_matrix& a32, const double* b, double* x, double rtol,
                    int max_iters, double update_factor, int max_updates, abhsf_cg_info* info, cudaStream_t user)
{
    check_square(a64);
    if (a32.m != a64.m || a32.n != a64.n)
        fail(ABHSF_ERROR_INVALID_VALUE, "the two matrices of the mixed solver differ in shape");
    const int64_t n = a64.n;
    const double f2 = update_factor * update_factor;
    solve_stream ss(user);
    cudaStream_t cs = ss.cs;
    scratch<double> r64(n, cs), xn(n, cs), partial(2 * kRedBlocks, cs);
    cg_work<float> w(n, cs);
    scratch<float> d(n, cs);  // the f32 solution since the last update
    scratch<cg_state> st_d(1, cs), st64_d(1, cs);
    cg_state st_h{};
    const double bb = norm2(b, n, partial.get(), st64_d.get(), &st_h, cs);
    const double tol2 = rtol * rtol * bb;
    residual<double>(a64, b, x, r64.get(), xn.get(), n, cs);
    double rr = norm2(r64.get(), n, partial.get(), st64_d.get(), &st_h, cs);
    int iters = 0, updates = 0;
    if (rr > tol2 && max_iters > 0) {
        k_to_f32<<<elem_grid(n), 256, 0, cs>>>(n, r64.get(), w.r.get());
        ABHSF_CUDA(cudaMemsetAsync(d.get(), 0, n * sizeof(float), cs));
        cg_start<float>(w, n, st_d.get(), partial.get(), 0.0, max_iters, cs);
        k_cg_resume<<<1, kRedThreads, 0, cs>>>(partial.get(), st_d.get(), f2);  // partials of r32 . r32
        cg_graph<float> g(a32, d.get(), w, n, st_d.get(), partial.get(), cs);
        for (;;) {
            iters = g.run(st_d.get(), cs);
            // reliable update: fold the f32 solution into x, replace r by b - A x in FP64
            k_fold<<<elem_grid(n), 256, 0, cs>>>(n, x, d.get());
            residual<double>(a64, b, x, r64.get(), xn.get(), n, cs);
            rr = norm2(r64.get(), n, partial.get(), st64_d.get(), &st_h, cs);
            ++updates;
            if (rr <= tol2 || iters >= max_iters || updates >= max_updates)
                break;
            k_to_f32<<<elem_grid(n), 256, 0, cs>>>(n, r64.get(), w.r.get());
            dot<float>(w.r.get(), w.r.get(), n, partial.get(), cs);
            k_cg_resume<<<1, kRedThreads, 0, cs>>>(partial.get(), st_d.get(), f2);
            ABHSF_CUDA(cudaGetLastError());
        }
    }
    info->iterations = iters;
    info->outer_iterations = updates;
    info->rel_residual = bb > 0.0 ? std::sqrt(rr / bb) : std::sqrt(rr);
    info->converged = info->rel_residual <= rtol ? 1 : 0;
}

}  // namespace abhsf
