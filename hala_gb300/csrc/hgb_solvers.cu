// Fused Krylov solvers over the SpMV / ILU kernels.
//
// CG / PCG follow solve_cg_core (hex/solvers/hala_solvers_cg.hpp:92-156) step for step, but the
// scalars never leave the device: <p,Ap> is reduced in the SpMV epilogue, ||r||^2 in the x/r
// update, and the convergence decision is taken on the device.  One iteration is six launches
// (SpMV+dot, update+norm, L solve, U solve, <r,z>, p update); ITERS_PER_GRAPH iterations are
// captured once into a CUDA graph and replayed, every launch of an iteration after convergence
// being a no-op, so the host synchronises once per graph replay instead of three times per
// iteration as the reference does (cublasDdot / cublasDnrm2 in host pointer mode).
#include "hgb_internal.cuh"
#include "hgb_kernels.cuh"
#include "hgb_complex.cuh"

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cmath>
#include <vector>

namespace hgb {

constexpr int kItersPerGraph = 16;

// Elements a thread takes per round in the CG vector kernels, their loads issued together: the
// kernels are short and latency-bound (14 elements per thread at 128^3), so a round's loads are all that one
// memory round trip brings.
template <typename X, int NARR = 2> __host__ __device__ constexpr int ew_unroll() {
    return (sizeof(X) == 8 ? 4 : 8) / (NARR > 2 ? 2 : 1);   // NARR: vectors read or written per element
}
// Two CTAs of 512 threads per SM, and sums and quotients in as few warps as do: an FP64 instruction takes an SM
// quarter's unit for 62 cycles, whichever of the warps repeats it.  With four CTAs of 256 threads each warp summed,
// divided and reduced: 128^3 FP32, from start to start of the launches, the d / r update 21.5 us, <r, z> 18.6; now
// 17 and 13.  (Shapes of 256 to 1,024 threads and 4 to 16 loads a round: the whole mixed solve within 1.5 %.)
constexpr int kEwThreads = 512, kEwCtas = 2;
static inline int vec_grid(const hgb_ctx *c, long n) {
    return (int)std::max<long>(1, std::min<long>((n + kEwThreads - 1) / kEwThreads, (long)c->num_sms * kEwCtas));
}

// The sum of np parts, or the value a grid reduction stored (np == 0), mapped by f in one thread and
// given to all: four warps, one per SM quarter, add the parts.
template <typename F>
__device__ __forceinline__ double vec_scalar(const double *part, int np, double stored, F f) {
    __shared__ double sh[4], res;
    const int tid = threadIdx.x;
    if (np > 0 && tid < 128) {
        double v = 0.0;
        for (int b = tid; b < np; b += 128) v += part[b];
        v = warp_sum(v);
        if ((tid & 31) == 0) sh[tid >> 5] = v;
    }
    __syncthreads();
    if (tid == 0) res = f(np > 0 ? (sh[0] + sh[1]) + (sh[2] + sh[3]) : stored);
    __syncthreads();
    return res;
}

// As grid_sum for NV values of kEwThreads threads: every CTA's part, the last CTA adds them in one order and runs
// fin(sums) in thread 0.  128 threads add four values each before a warp's lanes are added.
template <int NV, bool PARTS = false, typename Fin>
__device__ __forceinline__ void vec_grid_sum(const double (&v)[NV], double *partials, unsigned *counter, Fin fin) {
    __shared__ double sh[NV][kEwThreads], shw[NV][4];
    __shared__ bool last;
    const int tid = threadIdx.x, G = gridDim.x;
    auto finish = [&](double (&t)[NV]) {   // 128 threads' values -> thread 0
        if (tid < 128) {
#pragma unroll
            for (int k = 0; k < NV; k++) {
                t[k] = warp_sum(t[k]);
                if ((tid & 31) == 0) shw[k][tid >> 5] = t[k];
            }
        }
        __syncthreads();
        if (tid == 0) {
#pragma unroll
            for (int k = 0; k < NV; k++) t[k] = (shw[k][0] + shw[k][1]) + (shw[k][2] + shw[k][3]);
        }
    };
    double t[NV];
#pragma unroll
    for (int k = 0; k < NV; k++) sh[k][tid] = v[k];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) t[k] = 0.0;
    if (tid < 128) {
#pragma unroll
        for (int k = 0; k < NV; k++) {
            t[k] = sh[k][tid];
#pragma unroll
            for (int w = 128; w < kEwThreads; w += 128) t[k] += sh[k][tid + w];
        }
    }
    finish(t);
    if (tid == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++) partials[blockIdx.x * NV + k] = t[k];
    }
    if (PARTS) return;   // the parts are the result
    if (tid == 0) {
        __threadfence();
        last = atomicAdd(counter, 1u) == (unsigned)G - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int k = 0; k < NV; k++) t[k] = 0.0;
    if (tid < 128)
        for (int b = tid; b < G; b += 128)
#pragma unroll
            for (int k = 0; k < NV; k++) t[k] += __ldcg(partials + b * NV + k);
    finish(t);
    if (tid == 0) {
        *counter = 0u;
        fin(t);
    }
}

// acc + a x: one fused multiply-add in FP64 (half the unit's time), separately rounded in FP32
__device__ __forceinline__ double vec_axpy(double acc, double a, double x) { return fma(a, x, acc); }
__device__ __forceinline__ float vec_axpy(float acc, float a, float x) { return add_rn(acc, mul_rn(a, x)); }

template <typename X>
__global__ void __launch_bounds__(kEwThreads, kEwCtas) cg_update_kernel(long n, const SolverScalars *__restrict__ s_in, SolverScalars *s,
                                 const X *__restrict__ p, const X *__restrict__ Ap, X *__restrict__ x,
                                 X *__restrict__ r, double *partials, unsigned *counter, const double *pap_part,
                                 int pap_n) {
    if (s_in->done) return;
    constexpr int U = ew_unroll<X, 4>();
    const long T = (long)gridDim.x * blockDim.x;
    long base = blockIdx.x * (long)blockDim.x + threadIdx.x;
    X pv[U], av[U], xv[U], rv[U];
    auto load = [&] {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = base + u * T;
            if (i < n) {
                pv[u] = p[i];
                av[u] = Ap[i];
                xv[u] = x[i];
                rv[u] = r[i];
            }
        }
    };
    load();   // in flight while the scalar is summed
    // a = <r,z> / <p,Ap>; x += a p; r -= a Ap  (axpy(a,p,x), axpy(-a,Ap,r))
    double pap = 0.0;   // thread 0's
    const X a = (X)vec_scalar(pap_part, pap_n, s_in->pap, [&](double v) { pap = v; return s_in->nzr / v; });
    const X ma = -a;
    DotAcc<X> rr;
    while (base < n) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = base + u * T;
            if (i < n) {
                x[i] = vec_axpy(xv[u], a, pv[u]);
                const X ri = vec_axpy(rv[u], ma, av[u]);
                r[i] = ri;
                rr.add(ri, ri);
            }
        }
        base += T * U;
        load();
    }
    double acc[1] = {rr.get()};
    vec_grid_sum<1>(acc, partials, counter, [&](double (&v)[1]) {
        s->pap = pap;
        s->zr = s->nzr;
        s->rr = v[0];
        s->it += 1;
        s->done = (s->it >= s->max_iter) || (v[0] < s->tol2) || !(v[0] == v[0]);
    });
}

// <r, z>.  In the loop (RZ_PARTS) every CTA leaves its part and the direction update sums them: no last CTA holds the
// launch up.  Before it, one launch stores the first <r, z> (RZ_FIRST), and for the plain CG ||r||^2 with it (RZ_INIT).
enum RzMode { RZ_PARTS, RZ_FIRST, RZ_INIT };
template <typename X, RzMode MODE>
__global__ void __launch_bounds__(kEwThreads, kEwCtas) cg_rz_kernel(long n, SolverScalars *s, const X *__restrict__ r, const X *__restrict__ z,
                             double *partials, unsigned *counter) {
    if (MODE == RZ_PARTS && s->done) return;
    DotAcc<X> rz, rr;
    constexpr int U = ew_unroll<X>();
    const long T = (long)gridDim.x * blockDim.x;
    for (long base = blockIdx.x * (long)blockDim.x + threadIdx.x; base < n; base += T * U) {
        X rv[U], zv[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = base + u * T;
            if (i < n) {
                rv[u] = r[i];
                zv[u] = z[i];
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            if (base + u * T < n) {
                rz.add(rv[u], zv[u]);
                if (MODE == RZ_INIT) rr.add(rv[u], rv[u]);
            }
        }
    }
    constexpr int NV = MODE == RZ_INIT ? 2 : 1;
    double acc[NV] = {rz.get()};
    if (MODE == RZ_INIT) acc[NV - 1] = rr.get();
    vec_grid_sum<NV, MODE == RZ_PARTS>(acc, partials, counter, [&](double (&v)[NV]) {
        s->zr = s->nzr = v[0];
        if (MODE == RZ_INIT) {
            s->rr = v[NV - 1];
            s->r0 = sqrt(v[NV - 1]);
            if (s->rel > 0.0) {
                double t = s->rel * s->r0;
                s->tol2 = fmax(s->tol2, t * t);
            }
        }
    });
}

// p = (zr_new / zr_old) p + z   (scal(a, p); axpy(1, z, p)); the new <r, z> from its parts, one per CTA of a grid as large
template <typename X>
__global__ void __launch_bounds__(kEwThreads, kEwCtas) cg_p_kernel(long n, SolverScalars *s, X *__restrict__ p, const X *__restrict__ z,
                                                                    const double *rz_part) {
    if (s->done) return;
    constexpr int U = ew_unroll<X, 3>();
    const long T = (long)gridDim.x * blockDim.x;
    long base = blockIdx.x * (long)blockDim.x + threadIdx.x;
    X pv[U], zv[U];
    auto load = [&] {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = base + u * T;
            if (i < n) {
                pv[u] = p[i];
                zv[u] = z[i];
            }
        }
    };
    load();   // in flight while the scalar is summed
    const X bta = (X)vec_scalar(rz_part, gridDim.x, 0.0, [&](double nzr) {
        if (blockIdx.x == 0) s->nzr = nzr;   // the others read zr only
        return nzr / s->zr;
    });
    while (base < n) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = base + u * T;
            if (i < n) p[i] = vec_axpy(zv[u], bta, pv[u]);
        }
        base += T * U;
        load();
    }
}

__global__ void cg_init_kernel(SolverScalars *s, double tol2, double rel, int max_iter) {
    s->it = 1;
    s->done = 0;
    s->max_iter = max_iter;
    s->tol2 = tol2;
    s->rel = rel;
    s->zr = 0.0;
    s->nzr = 0.0;
    s->pap = 0.0;
    s->rr = 0.0;
}

template <typename X>
__global__ void copy_kernel(long n, const X *__restrict__ a, X *__restrict__ b) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) b[i] = a[i];
}

__global__ void f64_to_f32_kernel(long n, const double *__restrict__ a, float *__restrict__ b) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) b[i] = (float)a[i];
}

__global__ void add_f32_to_f64_kernel(long n, const float *__restrict__ d, double *__restrict__ x) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) x[i] += (double)d[i];
}

__global__ void zero_f32_kernel(long n, float *d) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) d[i] = 0.0f;
}

// r = b - A x in FP64 and ||r||^2 -> result slot (the refinement residual)
__global__ void residual_norm_kernel(long n, const double *__restrict__ r, double *partials, unsigned *counter,
                                     double *out) {
    double acc[1] = {0.0};
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        acc[0] = fma(r[i], r[i], acc[0]);
    grid_sum<1>(acc, partials, counter, [&](double (&v)[1]) { *out = v[0]; });
}

static inline int ew_grid(hgb_ctx *c, long n) {
    return std::max(1, (int)std::min<long>((n + 255) / 256, (long)c->num_sms * 4));
}

// Workspace of one fused CG run (X = vector type).
template <typename X>
struct CgWork {
    X *r = nullptr, *z = nullptr, *p = nullptr, *Ap = nullptr;
    hgb_ctx *c = nullptr;
    int alloc(hgb_ctx *ctx, long n, bool need_z) {
        c = ctx;
        if (ws_alloc(c, &r, n) || ws_alloc(c, &p, n) || ws_alloc(c, &Ap, n) || (need_z && ws_alloc(c, &z, n)))
            return cuda_fail(cudaErrorMemoryAllocation, "cg workspace");
        return HGB_OK;
    }
    void release() {
        if (!c) return;
        ws_free(c, r);
        ws_free(c, z);
        ws_free(c, p);
        ws_free(c, Ap);
    }
};

// y = alpha op(A) x + beta y with an optional fused <x, y>: into *dot, or (nparts, 'N' only) as
// per-CTA parts left for the consuming kernel (*nparts: their count; 0 when *dot was written)
template <typename V, typename X>
static int spmv_A(hgb_ctx *c, hgb_csr *A, X alpha, const X *x, X beta, X *y, double *dot, const int *skip,
                  bool trans = false, int *nparts = nullptr) {
    if (trans) {
        if (nparts) *nparts = 0;
        return spmv_t_fused_launch<V>(A, alpha, x, beta, y, x, dot, skip);
    }
    return spmv_n_launch<V>(c, csr_rows(A), csr_size(A), csr_pntr(A), csr_indx(A), (const V *)csr_vals(A), alpha, x, beta, y,
                            nparts ? nullptr : dot, skip, nparts);
}
template <>
int spmv_A<uint16_t, float>(hgb_ctx *c, hgb_csr *A, float alpha, const float *x, float beta, float *y, double *dot,
                           const int *skip, bool trans, int *nparts) {
    if (trans) return fail(HGB_ERR_UNSUPPORTED, "transposed product of a bf16 matrix");
    return spmv_n_launch<uint16_t>(c, csr_rows(A), csr_size(A), csr_pntr(A), csr_indx(A), (const uint16_t *)csr_vals(A), alpha, x,
                                   beta, y, nparts ? nullptr : dot, skip, nparts);
}

// One CG iteration: the launches captured into the graph.
template <typename V, typename X>
static int cg_iteration(hgb_ctx *c, hgb_csr *A, hgb_ilu *M, CgWork<X> &w, X *x, long n, bool trans) {
    SolverScalars *s = c->scal;
    const int *done = &s->done;
    int np = 0;
    HGB_TRY(spmv_A<V, X>(c, A, X(1), w.p, X(0), w.Ap, &s->pap, done, trans, &np));
    cg_update_kernel<X><<<vec_grid(c, n), kEwThreads, 0, c->stream>>>(n, s, s, w.p, w.Ap, x, w.r, c->partials,
                                                                           c->counter, c->partials + kSpmvPartsOffset, np);
    X *z = M ? w.z : w.r;
    if (M) HGB_TRY(ilu_apply_internal(M, trans ? 'T' : 'N', w.r, w.z, done));
    cg_rz_kernel<X, RZ_PARTS><<<vec_grid(c, n), kEwThreads, 0, c->stream>>>(n, s, w.r, z, c->partials, c->counter);
    cg_p_kernel<X><<<vec_grid(c, n), kEwThreads, 0, c->stream>>>(n, s, w.p, z, c->partials);
    return launch_check("cg iteration");
}

// ------------------------------------------------------------------ persistent CG -------
// Unpreconditioned CG on a system whose matrix and vectors stay in L2 (the 256^2 Poisson class):
// there the graph-replayed iteration is bound by its launches and their reductions' tails
// (about 27 us per iteration for six launches), not by bytes.  One cooperative launch runs up to
// kCgpChunk iterations.  Every CTA keeps its rows for the whole launch.  What bounds an iteration is the latency of
// its exchanges between CTAs and of FP64 instructions (each holds an SM quarter's unit for 62 cycles), so
// it has one reduction (after Chronopoulos and Gear's form of the method):
//   x += a p, r -= a q                       (q = A p)
//   s = A r, with the neighbours' r taken as they arrive (below); one reduction of <r, r>, <r, s>, <r, q> + <p, s>, <p, q>
//   b = <r, r> / <r, r>_old, <p', q'> = <r, s> + b (<r, q> + <p, s>) + b^2 <p, q>, a = <r, r> / <p', q'>
//   p' = r + b p, q' = s + b q
// That is <p', q'> of the vectors as they are, whatever became of the residuals' orthogonality (the shorter form of the
// method, <r, s> - b <r, r> / a, relies on it: 18 % more iterations on a 300-point biharmonic operator to 1e-13, 22 % on a
// spectrum over 13 decades).  Where the terms cancel to less than a quarter of <r, s>, more than two bits, the CTAs sum
// <p', q'> itself in a second reduction; on Poisson operators it stays near a half.  FP32 vectors and the rows in memory
// (RPT = 0) always take that second reduction: the first has only <r, r>.  A launch starts with q = A p and <p, q> itself.
// Every CTA sums all CTAs' parts in the same order, so every CTA takes the same decision with the same bits.  Rounding
// differs from the graph path's, so the iteration count can differ from it.  Every wait is bounded: one that
// runs out of polls sets DEV_ERR_TIMEOUT and every CTA returns.
// Per iteration, in two reductions by a counter that every CTA polls, and so: 24x24 7.1 -> 4.4 us, 256^2
// 9.5 -> 6.4, 300^2 15.4 -> 8.7, 500^2 21.4 -> 15.5; FP32 256^2 8.3 -> 8.1.  (With the shorter form 256^2 took 5.9, 300^2 7.3: two
// sums fewer.  Of its 12,000 cycles at 256^2 the mail took 2100, the neighbours' r 1300 to 2300, FP64 instructions of the rows
// 3100, and the sums with one division 5000.)
constexpr int kCgpThreads = 256;
constexpr int kCgpChunk = 4096;                 // iterations per launch
constexpr long kCgpMaxRows = 1L << 20;          // larger systems take the graph path
constexpr size_t kCgpMaxBytes = 48u << 20;      // matrix + vectors resident in L2 (129 MB)
constexpr int kCgpCluster = 8;                  // CTAs of a cluster at most (8, 4 or 2)
constexpr int kCgpLead = 4;                     // the warp that posts and polls
constexpr unsigned kCgpClusters = 64;           // clusters at most: mail entries of a sum
constexpr int kCgpSums = 4;                     // sums of a reduction at most

// acc += v * x: separately rounded (the exact SpMV mode) or one fused multiply-add
template <bool EXACT, typename X>
__device__ __forceinline__ X cgp_acc(X acc, X v, X x) {
    return EXACT ? add_rn(acc, mul_rn(v, x)) : fma(v, x, acc);
}
__device__ __forceinline__ void cgp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cgp_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// A value and the number of its step, complete when the number is right: 64-bit words are written whole, so a
// double goes as two words of half the value and the number each, whatever the order in which they arrive,
// and value and arrival come with one load.
struct CgpWord {
    unsigned long long x, y;
};
__device__ __forceinline__ CgpWord cgp_tag(double v, unsigned number) {
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v), n = (unsigned long long)number << 32;
    return {n | (bits & 0xffffffffu), n | (bits >> 32)};
}
__device__ __forceinline__ bool cgp_whole(const CgpWord &w, unsigned number, double &v) {
    v = __longlong_as_double((long long)(w.y << 32 | (w.x & 0xffffffffu)));
    return (unsigned)(w.x >> 32) == number && (unsigned)(w.y >> 32) == number;
}
__device__ __forceinline__ void cgp_store(CgpWord *p, const CgpWord &w) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(w.x), "l"(w.y) : "memory");
}
__device__ __forceinline__ CgpWord cgp_load(const CgpWord *p) {
    CgpWord w;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "l"(p) : "memory");
    return w;
}
// the tagged residual: 16 bytes an FP64 entry, 8 an FP32 one
template <typename X> struct CgpR;
template <> struct CgpR<double> {
    using T = CgpWord;
    static __device__ __forceinline__ void put(T *p, double v, unsigned number) { cgp_store(p, cgp_tag(v, number)); }
    static __device__ __forceinline__ bool get(const T *p, unsigned number, double &v) { return cgp_whole(cgp_load(p), number, v); }
};
template <> struct CgpR<float> {
    using T = unsigned long long;
    static __device__ __forceinline__ void put(T *p, float v, unsigned number) {
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((unsigned long long)number << 32 | __float_as_uint(v)) : "memory");
    }
    static __device__ __forceinline__ bool get(const T *p, unsigned number, float &v) {
        T w;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
        v = __uint_as_float((unsigned)w);
        return (unsigned)(w >> 32) == number;
    }
};
// false when the wait is over its bound, or another CTA's was
__device__ __forceinline__ bool cgp_wait_on(int &spins, const int *err) {
    if (++spins > kSpinLimit) return false;
    return (spins & 1023) != 0 || !(*(const volatile int *)err & DEV_ERR_TIMEOUT);
}

// A reduction of up to kCgpSums sums: the CTAs of a cluster exchange theirs through distributed shared memory, then the CTAs of
// equal rank exchange the clusters' through mailboxes in memory (every CTA has its own, one entry per cluster).
// 256^2, 128 CTAs: 2100 cycles for the mail, where 128 CTAs polling one set of entries waited 6500 and each its own
// mailbox of 128 entries 5000.  Two sets of entries take turns: a CTA posts to a set again only after every CTA
// has posted to the other one, which each does after reading this one.
// The sums are shaped to have few FP64 instructions in a row: the upper four warps' values are folded into the
// lower four (one per quarter), whose lanes then add one of the NV sums each, a group of 32 / NV lanes a sum, here
// and in the steps after it; the lead warp adds the warps' sums, posts, polls, and adds the rest in one order, the same
// bits in every CTA.
struct CgpShared {
    CgpWord peer[2][kCgpCluster][kCgpSums];
    double fold[kCgpSums][kCgpThreads / 2], warp[4 * kCgpSums], sum, alpha, beta;
    int ok, again;
};
__device__ __forceinline__ double cgp_add_xor(double v, int o) { return v + __shfl_xor_sync(0xffffffffu, v, o); }
// All threads call it.  ORDER: what every CTA wrote before is in memory for all after the caller's next barrier.
// meanwhile(): the lead warp's work between posting and polling.  The lead warp gets the sums;
// false when a wait ran out.
template <bool ORDER, int NV, typename F>
__device__ __forceinline__ bool cgp_exchange(double (&v)[NV], unsigned number, CgpWord *mail, int *err, CgpShared &sh, F meanwhile,
                                             double (&sum)[NV]) {
    constexpr unsigned G = 32 / NV;   // lanes of a sum
    static_assert(G >= kCgpCluster && NV <= kCgpSums, "a lane per peer");
    const int tid = threadIdx.x, wid = tid >> 5, set = number & 1;
    const unsigned lane = tid & 31, own = lane / G, at = lane % G;
    if (tid >= kCgpThreads / 2) {
#pragma unroll
        for (int j = 0; j < NV; j++) sh.fold[j][tid - kCgpThreads / 2] = v[j];
    }
    __syncthreads();
    if (tid < kCgpThreads / 2) {
#pragma unroll
        for (int j = 0; j < NV; j++) v[j] += sh.fold[j][tid];
#pragma unroll
        for (int h = NV / 2, o = 16; h > 0; h >>= 1, o >>= 1)   // each step leaves a lane half of its sums
#pragma unroll
            for (int j = 0; j < h; j++) {
                const double keep = lane & o ? v[j + h] : v[j], send = lane & o ? v[j] : v[j + h];
                v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) v[0] = cgp_add_xor(v[0], o);
        if (at == 0) sh.warp[own * 4 + wid] = v[0];
    } else if (ORDER && wid == kCgpLead) {
        cgp_fence();   // the CTA's writes, ordered before this by the barrier, before the posts below
    }
    __syncthreads();
    if (wid != kCgpLead) return true;
    unsigned rank, size, clusters;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(clusters));
    double t = sh.warp[own * 4 + (lane & 3)];
    t = cgp_add_xor(cgp_add_xor(t, 1), 2);
    if (at < size) {
        unsigned to;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"((unsigned)__cvta_generic_to_shared(&sh.peer[set][rank][own])), "r"(at));
        const CgpWord w = cgp_tag(t, number);
        asm volatile("st.relaxed.cluster.shared::cluster.v2.u64 [%0], {%1, %2};" ::"r"(to), "l"(w.x), "l"(w.y) : "memory");
    }
    const unsigned from = (unsigned)__cvta_generic_to_shared(&sh.peer[set][at & (size - 1)][own]);
    for (int spins = 0;;) {
        CgpWord w;
        asm volatile("ld.relaxed.cluster.shared::cta.v2.u64 {%0, %1}, [%2];" : "=l"(w.x), "=l"(w.y) : "r"(from) : "memory");
        if (__all_sync(0xffffffffu, cgp_whole(w, number, t))) break;
        if (__any_sync(0xffffffffu, !cgp_wait_on(spins, err))) return false;
    }
    for (unsigned o = 1; o < size; o *= 2) t = cgp_add_xor(t, o);
    if (ORDER) cgp_fence();   // what the peers ordered before their posts, before this CTA's
    if (clusters > 1) {
        mail += (size_t)set * gridDim.x * clusters * kCgpSums;
        for (unsigned k = at; k < clusters; k += G)
            cgp_store(mail + ((size_t)(k * size + rank) * clusters + blockIdx.x / size) * kCgpSums + own, cgp_tag(t, number));
    }
    meanwhile();
    if (clusters > 1) {
        constexpr int Q = kCgpClusters / G;   // entries a lane reads
        mail += (size_t)blockIdx.x * clusters * kCgpSums + own;
        double part[Q];
        for (int spins = 0;;) {
            bool here = true;
#pragma unroll
            for (int q = 0; q < Q; q++) {
                CgpWord w = {(unsigned long long)number << 32, (unsigned long long)number << 32};   // whole, and zero
                if (G * q + at < clusters) w = cgp_load(mail + kCgpSums * (G * q + at));
                here = cgp_whole(w, number, part[q]) && here;
            }
            if (__all_sync(0xffffffffu, here)) break;
            if (__any_sync(0xffffffffu, !cgp_wait_on(spins, err))) return false;
        }
        if (ORDER) cgp_fence();
        t = part[0];
#pragma unroll
        for (int q = 1; q < Q; q++) HGB_UNIFORM_IF(clusters > G * q) t += part[q];
        for (unsigned o = 1; o < clusters && o < G; o *= 2) t = cgp_add_xor(t, o);
    }
#pragma unroll
    for (int j = 0; j < NV; j++) sum[j] = __shfl_sync(0xffffffffu, t, j * G);
    return true;
}
// RPT > 0: a CTA owns RPT * 256 consecutive rows (RPT: 1, 2 or 4 per thread) for the whole launch and keeps their
// x, r, p, q and (rows of at most kCgpMaxE entries) their matrix entries in registers; r goes to shared memory for the
// CTA's own rows and to memory tagged with the iteration for the others', and a row's sum waits for its neighbours'
// entries alone.  RPT = 0: the rows are walked with grid-stride loops and every vector lives in memory (systems too
// large for one register-resident row set; rt is not used); a reduction orders the writes of r before the products.
constexpr int kCgpMaxE = 8;

template <typename V, typename X, bool EXACT, int RPT>
__global__ void __launch_bounds__(kCgpThreads, RPT == 0 ? 4 : 1)
cg_persistent_kernel(long n, const int *__restrict__ pntr, const int *__restrict__ indx, const V *__restrict__ vals,
                     X *x, X *r, X *p, X *Ap, typename CgpR<X>::T *rt, SolverScalars *s, CgpWord *mail, int *err) {
    __shared__ CgpShared sh;
    __shared__ X own[RPT > 0 ? RPT * kCgpThreads : 1];   // r of the CTA's rows
    const int G = gridDim.x;
    if (s->done) return;   // the whole grid
    double zr = s->zr, rrv = s->rr, alpha = 0.0, beta = 0.0;
    int it = s->it;
    const int max_iter = s->max_iter;
    const double tol2 = s->tol2;
    const long t0 = (long)blockIdx.x * blockDim.x + threadIdx.x, stride = (long)G * blockDim.x;
    const int first = blockIdx.x * RPT * kCgpThreads;   // the CTA's rows (RPT > 0)
    unsigned number = 0;   // of the last exchange
    bool done = false, good = true;
    const bool lead = threadIdx.x >> 5 == kCgpLead;
    if (threadIdx.x == 0) sh.ok = 1;
    if (threadIdx.x < 2 * kCgpCluster * kCgpSums) (&sh.peer[0][0][0])[threadIdx.x] = CgpWord{0, 0};
    cgp_cluster_sync();   // before a peer's first post
    constexpr bool ONE = sizeof(X) == 8 && RPT > 0;   // one reduction per iteration, or two where it takes a second
    constexpr int K = RPT > 0 ? RPT : 1;
    long row[K];
    int beg[K], len[K], most[K], ci[K][kCgpMaxE];
    X cv[K][kCgpMaxE], xv[K][kCgpMaxE], xr[K], rr[K], pr[K], qr[K], sr[K];
    if (RPT > 0) {
#pragma unroll
        for (int k = 0; k < K; k++) {
            row[k] = first + k * kCgpThreads + threadIdx.x;
            len[k] = 0;
            beg[k] = 0;
            xr[k] = rr[k] = pr[k] = qr[k] = sr[k] = X(0);
            if (row[k] < n) {
                beg[k] = pntr[row[k]];
                len[k] = pntr[row[k] + 1] - beg[k];
                xr[k] = x[row[k]];
                rr[k] = r[row[k]];
                pr[k] = p[row[k]];
#pragma unroll
                for (int e = 0; e < kCgpMaxE; e++)
                    if (e < len[k]) {
                        ci[k][e] = indx[beg[k] + e];   // below: -1 - its place among the CTA's own rows
                        cv[k][e] = Val<V>::get(vals[beg[k] + e]);
                    }
            }
            most[k] = __reduce_max_sync(0xffffffffu, len[k] <= kCgpMaxE ? len[k] : 0);
        }
    }
    // row k of this thread (RPT > 0) times the vector whose entries are in xv, or far(column) for longer rows
    auto row_product = [&](int k, auto far) -> X {
        X acc = X(0);
        auto term = [&](int e) {
            if (len[k] <= kCgpMaxE && e < len[k]) acc = cgp_acc<EXACT, X>(acc, cv[k][e], xv[k][e]);
        };
        term(0), term(1), term(2);
        HGB_UNIFORM_IF(most[k] > 3) term(3);
        HGB_UNIFORM_IF(most[k] > 4) term(4);
        HGB_UNIFORM_IF(most[k] > 5) { term(5); term(6); term(7); }
        if (len[k] > kCgpMaxE)
            for (int j = beg[k]; j < beg[k] + len[k]; j++) acc = cgp_acc<EXACT, X>(acc, Val<V>::get(vals[j]), far(indx[j]));
        return acc;
    };
    // row i (RPT = 0) times v, whose entries other CTAs wrote during this launch (__ldcg: from L2)
    auto memory_product = [&](long i, const X *v) -> X {
        X acc = X(0);
        for (int j = pntr[i]; j < pntr[i + 1]; j++) acc = cgp_acc<EXACT, X>(acc, Val<V>::get(vals[j]), __ldcg(v + indx[j]));
        return acc;
    };
    // The lead warp's last step: b = sum / den0 and a = sum / den1, one division in two lanes; then every thread's
    auto finish = [&](bool ok, double sum, double den0, double den1, bool second = false) {
        if (lead) {
            const double q = sum / (threadIdx.x & 1 ? den1 : den0);
            if ((threadIdx.x & 31) == 0) {
                if (!ok) sh.ok = 0;
                sh.sum = sum;
                sh.beta = q;
                sh.again = second;
            }
            if ((threadIdx.x & 31) == 1) sh.alpha = q;
        }
        __syncthreads();
        alpha = (double)(X)sh.alpha;
        beta = sh.beta;
        good = sh.ok != 0;
    };
    auto nothing = [] {};
    double sum[2] = {0.0, 0.0};
    // one sum of the whole grid, to the lead warp
    auto exchange = [&](double v) {
        number++;
        double two[2] = {v, 0.0};
        return cgp_exchange<false>(two, number, mail, err, sh, nothing, sum);
    };
    // q = A p for the direction the launch starts from, and a = <r, r> / <p, q>
    {
        DotAcc<X> pq;
        if (RPT > 0) {
#pragma unroll
            for (int k = 0; k < K; k++) {
#pragma unroll
                for (int e = 0; e < kCgpMaxE; e++)
                    if (len[k] <= kCgpMaxE && e < len[k]) {
                        xv[k][e] = __ldcg(p + ci[k][e]);
                        const int at = ci[k][e] - first;
                        if (at >= 0 && at < RPT * kCgpThreads) ci[k][e] = -1 - at;
                    }
                qr[k] = row_product(k, [&](int c) { return __ldcg(p + c); });
                pq.add(pr[k], qr[k]);
            }
        } else {
            for (long i = t0; i < n; i += stride) {
                const X q = memory_product(i, p);
                Ap[i] = q;
                pq.add(p[i], q);
            }
        }
        const bool ok = exchange(pq.get());
        finish(ok, zr, 1.0, sum[0]);
    }
    for (int c = 0; c < kCgpChunk && good; c++) {
        const X a = (X)alpha, ma = -a, bta = (X)beta;
        const bool next = ONE && c > 0;   // p and q of this direction are still to be formed
        DotAcc<X> rrd, rsd, crd, pqd;   // <r, r>, <r, s>, <r, q> + <p, s>, <p, q>
        if (RPT > 0) {
            const unsigned tag = c + 1;
            X was[K];   // r first: the others wait for it
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (next) qr[k] = cgp_acc<EXACT, X>(sr[k], bta, qr[k]);
                was[k] = rr[k];
                rr[k] = cgp_acc<EXACT, X>(rr[k], ma, qr[k]);
                own[k * kCgpThreads + threadIdx.x] = rr[k];
                if (row[k] < n) CgpR<X>::put(rt + row[k], rr[k], tag);
            }
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (next) pr[k] = cgp_acc<EXACT, X>(was[k], bta, pr[k]);
                xr[k] = cgp_acc<EXACT, X>(xr[k], a, pr[k]);
                rrd.add(rr[k], rr[k]);
                if (ONE) {
                    crd.add(rr[k], qr[k]);
                    pqd.add(pr[k], qr[k]);
                }
            }
            __syncthreads();
            // the neighbours' r: the whole warp waits as one (lanes leaving a loop one by one would stay apart)
            constexpr int KG = K < 2 ? K : 2;   // rows with their loads in flight together (registers)
#pragma unroll
            for (int kb = 0; kb < K; kb += KG) {
                for (int spins = 0;;) {
                    bool here = true;
#pragma unroll
                    for (int k = kb; k < kb + KG; k++)
#pragma unroll
                        for (int e = 0; e < kCgpMaxE; e++)
                            if (len[k] <= kCgpMaxE && e < len[k]) {
                                if (ci[k][e] >= 0) here = CgpR<X>::get(rt + ci[k][e], tag, xv[k][e]) && here;
                                else xv[k][e] = own[-1 - ci[k][e]];
                            }
                    if (__all_sync(0xffffffffu, here)) break;
                    if (__any_sync(0xffffffffu, !cgp_wait_on(spins, err))) {
                        sh.ok = 0;
                        break;
                    }
                }
#pragma unroll
                for (int k = kb; k < kb + KG; k++) {
                    sr[k] = row_product(k, [&](int col) {
                        X v;
                        for (int spins = 0; !CgpR<X>::get(rt + col, tag, v);)
                            if (!cgp_wait_on(spins, err)) {
                                sh.ok = 0;
                                break;
                            }
                        return v;
                    });
                    if (ONE) {
                        rsd.add(rr[k], sr[k]);
                        crd.add(pr[k], sr[k]);
                    }
                }
            }
        } else {
            for (long i = t0; i < n; i += stride) {
                x[i] = cgp_acc<EXACT, X>(x[i], a, p[i]);
                const X ri = cgp_acc<EXACT, X>(r[i], ma, Ap[i]);
                r[i] = ri;
                rrd.add(ri, ri);
            }
            number++;
            double two[2] = {rrd.get(), 0.0};
            const bool ok = cgp_exchange<true>(two, number, mail, err, sh, nothing, sum);
            finish(ok, sum[0], zr, 1.0);
            if (!good) break;
        }
        if (ONE) {
            number++;
            double four[4] = {rrd.get(), rsd.get(), crd.get(), pqd.get()}, s4[4] = {0.0, 0.0, 0.0, 0.0}, inv = 0.0;
            const bool ok = cgp_exchange<false>(four, number, mail, err, sh, [&] { inv = 1.0 / zr; }, s4);
            const double b = s4[0] * inv, pq = fma(b, fma(b, s4[3], s4[2]), s4[1]);
            finish(ok, s4[0], zr, pq, !(4.0 * pq > s4[1]));
            if (!good) break;
        } else if (RPT > 0) {
            const bool ok = exchange(rrd.get());
            finish(ok, sum[0], zr, 1.0);
            if (!good) break;
        }
        rrv = sh.sum;
        it++;
        done = (it >= max_iter) || (rrv < tol2) || !(rrv == rrv);
        if (done) break;
        zr = rrv;
        if (!ONE || sh.again) {   // the same in every CTA
            const X bt = (X)beta;
            const double beta_was = beta;
            DotAcc<X> pq;
            if (RPT > 0) {
#pragma unroll
                for (int k = 0; k < K; k++) {
                    const X pn = cgp_acc<EXACT, X>(rr[k], bt, pr[k]), qn = cgp_acc<EXACT, X>(sr[k], bt, qr[k]);
                    pq.add(pn, qn);
                    if (!ONE) {   // else formed with the next update
                        pr[k] = pn;
                        qr[k] = qn;
                    }
                }
            } else {
                for (long i = t0; i < n; i += stride) {
                    const X pi = cgp_acc<EXACT, X>(r[i], bt, p[i]);
                    const X qi = cgp_acc<EXACT, X>(memory_product(i, r), bt, Ap[i]);
                    p[i] = pi;
                    Ap[i] = qi;
                    pq.add(pi, qi);
                }
            }
            const bool ok = exchange(pq.get());
            finish(ok, zr, 1.0, sum[0]);
            beta = beta_was;
        }
    }
    if (ONE && good && !done) {   // the chunk's end: the next launch starts from this direction
        const X bt = (X)beta;
#pragma unroll
        for (int k = 0; k < K; k++) pr[k] = cgp_acc<EXACT, X>(rr[k], bt, pr[k]);
    }
    cgp_cluster_sync();   // no CTA ends before its peers' last posts to it
    if (!good) {
        if (threadIdx.x == 0) atomicOr(err, DEV_ERR_TIMEOUT);
        return;
    }
    if (RPT > 0) {
#pragma unroll
        for (int k = 0; k < K; k++)
            if (row[k] < n) {
                x[row[k]] = xr[k];
                r[row[k]] = rr[k];
                p[row[k]] = pr[k];
            }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        s->it = it;
        s->rr = rrv;
        s->nzr = s->zr;
        s->zr = zr;
        s->done = done ? 1 : 0;
    }
}

template <typename V, typename X, bool EXACT>
static const void *cgp_kernel(int rpt) {
    return rpt == 1   ? (const void *)cg_persistent_kernel<V, X, EXACT, 1>
           : rpt == 2 ? (const void *)cg_persistent_kernel<V, X, EXACT, 2>
           : rpt == 4 ? (const void *)cg_persistent_kernel<V, X, EXACT, 4>
                      : (const void *)cg_persistent_kernel<V, X, EXACT, 0>;
}

static cudaLaunchConfig_t cgp_config(int grid, int cluster, cudaStream_t stream, cudaLaunchAttribute (&at)[2]) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeCooperative;
    at[1].val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kCgpThreads);
    cfg.stream = stream;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    return cfg;
}

// Launch shape of the persistent CG: {grid, rows per thread (0: grid-stride)}; grid 0 when no
// co-resident grid exists.  Every row of a thread is one more serial stretch of its phase, so as few rows per
// thread as the co-resident clusters at one CTA per SM hold: one, two or four; else grid-stride loops.
// Clusters of eight, or of four or two where more CTAs are needed than clusters of eight fit (15, 36 and 76 of them on
// 152 SMs).  256^2: 5.9 us per iteration with two rows per thread on 128 CTAs, 9.9 (of an earlier form at 7.4) with four on 64.
struct CgpShape {
    int grid = 0, rpt = 0, cluster = 0;
};
template <typename V, typename X, bool EXACT>
static CgpShape cgp_shape(const hgb_ctx *c, long n) {
    static std::atomic<int> fit[64][5][kCgpCluster + 1];   // co-resident clusters + 1, by device, rows per thread, size
    CgpShape sh;
    if (c->device < 0 || c->device >= 64) return sh;
    for (int rpt : {1, 2, 4, 0})
        for (int cluster = kCgpCluster; cluster > 1; cluster /= 2) {
            std::atomic<int> &known = fit[c->device][rpt][cluster];
            int clusters = known.load() - 1;
            if (clusters < 0) {
                cudaLaunchAttribute at[2];
                const cudaLaunchConfig_t cfg = cgp_config(cluster, cluster, nullptr, at);
                if (cudaOccupancyMaxActiveClusters(&clusters, cgp_kernel<V, X, EXACT>(rpt), &cfg) != cudaSuccess) {
                    cudaGetLastError();
                    return sh;
                }
                known = clusters + 1;
            }
            clusters = std::min(clusters, (int)kCgpClusters);
            const long rows = (rpt ? rpt : 4) * (long)kCgpThreads * cluster;   // of a cluster
            const long want = (n + rows - 1) / rows;
            if (clusters < 1 || (rpt && want > clusters)) continue;
            sh.grid = (int)std::min<long>(want, clusters) * cluster;
            sh.rpt = rpt;
            sh.cluster = cluster;
            return sh;
        }
    return sh;
}

template <typename V, typename X>
static bool cgp_eligible(hgb_csr *A, hgb_ilu *M, bool trans) {
    const long n = csr_rows(A);
    const size_t bytes = (size_t)csr_nnz(A) * (sizeof(V) + 4) + (size_t)(n + 1) * 4 + (size_t)n * sizeof(X) * 5;
    return !M && !trans && n > 0 && n <= kCgpMaxRows && bytes <= kCgpMaxBytes;
}

// Runs the loop of an initialised CgWork (r, p, the scalars' zr / it / tol2) to the end.
template <typename V, typename X>
static int cgp_run(hgb_ctx *c, hgb_csr *A, CgWork<X> &w, X *x, long n, long long *launches, SolverScalars &hs) {
    const bool exact = (c->spmv_mode == HGB_SPMV_EXACT);
    const CgpShape sh = exact ? cgp_shape<V, X, true>(c, n) : cgp_shape<V, X, false>(c, n);
    const int G = sh.grid;
    if (G < 1) return fail(HGB_ERR_UNSUPPORTED, "persistent cg: no co-resident grid");
    CgpWord *mail = nullptr;   // two sets of an entry (kCgpSums words) per CTA and cluster
    typename CgpR<X>::T *rt = nullptr;
    const size_t nmail = 2 * (size_t)G * (G / sh.cluster) * kCgpSums;
    int st = HGB_OK;
    if (ws_alloc(c, &mail, nmail) || ws_alloc(c, &rt, n)) st = cuda_fail(cudaErrorMemoryAllocation, "persistent cg");
    const int *pntr = csr_pntr(A), *indx = csr_indx(A);
    const V *vals = (const V *)csr_vals(A);
    SolverScalars *s = c->scal;
    int *err = c->err;
    X *r = w.r, *p = w.p, *Ap = w.Ap;
    void *args[] = {&n, &pntr, &indx, &vals, &x, &r, &p, &Ap, &rt, &s, &mail, &err};
    while (!st) {
        if (cudaMemsetAsync(mail, 0, sizeof(CgpWord) * nmail, c->stream) != cudaSuccess ||
            cudaMemsetAsync(rt, 0, sizeof(typename CgpR<X>::T) * n, c->stream) != cudaSuccess) {
            st = cuda_fail(cudaGetLastError(), "persistent cg");
            break;
        }
        const void *fn = exact ? cgp_kernel<V, X, true>(sh.rpt) : cgp_kernel<V, X, false>(sh.rpt);
        cudaLaunchAttribute at[2];
        const cudaLaunchConfig_t cfg = cgp_config(G, sh.cluster, c->stream, at);
        if (cudaLaunchKernelExC(&cfg, fn, args) != cudaSuccess) {
            st = cuda_fail(cudaGetLastError(), "persistent cg launch");
            break;
        }
        *launches += 1;
        if (cudaMemcpyAsync(c->host_result, s, sizeof(SolverScalars), cudaMemcpyDeviceToHost, c->stream) != cudaSuccess ||
            cudaStreamSynchronize(c->stream) != cudaSuccess) {
            st = cuda_fail(cudaGetLastError(), "persistent cg sync");
            break;
        }
        memcpy(&hs, c->host_result, sizeof(SolverScalars));
        if ((st = collect_dev_error(c))) break;
        if (hs.done) break;
    }
    ws_free(c, mail);
    ws_free(c, rt);
    return st;
}

// Runs CG on (A, M) for b -> x (x holds the initial guess).  zero_x0: skip r = b - A x.
// kernels per captured CG iteration: SpMV+dot, update+norm, [L solve, U solve], <r,z>, p update
static int cg_launches_per_iter(bool precond) { return precond ? 6 : 4; }

template <typename V, typename X>
static int cg_run(hgb_ctx *c, hgb_csr *A, hgb_ilu *M, const X *b, X *x, double tol2, double rel, int max_iter,
                  bool zero_x0, int *iters, double *rr_out, long long *launches, bool trans = false) {
    const long n = csr_rows(A);
    CaptureStream cs(c);
    CgWork<X> w;
    int st = w.alloc(c, n, M != nullptr);
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    SolverScalars hs{};
    do {
        if (st) break;
        SolverScalars *s = c->scal;
        cg_init_kernel<<<1, 1, 0, c->stream>>>(s, tol2, rel, max_iter);
        *launches += 1 + (zero_x0 ? 0 : 1) + (M ? 2 : 0) + 2;   // init, SpMV, L/U solves, copy, <r,z>
        // r = b - A x  (r = b; r += -1 * A x)
        if (cudaMemcpyAsync(w.r, b, sizeof(X) * n, cudaMemcpyDeviceToDevice, c->stream)) { st = cuda_fail(cudaGetLastError(), "cg"); break; }
        if (trans && (st = csr_ensure_transpose(A))) break;
        if (!zero_x0 && (st = spmv_A<V, X>(c, A, X(-1), x, X(1), w.r, nullptr, nullptr, trans))) break;
        X *z = M ? w.z : w.r;
        if (M && (st = ilu_apply_internal(M, trans ? 'T' : 'N', w.r, w.z, nullptr))) break;
        copy_kernel<X><<<ew_grid(c, n), 256, 0, c->stream>>>(n, z, w.p);
        cg_rz_kernel<X, RZ_INIT><<<vec_grid(c, n), kEwThreads, 0, c->stream>>>(n, s, w.r, z, c->partials, c->counter);
        if ((st = launch_check("cg init"))) break;
        if (cgp_eligible<V, X>(A, M, trans)) {   // small, L2-resident, unpreconditioned: one persistent launch
            st = cgp_run<V, X>(c, A, w, x, n, launches, hs);
            break;
        }
        // capture ITERS_PER_GRAPH iterations
        cudaStreamCaptureMode mode = cudaStreamCaptureModeThreadLocal;
        if (cudaStreamBeginCapture(c->stream, mode)) { st = cuda_fail(cudaGetLastError(), "begin capture"); break; }
        for (int k = 0; k < kItersPerGraph && !st; k++) st = cg_iteration<V, X>(c, A, M, w, x, n, trans);
        cudaError_t ce = cudaStreamEndCapture(c->stream, &graph);
        if (st) break;
        if (ce != cudaSuccess) { st = cuda_fail(ce, "end capture"); break; }
        if (cudaGraphInstantiate(&exec, graph, 0)) { st = cuda_fail(cudaGetLastError(), "graph instantiate"); break; }
        for (;;) {
            if (cudaGraphLaunch(exec, c->stream)) { st = cuda_fail(cudaGetLastError(), "graph launch"); break; }
            *launches += (long long)kItersPerGraph * cg_launches_per_iter(M != nullptr);
            if (cudaMemcpyAsync(c->host_result, s, sizeof(SolverScalars), cudaMemcpyDeviceToHost, c->stream)) { st = cuda_fail(cudaGetLastError(), "cg"); break; }
            if (cudaStreamSynchronize(c->stream)) { st = cuda_fail(cudaGetLastError(), "cg sync"); break; }
            memcpy(&hs, c->host_result, sizeof(SolverScalars));
            if (hs.done) break;
        }
    } while (0);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    w.release();
    if (st) return st;
    HGB_TRY(collect_dev_error(c));
    *iters = hs.it;
    *rr_out = hs.rr;
    return HGB_OK;
}

static int true_residual(hgb_ctx *c, hgb_csr *A64, const double *b, const double *x, double *r, double *res,
                         long long *launches, bool trans = false) {
    *launches += 2;
    const long n = csr_rows(A64);
    HGB_CUDA(cudaMemcpyAsync(r, b, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream));
    if (trans) HGB_TRY(csr_ensure_transpose(A64));
    HGB_TRY(spmv_A<double, double>(c, A64, -1.0, x, 1.0, r, nullptr, nullptr, trans));
    residual_norm_kernel<<<reduce_grid(c, n, 256 * 4), 256, 0, c->stream>>>(n, r, c->partials, c->counter, c->result);
    HGB_TRY(launch_check("residual_norm_kernel"));
    HGB_CUDA(cudaMemcpyAsync(c->host_result, c->result, sizeof(double), cudaMemcpyDeviceToHost, c->stream));
    HGB_CUDA(cudaStreamSynchronize(c->stream));
    *res = sqrt(c->host_result[0]);
    return HGB_OK;
}

}  // namespace hgb

using namespace hgb;

extern "C" {

int hgb_cg_solve(hgb_ctx *c, hgb_csr *A, hgb_ilu *M, const void *b, void *x, double tol, int max_iter,
                 hgb_solve_info *info) {
    return hgb_cg_solve_op(c, A, M, 'N', b, x, tol, max_iter, info);
}

int hgb_cg_solve_op(hgb_ctx *c, hgb_csr *A, hgb_ilu *M, char trans, const void *b, void *x, double tol, int max_iter,
                    hgb_solve_info *info) {
    if (!c || !A || !b || !x) return fail(HGB_ERR_ARG, "cg_solve: bad arguments");
    const bool tr = (trans == 'T' || trans == 't' || trans == 'C' || trans == 'c');
    if (!tr && trans != 'N' && trans != 'n') return fail(HGB_ERR_ARG, "cg_solve: trans '%c'", trans);
    if (csr_rows(A) != csr_cols(A)) return fail(HGB_ERR_ARG, "cg_solve: square matrix required");
    if (max_iter < 1) return fail(HGB_ERR_ARG, "cg_solve: max_iter < 1");
    DeviceGuard g(c->device);
    hgb_dtype dt = csr_dtype(A);
    if (M) {
        if (ilu_n(M) != csr_rows(A)) return fail(HGB_ERR_ARG, "cg_solve: preconditioner size");
        if (!ilu_matches(ilu_store(M), dt)) return fail(HGB_ERR_ARG, "cg_solve: preconditioner precision does not match the matrix");
    }
    if (dt == HGB_C128 || dt == HGB_C64) {
        if (tr) return fail(HGB_ERR_UNSUPPORTED, "cg_solve: transposed complex solves");
        return zcg_solve(c, A, M ? ilu_zfactor(M) : nullptr, b, x, tol, max_iter, info);
    }
    int it = 0;
    double rr = 0.0;
    double tol2 = tol * tol;
    long long launches = 0;
    int st;
    if (dt == HGB_F64) st = cg_run<double, double>(c, A, M, (const double *)b, (double *)x, tol2, 0.0, max_iter, false, &it, &rr, &launches, tr);
    else if (dt == HGB_F32) st = cg_run<float, float>(c, A, M, (const float *)b, (float *)x, tol2, 0.0, max_iter, false, &it, &rr, &launches, tr);
    else st = cg_run<uint16_t, float>(c, A, M, (const float *)b, (float *)x, tol2, 0.0, max_iter, false, &it, &rr, &launches, tr);
    if (st) return st;
    if (info) {
        info->iterations = it;
        info->outer = 0;
        info->residual = sqrt(rr);
        info->true_residual = -1.0;
        info->kernel_launches = launches;
    }
    return HGB_OK;
}

int hgb_ir_pcg_solve(hgb_ctx *c, hgb_csr *A64, hgb_csr *Ai, hgb_ilu *Mi, const double *b, double *x, double tol,
                     double inner_rtol, int max_inner, int max_outer, hgb_solve_info *info) {
    return hgb_ir_pcg_solve_op(c, A64, Ai, Mi, 'N', b, x, tol, inner_rtol, max_inner, max_outer, info);
}

int hgb_ir_pcg_solve_op(hgb_ctx *c, hgb_csr *A64, hgb_csr *Ai, hgb_ilu *Mi, char trans, const double *b, double *x,
                        double tol, double inner_rtol, int max_inner, int max_outer, hgb_solve_info *info) {
    if (!c || !A64 || !Ai || !b || !x) return fail(HGB_ERR_ARG, "ir_pcg: bad arguments");
    const bool tr = (trans == 'T' || trans == 't' || trans == 'C' || trans == 'c');
    if (!tr && trans != 'N' && trans != 'n') return fail(HGB_ERR_ARG, "ir_pcg: trans '%c'", trans);
    if (tr && csr_dtype(Ai) == HGB_BF16) return fail(HGB_ERR_UNSUPPORTED, "ir_pcg: transposed solve with a bf16 matrix");
    if (csr_dtype(A64) != HGB_F64) return fail(HGB_ERR_ARG, "ir_pcg: the outer matrix must be F64");
    if (!real_inner(csr_dtype(Ai))) return fail(HGB_ERR_ARG, "ir_pcg: the inner matrix must be F32 or BF16");
    if (Mi && !real_inner(ilu_store(Mi))) return fail(HGB_ERR_ARG, "ir_pcg: the inner preconditioner must store F32 or BF16");
    const long n = csr_rows(A64);
    if (csr_rows(Ai) != n || csr_cols(A64) != n) return fail(HGB_ERR_ARG, "ir_pcg: sizes");
    if (max_inner < 1 || max_outer < 0 || !(inner_rtol > 0.0)) return fail(HGB_ERR_ARG, "ir_pcg: limits");
    DeviceGuard g(c->device);
    double *r64 = nullptr;
    float *r32 = nullptr, *d32 = nullptr;
    int st = HGB_OK;
    int total = 0, outer = 0;
    double res = 0.0;
    long long launches = 0;
    do {
        if (ws_alloc(c, &r64, n) || ws_alloc(c, &r32, n) || ws_alloc(c, &d32, n)) {
            st = cuda_fail(cudaErrorMemoryAllocation, "ir_pcg workspace");
            break;
        }
        for (;;) {
            if ((st = true_residual(c, A64, b, x, r64, &res, &launches, tr))) break;
            if (res < tol || res == 0.0 || outer >= max_outer || !(res == res)) break;   // 0: x is exact
            f64_to_f32_kernel<<<ew_grid(c, n), 256, 0, c->stream>>>(n, r64, r32);
            zero_f32_kernel<<<ew_grid(c, n), 256, 0, c->stream>>>(n, d32);
            int it = 0;
            double rr = 0.0;
            launches += 3;   // residual cast, zero, update
            // reduce this sweep's residual only as far as the target needs (with a factor 2 of
            // margin), never by less than inner_rtol: the last sweep stops early
            const double rel = std::min(0.5, std::max(inner_rtol, 0.5 * tol / res));
            if (csr_dtype(Ai) == HGB_F32)
                st = cg_run<float, float>(c, Ai, Mi, r32, d32, 0.0, rel, max_inner, true, &it, &rr, &launches, tr);
            else
                st = cg_run<uint16_t, float>(c, Ai, Mi, r32, d32, 0.0, rel, max_inner, true, &it, &rr, &launches);
            if (st) break;
            total += it;
            add_f32_to_f64_kernel<<<ew_grid(c, n), 256, 0, c->stream>>>(n, d32, x);
            if ((st = launch_check("ir update"))) break;
            outer++;
        }
    } while (0);
    ws_free(c, r64);
    ws_free(c, r32);
    ws_free(c, d32);
    if (st) return st;
    if (info) {
        info->iterations = total;
        info->outer = outer;
        info->residual = res;
        info->true_residual = res;
        info->kernel_launches = launches;
    }
    if (!(res < tol || res == 0.0)) return fail(HGB_ERR_NOT_CONVERGED, "ir_pcg: ||b-Ax|| = %g after %d sweeps (tol %g)", res, outer, tol);
    return HGB_OK;
}

}  // extern "C"

// ============================================== mixed PCG with reliable updates =======
// One FP32 ILU(0)-PCG (solve_cg_core's order, hex/solvers/hala_solvers_cg.hpp:92-156) on the
// correction d, with FP64 reliable updates (van der Vorst and Ye, "Residual replacement
// strategies for Krylov subspace iterative methods for the convergence of true residuals",
// SIAM J. Sci. Comput. 22 (2000)): when ||r|| falls below delta times its largest value since
// the last update (or below tol, or at the iteration limit), x += d in FP64, r = b - A x in FP64
// and the iteration continues from the new residual with the same search direction, or restarts
// (beta = 0) when that update reduced the FP64 residual less than twice.  Unlike a
// restarted refinement, the Krylov space is kept, so the iterations stay those of FP64 PCG.
// No reference counterpart.  One iteration is nine launches, three of them (the update) no-ops
// except in update iterations; kItersPerGraph iterations are one CUDA graph.
namespace hgb {

__global__ void ru_init_kernel(SolverScalars *s, double tol2, double delta2, double rr, int max_iter) {
    s->it = 0;
    s->done = 0;
    s->max_iter = max_iter;
    s->tol2 = tol2;
    s->rel = 0.0;
    s->zr = s->nzr = s->pap = 0.0;
    s->rr = rr;
    s->rmax2 = rr;
    s->delta2 = delta2;
    s->ru_skip = 1;
    s->updates = 0;
    s->last2 = rr;
    s->restart = 0;
}

// a = <r,z>/<p,Ap>; d += a p; r -= a Ap; ||r||^2; decide whether this iteration updates
__global__ void __launch_bounds__(kEwThreads, kEwCtas) ru_step_kernel(long n, SolverScalars *s, const float *__restrict__ p, const float *__restrict__ Ap,
                               float *__restrict__ d, float *__restrict__ r, double *partials, unsigned *counter,
                               const double *pap_part, int pap_n) {
    if (s->done) return;
    constexpr int U = ew_unroll<float, 4>();
    const long T = (long)gridDim.x * blockDim.x;
    long base = blockIdx.x * (long)blockDim.x + threadIdx.x;
    float pv[U], av[U], dv[U], rv[U];
    auto load = [&] {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = base + u * T;
            if (i < n) {
                pv[u] = p[i];
                av[u] = Ap[i];
                dv[u] = d[i];
                rv[u] = r[i];
            }
        }
    };
    load();   // in flight while the scalar is summed
    // a = <r,z> / <p,Ap>; d += a p; r -= a Ap
    double pap = 0.0;   // thread 0's
    const float a = (float)vec_scalar(pap_part, pap_n, s->pap, [&](double v) { pap = v; return s->nzr / v; });
    const float ma = -a;
    DotAcc<float> rr;
    while (base < n) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = base + u * T;
            if (i < n) {
                d[i] = vec_axpy(dv[u], a, pv[u]);
                const float ri = vec_axpy(rv[u], ma, av[u]);
                r[i] = ri;
                rr.add(ri, ri);
            }
        }
        base += T * U;
        load();
    }
    double acc[1] = {rr.get()};
    vec_grid_sum<1>(acc, partials, counter, [&](double (&v)[1]) {
        const double rr = v[0];
        s->pap = pap;
        s->zr = s->nzr;
        s->rr = rr;
        s->it += 1;
        s->rmax2 = fmax(s->rmax2, rr);
        const bool upd = (rr < s->delta2 * s->rmax2) || (rr < s->tol2) || !(rr == rr) || (s->it >= s->max_iter);
        s->ru_skip = upd ? 0 : 1;
        s->restart = 0;
    });
}

// x += d (FP64); d = 0; r64 = b   (the FP64 product follows)
__global__ void ru_fold_kernel(long n, const SolverScalars *__restrict__ s, const double *__restrict__ b,
                               float *__restrict__ d, double *__restrict__ x, double *__restrict__ r64) {
    if (s->ru_skip) return;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        x[i] += (double)d[i];
        d[i] = 0.0f;
        r64[i] = b[i];
    }
}

// r = (float) r64; ||r64||^2; the stopping test on the FP64 residual
__global__ void ru_replace_kernel(long n, SolverScalars *s, const double *__restrict__ r64, float *__restrict__ r,
                                  double *partials, unsigned *counter) {
    if (s->ru_skip) return;
    double acc[1] = {0.0};
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const double v = r64[i];
        r[i] = (float)v;
        acc[0] = fma(v, v, acc[0]);
    }
    grid_sum<1>(acc, partials, counter, [&](double (&v)[1]) {
        const double rr = v[0];
        s->rr = rr;
        s->rmax2 = rr;
        s->updates += 1;
        s->done = (rr < s->tol2) || !(rr == rr) || (s->it >= s->max_iter);
        s->ru_skip = 1;
        // an update that reduced ||r|| less than twice: the kept directions are stale (FP32
        // recurrences on an ill-conditioned operator), restart from the new residual
        s->restart = rr > 0.25 * s->last2;
        s->last2 = rr;
    });
}

// p = beta p + z with beta = <r,z> / <r,z>_old, or p = z after a restart
__global__ void __launch_bounds__(kEwThreads, kEwCtas) ru_p_kernel(long n, SolverScalars *s, float *__restrict__ p,
                            const float *__restrict__ z, const double *rz_part) {
    if (s->done) return;
    constexpr int U = ew_unroll<float, 3>();
    const long T = (long)gridDim.x * blockDim.x;
    long base = blockIdx.x * (long)blockDim.x + threadIdx.x;
    float pv[U], zv[U];
    auto load = [&] {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = base + u * T;
            if (i < n) {
                pv[u] = p[i];
                zv[u] = z[i];
            }
        }
    };
    load();   // in flight while the scalar is summed
    const float ratio = (float)vec_scalar(rz_part, gridDim.x, 0.0, [&](double nzr) {
        if (blockIdx.x == 0) s->nzr = nzr;   // the others read zr only
        return nzr / s->zr;
    });
    const float bta = s->restart ? 0.0f : ratio;
    while (base < n) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const long i = base + u * T;
            if (i < n) p[i] = vec_axpy(zv[u], bta, pv[u]);
        }
        base += T * U;
        load();
    }
}

template <typename V>
static int ru_iteration(hgb_ctx *c, hgb_csr *A64, hgb_csr *Ai, hgb_ilu *M, CgWork<float> &w, float *d, double *x,
                        double *r64, const double *b, long n, bool trans) {
    SolverScalars *s = c->scal;
    const int *done = &s->done;
    int np = 0;
    HGB_TRY(spmv_A<V, float>(c, Ai, 1.0f, w.p, 0.0f, w.Ap, &s->pap, done, trans, &np));
    ru_step_kernel<<<vec_grid(c, n), kEwThreads, 0, c->stream>>>(n, s, w.p, w.Ap, d, w.r, c->partials, c->counter,
                                                                      c->partials + kSpmvPartsOffset, np);
    ru_fold_kernel<<<ew_grid(c, n), 256, 0, c->stream>>>(n, s, b, d, x, r64);
    HGB_TRY(spmv_A<double, double>(c, A64, -1.0, x, 1.0, r64, nullptr, &s->ru_skip, trans));
    ru_replace_kernel<<<reduce_grid(c, n, 256 * 4), 256, 0, c->stream>>>(n, s, r64, w.r, c->partials, c->counter);
    float *z = M ? w.z : w.r;
    if (M) HGB_TRY(ilu_apply_internal(M, trans ? 'T' : 'N', w.r, w.z, done));
    cg_rz_kernel<float, RZ_PARTS><<<vec_grid(c, n), kEwThreads, 0, c->stream>>>(n, s, w.r, z, c->partials, c->counter);
    ru_p_kernel<<<vec_grid(c, n), kEwThreads, 0, c->stream>>>(n, s, w.p, z, c->partials);
    return launch_check("ru iteration");
}

static int ru_launches_per_iter(bool precond) { return precond ? 9 : 7; }

template <typename V>
static int ru_run(hgb_ctx *c, hgb_csr *A64, hgb_csr *Ai, hgb_ilu *M, const double *b, double *x, double tol,
                  double delta, int max_iter, int *iters, int *updates, double *res, long long *launches,
                  bool trans = false) {
    const long n = csr_rows(A64);
    CaptureStream cs(c);
    CgWork<float> w;
    float *d = nullptr;
    double *r64 = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    SolverScalars hs{};
    int st = w.alloc(c, n, M != nullptr);
    do {
        if (st) break;
        if (ws_alloc(c, &d, n) || ws_alloc(c, &r64, n)) {
            st = cuda_fail(cudaErrorMemoryAllocation, "ru_pcg workspace");
            break;
        }
        double rn = 0.0;
        if (trans && (st = csr_ensure_transpose(Ai))) break;
        if ((st = true_residual(c, A64, b, x, r64, &rn, launches, trans))) break;
        *iters = 0;
        *updates = 0;
        *res = rn;
        if (rn < tol || rn == 0.0 || !(rn == rn) || max_iter < 1) break;   // 0: x is exact
        SolverScalars *s = c->scal;
        ru_init_kernel<<<1, 1, 0, c->stream>>>(s, tol * tol, delta * delta, rn * rn, max_iter);
        f64_to_f32_kernel<<<ew_grid(c, n), 256, 0, c->stream>>>(n, r64, w.r);
        zero_f32_kernel<<<ew_grid(c, n), 256, 0, c->stream>>>(n, d);
        float *z = M ? w.z : w.r;
        if (M && (st = ilu_apply_internal(M, trans ? 'T' : 'N', w.r, w.z, nullptr))) break;
        copy_kernel<float><<<ew_grid(c, n), 256, 0, c->stream>>>(n, z, w.p);
        // <r,z> of the first direction (the rr slot keeps the FP64 residual)
        cg_rz_kernel<float, RZ_FIRST><<<vec_grid(c, n), kEwThreads, 0, c->stream>>>(n, s, w.r, z, c->partials, c->counter);
        *launches += 5 + (M ? 2 : 0);
        if ((st = launch_check("ru init"))) break;
        if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal)) { st = cuda_fail(cudaGetLastError(), "begin capture"); break; }
        for (int k = 0; k < kItersPerGraph && !st; k++) st = ru_iteration<V>(c, A64, Ai, M, w, d, x, r64, b, n, trans);
        cudaError_t ce = cudaStreamEndCapture(c->stream, &graph);
        if (st) break;
        if (ce != cudaSuccess) { st = cuda_fail(ce, "end capture"); break; }
        if (cudaGraphInstantiate(&exec, graph, 0)) { st = cuda_fail(cudaGetLastError(), "graph instantiate"); break; }
        for (;;) {
            if (cudaGraphLaunch(exec, c->stream)) { st = cuda_fail(cudaGetLastError(), "graph launch"); break; }
            *launches += (long long)kItersPerGraph * ru_launches_per_iter(M != nullptr);
            if (cudaMemcpyAsync(c->host_result, s, sizeof(SolverScalars), cudaMemcpyDeviceToHost, c->stream) ||
                cudaStreamSynchronize(c->stream)) { st = cuda_fail(cudaGetLastError(), "ru_pcg sync"); break; }
            memcpy(&hs, c->host_result, sizeof(SolverScalars));
            if (hs.done) break;
        }
        *iters = hs.it;
        *updates = hs.updates;
        *res = sqrt(hs.rr);
    } while (0);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    w.release();
    ws_free(c, d);
    ws_free(c, r64);
    if (st) return st;
    return collect_dev_error(c);
}

}  // namespace hgb

extern "C" int hgb_ru_pcg_solve(hgb_ctx *c, hgb_csr *A64, hgb_csr *Ai, hgb_ilu *Mi, const double *b, double *x,
                                double tol, double delta, int max_iter, hgb_solve_info *info) {
    return hgb_ru_pcg_solve_op(c, A64, Ai, Mi, 'N', b, x, tol, delta, max_iter, info);
}

extern "C" int hgb_ru_pcg_solve_op(hgb_ctx *c, hgb_csr *A64, hgb_csr *Ai, hgb_ilu *Mi, char trans, const double *b,
                                   double *x, double tol, double delta, int max_iter, hgb_solve_info *info) {
    if (!c || !A64 || !Ai || !b || !x) return fail(HGB_ERR_ARG, "ru_pcg: bad arguments");
    const bool tr = (trans == 'T' || trans == 't' || trans == 'C' || trans == 'c');
    if (!tr && trans != 'N' && trans != 'n') return fail(HGB_ERR_ARG, "ru_pcg: trans '%c'", trans);
    if (tr && csr_dtype(Ai) == HGB_BF16) return fail(HGB_ERR_UNSUPPORTED, "ru_pcg: transposed solve with a bf16 matrix");
    if (csr_dtype(A64) != HGB_F64) return fail(HGB_ERR_ARG, "ru_pcg: the outer matrix must be F64");
    if (!real_inner(csr_dtype(Ai))) return fail(HGB_ERR_ARG, "ru_pcg: the inner matrix must be F32 or BF16");
    if (Mi && !real_inner(ilu_store(Mi))) return fail(HGB_ERR_ARG, "ru_pcg: the preconditioner must store F32 or BF16");
    const long n = csr_rows(A64);
    if (csr_rows(Ai) != n || csr_cols(A64) != n || csr_cols(Ai) != n || (Mi && ilu_n(Mi) != n))
        return fail(HGB_ERR_ARG, "ru_pcg: sizes");
    if (max_iter < 0 || !(delta > 0.0 && delta < 1.0)) return fail(HGB_ERR_ARG, "ru_pcg: limits (0 < delta < 1)");
    DeviceGuard g(c->device);
    int it = 0, upd = 0;
    double res = 0.0;
    long long launches = 0;
    int st = (csr_dtype(Ai) == HGB_F32)
                 ? ru_run<float>(c, A64, Ai, Mi, b, x, tol, delta, max_iter, &it, &upd, &res, &launches, tr)
                 : ru_run<uint16_t>(c, A64, Ai, Mi, b, x, tol, delta, max_iter, &it, &upd, &res, &launches);
    if (st) return st;
    if (info) {
        info->iterations = it;
        info->outer = upd;
        info->residual = res;
        info->true_residual = res;
        info->kernel_launches = launches;
    }
    if (!(res < tol || res == 0.0)) return fail(HGB_ERR_NOT_CONVERGED, "ru_pcg: ||b-Ax|| = %g after %d iterations (tol %g)", res, it, tol);
    return HGB_OK;
}

// ===================================================================== GMRES ===========
// solve_gmres (hex/solvers/hala_solvers_gmres.hpp:127-230), device resident.  The reference
// reads the projection coefficients back to the host in every inner iteration (:67-72) and
// rotates on the host; here the Hessenberg columns, the Givens rotations, the residual estimate
// and the back substitution (tpsv) live in a GmresState in device memory and are updated by the
// last CTA of the projection's grid reduction.  Inner iteration j of a cycle always projects
// against j+1 basis vectors, so one whole restart cycle is captured once into a CUDA graph; the
// launches of iterations after the inner stop are no-ops, and the host reads the state once per
// cycle.  The arithmetic of the rotations and of tpsv is the reference's operation for operation
// (explicitly rounded, no contraction); the inner products are parallel, and the updates of r and x take the
// columns in the reference's order with fused multiply-adds.
namespace hgb {

constexpr int kGmresMaxRestart = 512;   // the Hessenberg factor (1 MB) lives in device memory

struct GmresState {
    // header (read by the host after every cycle)
    double tol;          // threshold on the preconditioned residual estimate
    double rel;          // > 0: tol = max(tol, rel * first estimate) (inner solves of a refinement)
    double inner_res, outer_res;
    double inv;          // reciprocal of the norm of the vector being appended
    int k, stop, done, wcol, upd, total, outer, max_outer, restart, first;
    // rotations and the triangular factor
    double Z[kGmresMaxRestart + 1];
    double C[kGmresMaxRestart], S[kGmresMaxRestart];
    double H[kGmresMaxRestart * (kGmresMaxRestart + 1) / 2];
};

__device__ __forceinline__ void gm_rotg(double &a, double &b, double &c, double &s) {
    double roe = (fabs(a) > fabs(b)) ? a : b;
    double scale = __dadd_rn(fabs(a), fabs(b)), r, z;
    if (scale == 0.0) {
        c = 1.0; s = 0.0; r = 0.0; z = 0.0;
    } else {
        double as = __ddiv_rn(a, scale), bs = __ddiv_rn(b, scale);
        r = __dmul_rn(scale, __dsqrt_rn(__dadd_rn(__dmul_rn(as, as), __dmul_rn(bs, bs))));
        if (roe < 0.0) r = -r;
        c = __ddiv_rn(a, r);
        s = __ddiv_rn(b, r);
        z = 1.0;
        if (fabs(a) > fabs(b)) z = s;
        if (fabs(b) >= fabs(a) && c != 0.0) z = __ddiv_rn(1.0, c);
    }
    a = r;
    b = z;
}

__device__ __forceinline__ void gm_rot(double &x, double &y, double c, double s) {
    double t = __dadd_rn(__dmul_rn(c, x), __dmul_rn(s, y));
    y = __dsub_rn(__dmul_rn(c, y), __dmul_rn(s, x));
    x = t;
}

__global__ void gm_init_kernel(GmresState *st, double tol, double rel, int max_outer, int restart) {
    st->tol = tol;
    st->rel = rel;
    st->inner_res = 0.0;
    st->outer_res = tol + 1.0;
    st->inv = 0.0;
    st->k = 0;
    st->stop = 1;
    st->done = !(max_outer > 0);
    st->wcol = -1;
    st->upd = 0;
    st->total = 0;
    st->outer = 0;
    st->max_outer = max_outer;
    st->restart = restart;
    st->first = 1;
}

__global__ void gm_begin_kernel(GmresState *st) {
    st->k = 0;
    st->upd = 0;
    st->wcol = -1;
    st->stop = 1;
}

template <typename X>
__global__ void gm_copy_kernel(long n, const int *skip, const X *__restrict__ a, X *__restrict__ b) {
    if (*skip) return;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) b[i] = a[i];
}

// beta = ||P^-1 (b - A x)||: the first estimate of the cycle (Z[0]); basis vector 0 follows
template <typename X>
__global__ void gm_start_kernel(long n, GmresState *st, const X *__restrict__ r, double *partials,
                                unsigned *counter) {
    if (st->done) return;
    double acc[1] = {0.0};
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        acc[0] = fma((double)r[i], (double)r[i], acc[0]);
    grid_sum<1>(acc, partials, counter, [&](double (&v)[1]) {
        double beta = __dsqrt_rn(v[0]);
        if (st->first) {
            st->first = 0;
            if (st->rel > 0.0) st->tol = fmax(st->tol, st->rel * beta);
        }
        st->total += 1;
        st->inner_res = beta;
        st->Z[0] = beta;
        bool go = beta > st->tol;
        st->stop = !go;
        st->wcol = go ? 0 : -1;
        st->inv = __ddiv_rn(1.0, beta);
    });
}

// r *= inv; W[:, wcol] = r   (scal(1/nrm, r) and the copy into the basis)
template <typename X>
__global__ void gm_scale_kernel(long n, const GmresState *__restrict__ st, X *__restrict__ r, X *__restrict__ W) {
    const int col = st->wcol;
    if (col < 0) return;
    const X a = (X)st->inv;
    X *w = W + (long)col * n;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        X v = mul_rn(r[i], a);
        r[i] = v;
        w[i] = v;
    }
}

// The basis kernels below read k columns of n and do one FP64 operation per entry (two a warp-wide instruction, 62
// cycles of an SM quarter's unit each, were it rounded separately): at 96^3 a column costs 1.4 us of the unit
// and 1.0 us of HBM.  So they take fused multiply-adds, keep instructions for absent columns as branches
// (HGB_UNIFORM_IF), and sum 32 lanes' 32 columns with 31 additions a lane instead of 160.

// Sums v[j] over the warp for KMAX columns j: column lane % KMAX's sum in v[0].  Each step adds two lanes' halves of the
// columns and leaves each lane one of them.
template <int KMAX>
__device__ __forceinline__ void gm_warp_columns(double (&v)[KMAX]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o >= KMAX; o >>= 1)
#pragma unroll
        for (int j = 0; j < KMAX; j++) v[j] += __shfl_xor_sync(0xffffffffu, v[j], o);
#pragma unroll
    for (int o = KMAX < 32 ? KMAX / 2 : 16; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < o; j++) {
            const double keep = lane & o ? v[j + o] : v[j], send = lane & o ? v[j] : v[j + o];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
}

// cf[0..k] = W[:, 0..k]^T r   (krylov_project's gemv 'T', :67-70), for the k1 columns from W and cf
// on (one group of up to 32 columns per launch).  All columns' loads of a row are in flight together; 96^3 FP64,
// 30 columns: 180 -> 62 us.
template <typename X, int KMAX>
__global__ void __launch_bounds__(256, 32 / KMAX)
gm_dots_kernel(long n, int k1, const GmresState *__restrict__ st, const X *__restrict__ W,
               const X *__restrict__ r, double *cf, double *partials, unsigned *counter) {
    if (st->stop) return;
    __shared__ double sh[8 * KMAX];
    __shared__ bool last;
    double acc[KMAX];
#pragma unroll
    for (int j = 0; j < KMAX; j++) acc[j] = 0.0;
    const int tid = threadIdx.x;
    const long stride = (long)gridDim.x * 256;
    X wn[KMAX], rn = X(0);   // the next row's
    auto load = [&](long i) {
        rn = i < n ? r[i] : X(0);
#pragma unroll
        for (int j = 0; j < KMAX; j++) wn[j] = j < k1 && i < n ? W[(long)j * n + i] : X(0);
    };
    long ib = (long)blockIdx.x * 256 + (tid & ~31);
    load(ib + (tid & 31));
    for (; ib < n; ib += stride) {
        const double ri = (double)rn;
        X w[KMAX];
#pragma unroll
        for (int j = 0; j < KMAX; j++) w[j] = wn[j];
        load(ib + stride + (tid & 31));
#pragma unroll
        for (int j = 0; j < KMAX; j += 2)
            HGB_UNIFORM_IF(j < k1) {
                acc[j] = fma((double)w[j], ri, acc[j]);
                acc[j + 1] = fma((double)w[j + 1], ri, acc[j + 1]);
            }
    }
    gm_warp_columns<KMAX>(acc);
    if ((tid & 31) < KMAX) sh[(tid >> 5) * KMAX + (tid & 31)] = acc[0];
    __syncthreads();
    auto column = [&] {
        double t = sh[tid];
#pragma unroll
        for (int w = 1; w < 8; w++) t += sh[w * KMAX + tid];
        return t;
    };
    if (tid < 32) {
        if (tid < KMAX) {
            partials[blockIdx.x * KMAX + tid] = column();
            __threadfence();
        }
        __syncwarp();
        if (tid == 0) last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0.0;   // the last CTA: column tid % KMAX, every (256 / KMAX)-th CTA's part
    for (int b = tid / KMAX; b < (int)gridDim.x; b += 256 / KMAX) t += __ldcg(partials + b * KMAX + tid % KMAX);
#pragma unroll
    for (int o = KMAX; o < 32; o *= 2) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((tid & 31) < KMAX) sh[(tid >> 5) * KMAX + (tid & 31)] = t;
    __syncthreads();
    if (tid < k1) cf[tid] = column();
    if (tid == 0) *counter = 0u;
}

// v + sum over j < k of c[j] W[j * n + i], column by column; eight columns' loads in flight
template <typename X>
__device__ __forceinline__ X gm_combine(X v, long n, long i, int k, const X *__restrict__ W, const X *c) {
    for (int j0 = 0; j0 < k; j0 += 8) {
        X w[8];
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (j0 + q < k) w[q] = W[(long)(j0 + q) * n + i];
#pragma unroll
        for (int q = 0; q < 8; q++) HGB_UNIFORM_IF(j0 + q < k) v = fma(c[j0 + q], w[q], v);
    }
    return v;
}

// r -= W cf (krylov_project's gemv 'N', :71-76), ||r||, then in the last CTA the Givens step of
// solve_gmres (:190-216) for column k of the Hessenberg matrix.  96^3 FP64, 30 columns: 123 -> 66 us.
template <typename X>
__global__ void __launch_bounds__(256, 4)
gm_update_kernel(long n, int k, GmresState *st, const X *__restrict__ W, const double *__restrict__ cf,
                 X *__restrict__ r, double *partials, unsigned *counter) {
    if (st->stop) return;
    __shared__ X c[kGmresMaxRestart];
    __shared__ double cs[2][kGmresMaxRestart];   // the previous rotations, for the last CTA's chain
    for (int j = threadIdx.x; j <= k; j += 256) {
        c[j] = (X)-cf[j];
        cs[0][j] = st->C[j];
        cs[1][j] = st->S[j];
    }
    __syncthreads();
    double acc[1] = {0.0};
    for (long i = blockIdx.x * 256L + threadIdx.x; i < n; i += gridDim.x * 256L) {
        const X ri = gm_combine(r[i], n, i, k + 1, W, c);
        r[i] = ri;
        acc[0] = fma((double)ri, (double)ri, acc[0]);
    }
    grid_sum<1>(acc, partials, counter, [&](double (&v)[1]) {
        const double nrm = __dsqrt_rn(v[0]);
        // the previous rotations applied to the new column in order, carrying h[i + 1] in a register
        double *Hk = st->H + (long)k * (k + 1) / 2;
        double hi = cf[0];
        for (int i = 0; i < k; i++) {
            double hn = cf[i + 1];
            gm_rot(hi, hn, cs[0][i], cs[1][i]);
            Hk[i] = hi;
            hi = hn;
        }
        double beta = nrm, ic, is;
        gm_rotg(hi, beta, ic, is);
        Hk[k] = hi;
        st->S[k] = is;
        st->C[k] = ic;
        const double res = fabs(__dmul_rn(is, st->Z[k]));
        st->inner_res = res;
        st->total += 1;
        st->k = k + 1;
        const bool expand = (res > st->tol) && (k + 1 < st->restart);
        if (expand) {
            st->Z[k + 1] = 0.0;
            gm_rot(st->Z[k], st->Z[k + 1], ic, is);
            st->wcol = k + 1;
            st->inv = __ddiv_rn(1.0, nrm);
        } else {
            st->wcol = -1;
            st->stop = 1;
        }
    });
}

// End of a cycle: tpsv('U','N','N', k, H, Z) (:219-223), the restart bookkeeping (:225-229).  One warp: a column's
// subtractions in parallel (restart 30: 77 -> 32 us)
__global__ void gm_end_kernel(GmresState *st) {
    if (st->done) return;
    const int nz = st->k, lane = threadIdx.x;
    for (int j = nz - 1; j >= 0; j--) {
        const double *Hj = st->H + (long)j * (j + 1) / 2;
        if (st->Z[j] != 0.0) {
            const double tt = __ddiv_rn(st->Z[j], Hj[j]);
            __syncwarp();   // every lane has read Z[j]
            for (int i = lane; i < j; i += 32) st->Z[i] = __dsub_rn(st->Z[i], __dmul_rn(tt, Hj[i]));
            if (lane == 0) st->Z[j] = tt;
        }
        __syncwarp();
    }
    if (lane == 0) {
        if (nz > 0) st->upd = 1;
        st->outer += 1;
        st->outer_res = st->inner_res;
        st->done = !(st->outer_res > st->tol && st->outer < st->max_outer);
    }
}

// x += W[:, 0..k-1] Z   (krylov_combine, :53-60), column by column, a fused multiply-add each
template <typename X>
__global__ void __launch_bounds__(256, 4)
gm_xupdate_kernel(long n, const GmresState *__restrict__ st, const X *__restrict__ W, X *__restrict__ x) {
    if (!st->upd) return;
    __shared__ X c[kGmresMaxRestart];
    const int nz = st->k;
    for (int j = threadIdx.x; j < nz; j += 256) c[j] = (X)st->Z[j];
    __syncthreads();
    for (long i = blockIdx.x * 256L + threadIdx.x; i < n; i += gridDim.x * 256L) x[i] = gm_combine(x[i], n, i, nz, W, c);
}

template <typename X>
static int gm_dots_launch(hgb_ctx *c, long n, int k1, const GmresState *st, const X *W, const X *r, double *cf) {
    for (int j0 = 0; j0 < k1; j0 += 32) {   // groups of up to 32 columns, one grid reduction each
        const int kk = std::min(32, k1 - j0);
        const X *Wj = W + (long)j0 * n;
        double *cj = cf + j0;
        // resident CTAs (KMAX loads and sums a thread: 32 / KMAX CTAs per SM); at most 32 parts per CTA
        auto grid = [&](int kmax) { return (int)std::max<long>(1, std::min<long>((n + 255) / 256, (long)c->num_sms * (32 / kmax))); };
        if (kk <= 8) gm_dots_kernel<X, 8><<<grid(8), 256, 0, c->stream>>>(n, kk, st, Wj, r, cj, c->partials, c->counter);
        else if (kk <= 16) gm_dots_kernel<X, 16><<<grid(16), 256, 0, c->stream>>>(n, kk, st, Wj, r, cj, c->partials, c->counter);
        else gm_dots_kernel<X, 32><<<grid(32), 256, 0, c->stream>>>(n, kk, st, Wj, r, cj, c->partials, c->counter);
        HGB_TRY(launch_check("gm_dots_kernel"));
    }
    return HGB_OK;
}

// Runs restarted GMRES on (A, M) for b -> x (x holds the initial guess).  tol: absolute threshold
// on the preconditioned residual estimate; rel > 0 also stops at rel * the first estimate;
// max_outer: restart cycles.
template <typename V, typename X>
static int gmres_run(hgb_ctx *c, hgb_csr *A, hgb_ilu *M, int restart, const X *b, X *x, double tol, double rel,
                     int max_outer, int *total, int *outer, double *res, long long *launches) {
    const long n = csr_rows(A);
    CaptureStream cs(c);
    X *t = nullptr, *r = nullptr, *W = nullptr;
    double *cf = nullptr;
    GmresState *st = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    const int pre = M ? 2 : 1;          // ILU: L and U sweeps; none: a copy
    long long per_cycle = 6 + pre + (long long)restart * (3 + pre);
    for (int k = 0; k < restart; k++) per_cycle += k / 32 + 1;   // gm_dots_launch's groups
    int rc = HGB_OK;
    do {
        if (ws_alloc(c, &t, n) || ws_alloc(c, &r, n) || ws_alloc(c, &W, (size_t)n * restart) ||
            ws_alloc(c, &cf, kGmresMaxRestart + 1) || ws_alloc(c, &st, 1)) {
            rc = cuda_fail(cudaErrorMemoryAllocation, "gmres workspace");
            break;
        }
        gm_init_kernel<<<1, 1, 0, c->stream>>>(st, tol, rel, max_outer, restart);
        *launches += 1;
        if ((rc = launch_check("gm_init_kernel"))) break;
        auto precon = [&](const X *in, X *out, const int *skip) -> int {
            if (M) return ilu_apply_internal(M, 'N', in, out, skip);
            gm_copy_kernel<X><<<ew_grid(c, n), 256, 0, c->stream>>>(n, skip, in, out);
            return launch_check("gm_copy_kernel");
        };
        if (cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal)) { rc = cuda_fail(cudaGetLastError(), "begin capture"); break; }
        do {
            // t = b - A x ; r = P^-1 t ; beta = ||r|| ; W[:,0] = r / beta
            gm_begin_kernel<<<1, 1, 0, c->stream>>>(st);
            gm_copy_kernel<X><<<ew_grid(c, n), 256, 0, c->stream>>>(n, &st->done, b, t);
            if ((rc = spmv_A<V, X>(c, A, X(-1), x, X(1), t, nullptr, &st->done))) break;
            if ((rc = precon(t, r, &st->done))) break;
            gm_start_kernel<X><<<reduce_grid(c, n, 256 * 4), 256, 0, c->stream>>>(n, st, r, c->partials, c->counter);
            gm_scale_kernel<X><<<ew_grid(c, n), 256, 0, c->stream>>>(n, st, r, W);
            for (int k = 0; k < restart && !rc; k++) {
                if ((rc = spmv_A<V, X>(c, A, X(1), r, X(0), t, nullptr, &st->stop))) break;
                if ((rc = precon(t, r, &st->stop))) break;
                if ((rc = gm_dots_launch<X>(c, n, k + 1, st, W, r, cf))) break;
                gm_update_kernel<X><<<reduce_grid(c, n, 256 * 4), 256, 0, c->stream>>>(n, k, st, W, cf, r, c->partials,
                                                                                       c->counter);
                gm_scale_kernel<X><<<ew_grid(c, n), 256, 0, c->stream>>>(n, st, r, W);
            }
            if (rc) break;
            gm_end_kernel<<<1, 32, 0, c->stream>>>(st);
            gm_xupdate_kernel<X><<<ew_grid(c, n), 256, 0, c->stream>>>(n, st, W, x);
            rc = launch_check("gmres cycle");
        } while (0);
        cudaError_t ce = cudaStreamEndCapture(c->stream, &graph);
        if (rc) break;
        if (ce != cudaSuccess) { rc = cuda_fail(ce, "end capture"); break; }
        if (cudaGraphInstantiate(&exec, graph, 0)) { rc = cuda_fail(cudaGetLastError(), "graph instantiate"); break; }
        GmresState hs{};
        const size_t head = offsetof(GmresState, Z);
        for (;;) {
            if (cudaGraphLaunch(exec, c->stream)) { rc = cuda_fail(cudaGetLastError(), "graph launch"); break; }
            *launches += per_cycle;
            if (cudaMemcpyAsync(c->host_result, st, head, cudaMemcpyDeviceToHost, c->stream) ||
                cudaStreamSynchronize(c->stream)) { rc = cuda_fail(cudaGetLastError(), "gmres"); break; }
            memcpy(&hs, c->host_result, head);
            if (hs.done) break;
        }
        *total = hs.total;
        *outer = hs.outer;
        *res = hs.inner_res;
    } while (0);
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    ws_free(c, t);
    ws_free(c, r);
    ws_free(c, W);
    ws_free(c, cf);
    ws_free(c, st);
    if (rc) return rc;
    return collect_dev_error(c);
}

}  // namespace hgb

extern "C" int hgb_gmres_solve(hgb_ctx *c, hgb_csr *A, hgb_ilu *M, int restart, const void *bv, void *xv, double tol,
                               int max_iter, hgb_solve_info *info) {
    if (!c || !A || !bv || !xv || restart < 1 || restart > kGmresMaxRestart)
        return fail(HGB_ERR_ARG, "gmres: bad arguments (restart 1..%d)", kGmresMaxRestart);
    if (csr_rows(A) != csr_cols(A)) return fail(HGB_ERR_ARG, "gmres: square matrix required");
    const hgb_dtype dt = csr_dtype(A);
    if (M) {
        if (ilu_n(M) != csr_rows(A)) return fail(HGB_ERR_ARG, "gmres: preconditioner size");
        if (!ilu_matches(ilu_store(M), dt)) return fail(HGB_ERR_ARG, "gmres: preconditioner precision does not match the matrix");
    }
    DeviceGuard g(c->device);
    if (dt == HGB_C128 || dt == HGB_C64)
        return zgmres_solve(c, A, M ? ilu_zfactor(M) : nullptr, restart, bv, xv, tol, max_iter, info);
    int total = 0, outer = 0;
    double res = 0.0;
    long long launches = 0;
    int st;
    if (dt == HGB_F64)
        st = gmres_run<double, double>(c, A, M, restart, (const double *)bv, (double *)xv, tol, 0.0, max_iter, &total, &outer, &res, &launches);
    else if (dt == HGB_F32)
        st = gmres_run<float, float>(c, A, M, restart, (const float *)bv, (float *)xv, tol, 0.0, max_iter, &total, &outer, &res, &launches);
    else
        st = gmres_run<uint16_t, float>(c, A, M, restart, (const float *)bv, (float *)xv, tol, 0.0, max_iter, &total, &outer, &res, &launches);
    if (st) return st;
    if (info) {
        info->iterations = total;
        info->outer = outer;
        info->residual = res;
        info->true_residual = -1.0;
        info->kernel_launches = launches;
    }
    return HGB_OK;
}

// Mixed-precision GMRES: FP64 iterative refinement around an FP32-vector GMRES(restart) with an
// FP32 or BF16 matrix and ILU(0) (no reference counterpart; the inner solver is solve_gmres).
extern "C" int hgb_ir_gmres_solve(hgb_ctx *c, hgb_csr *A64, hgb_csr *Ai, hgb_ilu *Mi, int restart, const double *b,
                                  double *x, double tol, double inner_rtol, int max_inner, int max_outer,
                                  hgb_solve_info *info) {
    if (!c || !A64 || !Ai || !b || !x || restart < 1 || restart > kGmresMaxRestart)
        return fail(HGB_ERR_ARG, "ir_gmres: bad arguments (restart 1..%d)", kGmresMaxRestart);
    if (csr_dtype(A64) != HGB_F64) return fail(HGB_ERR_ARG, "ir_gmres: the outer matrix must be F64");
    if (!real_inner(csr_dtype(Ai))) return fail(HGB_ERR_ARG, "ir_gmres: the inner matrix must be F32 or BF16");
    if (Mi && !real_inner(ilu_store(Mi))) return fail(HGB_ERR_ARG, "ir_gmres: the inner preconditioner must store F32 or BF16");
    const long n = csr_rows(A64);
    if (csr_rows(Ai) != n || csr_cols(A64) != n || csr_cols(Ai) != n || (Mi && ilu_n(Mi) != n))
        return fail(HGB_ERR_ARG, "ir_gmres: sizes");
    if (max_inner < 1 || max_outer < 0 || !(inner_rtol > 0.0)) return fail(HGB_ERR_ARG, "ir_gmres: limits");
    DeviceGuard g(c->device);
    double *r64 = nullptr;
    float *r32 = nullptr, *d32 = nullptr;
    int st = HGB_OK;
    int total = 0, outer = 0;
    double res = 0.0;
    long long launches = 0;
    const int cycles = (max_inner + restart - 1) / restart;
    do {
        if (ws_alloc(c, &r64, n) || ws_alloc(c, &r32, n) || ws_alloc(c, &d32, n)) {
            st = cuda_fail(cudaErrorMemoryAllocation, "ir_gmres workspace");
            break;
        }
        for (;;) {
            if ((st = true_residual(c, A64, b, x, r64, &res, &launches))) break;
            if (res < tol || res == 0.0 || outer >= max_outer || !(res == res)) break;   // 0: x is exact
            f64_to_f32_kernel<<<ew_grid(c, n), 256, 0, c->stream>>>(n, r64, r32);
            zero_f32_kernel<<<ew_grid(c, n), 256, 0, c->stream>>>(n, d32);
            launches += 3;   // residual cast, zero, update
            // as the refinement CG: this sweep reduces its (preconditioned) residual as far as the
            // target needs with a factor 2 of margin, never by less than inner_rtol
            const double rel = std::min(0.5, std::max(inner_rtol, 0.5 * tol / res));
            int it = 0, cyc = 0;
            double ires = 0.0;
            if (csr_dtype(Ai) == HGB_F32)
                st = gmres_run<float, float>(c, Ai, Mi, restart, r32, d32, 0.0, rel, cycles, &it, &cyc, &ires, &launches);
            else
                st = gmres_run<uint16_t, float>(c, Ai, Mi, restart, r32, d32, 0.0, rel, cycles, &it, &cyc, &ires, &launches);
            if (st) break;
            total += it;
            add_f32_to_f64_kernel<<<ew_grid(c, n), 256, 0, c->stream>>>(n, d32, x);
            if ((st = launch_check("ir update"))) break;
            outer++;
        }
    } while (0);
    ws_free(c, r64);
    ws_free(c, r32);
    ws_free(c, d32);
    if (st) return st;
    if (info) {
        info->iterations = total;
        info->outer = outer;
        info->residual = res;
        info->true_residual = res;
        info->kernel_launches = launches;
    }
    if (!(res < tol || res == 0.0)) return fail(HGB_ERR_NOT_CONVERGED, "ir_gmres: ||b-Ax|| = %g after %d sweeps (tol %g)", res, outer, tol);
    return HGB_OK;
}

// ========================================================== host-buffer (mixed) solve ====
extern "C" int hgb_mixed_cg_solve(hgb_ctx *c, int n, int nnz, const int *pntr_h, const int *indx_h, const double *vals_h,
                                  hgb_ilu *M, const double *b_h, double *x_h, double tol, int max_iter,
                                  hgb_solve_info *info) {
    if (!c || n <= 0 || nnz < 0 || !pntr_h || !indx_h || !vals_h || !b_h || !x_h) return fail(HGB_ERR_ARG, "mixed_cg: bad arguments");
    DeviceGuard g(c->device);
    auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
    size_t op = 0, oi = op + al(sizeof(int) * (n + 1)), ov = oi + al(sizeof(int) * (size_t)nnz);
    size_t ob = ov + al(sizeof(double) * (size_t)nnz), ox = ob + al(sizeof(double) * n), total = ox + al(sizeof(double) * n);
    if (c->arena_bytes < total) {
        cudaFree(c->arena);
        c->arena = nullptr;
        c->arena_bytes = 0;
        HGB_CUDA(cudaMalloc(&c->arena, total));
        c->arena_bytes = total;
    }
    char *base = (char *)c->arena;
    int *dp = (int *)(base + op), *di = (int *)(base + oi);
    double *dv = (double *)(base + ov), *db = (double *)(base + ob), *dx = (double *)(base + ox);
    // the loads (gpu_engine::load, wax/hala_lib_extensions.hpp:137-146) in chunks on the copy stream,
    // ordered after the caller's earlier work on the context's stream and before the solve
    HGB_CUDA(cudaEventRecord(c->ev_in, c->stream));
    HGB_CUDA(cudaStreamWaitEvent(c->copy, c->ev_in, 0));
    HGB_TRY(h2d_chunked(c, c->copy, dp, pntr_h, sizeof(int) * (n + 1)));
    HGB_TRY(h2d_chunked(c, c->copy, di, indx_h, sizeof(int) * (size_t)nnz));
    HGB_TRY(h2d_chunked(c, c->copy, dv, vals_h, sizeof(double) * (size_t)nnz));
    HGB_TRY(h2d_chunked(c, c->copy, db, b_h, sizeof(double) * n));
    HGB_TRY(h2d_chunked(c, c->copy, dx, x_h, sizeof(double) * n));
    HGB_CUDA(cudaEventRecord(c->ev_out, c->copy));
    HGB_CUDA(cudaStreamWaitEvent(c->stream, c->ev_out, 0));
    hgb_csr *A = nullptr;
    HGB_TRY(hgb_csr_create(c, n, n, nnz, dp, di, dv, HGB_F64, &A));
    int st = hgb_cg_solve(c, A, M, db, dx, tol, max_iter, info);
    hgb_csr_destroy(A);
    if (st) return st;
    HGB_CUDA(cudaMemcpyAsync(x_h, dx, sizeof(double) * n, cudaMemcpyDeviceToHost, c->stream));
    HGB_CUDA(cudaStreamSynchronize(c->stream));
    return HGB_OK;
}

namespace hgb {
__global__ void f64_to_inner_kernel(long n, const double *__restrict__ a, float *f32, uint16_t *b16) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        float v = (float)a[i];
        if (f32) f32[i] = v;
        if (b16) {
            uint32_t u = __float_as_uint(v);
            b16[i] = ((u & 0x7fffffffu) > 0x7f800000u) ? (uint16_t)((u >> 16) | 0x40u)
                                                      : (uint16_t)((u + 0x7fffu + ((u >> 16) & 1u)) >> 16);
        }
    }
}
}  // namespace hgb

// Host-buffer mixed solves: pntr/indx/vals (FP64) and b/x are loaded into the context's arena, the
// inner matrix is converted on the device to Mi's store precision, the solver runs on the device
// copies and x is read back (also when the solve did not converge).
template <typename Solve>
static int mixed_host_solve(hgb_ctx *c, const char *what, int n, int nnz, const int *pntr_h, const int *indx_h,
                            const double *vals_h, hgb_ilu *Mi, const double *b_h, double *x_h, hgb_solve_info *info,
                            Solve solve) {
    if (!c || n <= 0 || nnz < 0 || !pntr_h || !indx_h || !vals_h || !b_h || !x_h || !Mi)
        return fail(HGB_ERR_ARG, "%s: bad arguments", what);
    if (!real_inner(ilu_store(Mi))) return fail(HGB_ERR_ARG, "%s: the preconditioner must store F32 or BF16", what);
    DeviceGuard g(c->device);
    // the inner operator is FP32 whatever the factor's store: BF16 values shift the operator (on the
    // 128^3 system the rounded diagonal moves it by nine times its smallest eigenvalue) and the
    // refinement's fixed point with it, while a BF16 factor only changes the preconditioner
    auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
    size_t op = 0, oi = op + al(sizeof(int) * (n + 1)), ov = oi + al(sizeof(int) * (size_t)nnz);
    size_t ow = ov + al(sizeof(double) * (size_t)nnz), ob = ow + al(sizeof(float) * (size_t)nnz);
    size_t ox = ob + al(sizeof(double) * n), total = ox + al(sizeof(double) * n);
    if (c->arena_bytes < total) {
        cudaFree(c->arena);
        c->arena = nullptr;
        c->arena_bytes = 0;
        HGB_CUDA(cudaMalloc(&c->arena, total));
        c->arena_bytes = total;
    }
    char *base = (char *)c->arena;
    int *dp = (int *)(base + op), *di = (int *)(base + oi);
    double *dv = (double *)(base + ov), *db = (double *)(base + ob), *dx = (double *)(base + ox);
    void *dw = base + ow;
    // The loads in chunks on the copy stream, overlapped with the conversion of the values to the
    // inner precision on the context's stream: each chunk of values is converted as soon as it has
    // landed, while the next chunks are in flight.
    HGB_CUDA(cudaEventRecord(c->ev_in, c->stream));
    HGB_CUDA(cudaStreamWaitEvent(c->copy, c->ev_in, 0));
    HGB_TRY(h2d_chunked(c, c->copy, dp, pntr_h, sizeof(int) * (n + 1)));
    HGB_TRY(h2d_chunked(c, c->copy, di, indx_h, sizeof(int) * (size_t)nnz));
    constexpr long kChunk = 1L << 21;   // values per conversion chunk (16 MB of FP64)
    for (long o = 0; o < nnz; o += kChunk) {
        const long m = std::min(kChunk, (long)nnz - o);
        HGB_TRY(h2d_chunked(c, c->copy, dv + o, vals_h + o, sizeof(double) * (size_t)m));
        HGB_CUDA(cudaEventRecord(c->ev_out, c->copy));
        HGB_CUDA(cudaStreamWaitEvent(c->stream, c->ev_out, 0));   // waits on this record, not later ones
        f64_to_inner_kernel<<<ew_grid(c, m), 256, 0, c->stream>>>(
            m, dv + o, (float *)dw + o, nullptr);
        HGB_TRY(launch_check("f64_to_inner_kernel"));
    }
    HGB_TRY(h2d_chunked(c, c->copy, db, b_h, sizeof(double) * n));
    HGB_TRY(h2d_chunked(c, c->copy, dx, x_h, sizeof(double) * n));
    HGB_CUDA(cudaEventRecord(c->ev_out, c->copy));
    HGB_CUDA(cudaStreamWaitEvent(c->stream, c->ev_out, 0));
    hgb_csr *A64 = nullptr, *Ai = nullptr;
    HGB_TRY(hgb_csr_create(c, n, n, nnz, dp, di, dv, HGB_F64, &A64));
    int st = hgb_csr_create(c, n, n, nnz, dp, di, dw, HGB_F32, &Ai);
    if (!st) st = solve(A64, Ai, db, dx);
    hgb_csr_destroy(A64);
    hgb_csr_destroy(Ai);
    if (info) info->kernel_launches += 1;
    if (st && st != HGB_ERR_NOT_CONVERGED) return st;
    HGB_CUDA(cudaMemcpyAsync(x_h, dx, sizeof(double) * n, cudaMemcpyDeviceToHost, c->stream));
    HGB_CUDA(cudaStreamSynchronize(c->stream));
    return st;
}

extern "C" int hgb_mixed_ir_pcg_solve(hgb_ctx *c, int n, int nnz, const int *pntr_h, const int *indx_h,
                                      const double *vals_h, hgb_ilu *Mi, const double *b_h, double *x_h,
                                      double tol, double inner_rtol, int max_inner, int max_outer,
                                      hgb_solve_info *info) {
    return mixed_host_solve(c, "mixed_ir_pcg", n, nnz, pntr_h, indx_h, vals_h, Mi, b_h, x_h, info,
                            [&](hgb_csr *A64, hgb_csr *Ai, const double *db, double *dx) {
                                return hgb_ir_pcg_solve(c, A64, Ai, Mi, db, dx, tol, inner_rtol, max_inner, max_outer,
                                                        info);
                            });
}

extern "C" int hgb_mixed_ru_pcg_solve(hgb_ctx *c, int n, int nnz, const int *pntr_h, const int *indx_h,
                                      const double *vals_h, hgb_ilu *Mi, const double *b_h, double *x_h,
                                      double tol, double delta, int max_iter, hgb_solve_info *info) {
    return mixed_host_solve(c, "mixed_ru_pcg", n, nnz, pntr_h, indx_h, vals_h, Mi, b_h, x_h, info,
                            [&](hgb_csr *A64, hgb_csr *Ai, const double *db, double *dx) {
                                return hgb_ru_pcg_solve(c, A64, Ai, Mi, db, dx, tol, delta, max_iter, info);
                            });
}
