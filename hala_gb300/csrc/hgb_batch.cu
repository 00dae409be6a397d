// Batched CG for many independent sparse SPD systems of uneven size.
//
// The batch is a block-diagonal CSR (global column indices) with system row offsets sys_ptr.  Per
// system: FP32 CG, FP64 iterative refinement against the FP64 residual of the FP32-stored matrix,
// stopping at ||b - A x|| <= rtol ||b|| per system.  Work items are handed out by atomic tickets,
// largest systems first, in persistent launches that run side by side:
//
//  - batch_onchip_kernel: a CTA keeps the whole system on chip for its iterations: the off-diagonal
//    entries in shared memory (FP32 value, 16-bit column; the rows sorted by length and cut into slices
//    of 32, entry k of a slice's rows side by side, so that a warp's reads are consecutive), the
//    search direction beside them, a thread's rows of the other vectors in registers.  The row order, the
//    columns and the entries' positions are laid out once per batch (the pattern is the batch's own);
//    the values are read at every solve.  Inner products are compensated FP32 sums (two-product and
//    two-sum), and the scalars are formed from such pairs: an FP64 instruction holds its SM quarter's
//    unit for 62 cycles, and FP64 inner products with a division per thread took more time than
//    the matrix.  A pair holds 46 to 48 bits, of which the step and the direction's factor, floats, keep 24.  Its range
//    is FP32's: a matrix far from 1 is solved scaled by a power of two, and the residual and the direction change
//    their unit as they shrink.  Four shapes by the system's size in shared memory (kShapes).
//    Bound: the shared-memory gathers of the direction (about 3.5 of 5.5 cycles per 32 entries).
//  - batch_cg_kernel for systems that do not fit: vectors in shared memory, the matrix streamed from
//    L2; a "large" item is one system solved by the whole CTA, a "small" item packs up to (threads/32)
//    systems, one per warp.  Its block size and warp/CTA threshold are the batch's configuration,
//    which hgb_batch_autotune chooses by timing the candidates and caches in a small text file.
//
// 4,096 graph Laplacians of 64 to 4,096 rows to 1e-12 (GB300): 4.9 ms; 15.0 ms with every system in
// batch_cg_kernel.
#include "hgb_internal.cuh"
#include "hgb_kernels.cuh"

#include <algorithm>
#include <chrono>
#include <cstring>
#include <fstream>
#include <sstream>
#include <string>
#include <vector>

namespace hgb {

constexpr int kBatchSmem = 64 * 1024;    // per CTA: 4 float vectors of up to 4096 rows
constexpr int kBatchUnroll = 4;          // matrix entries whose loads are issued together

// ------------------------------------------------------------------ on-chip systems ------
// a sum held as a pair of floats (s the rounded sum, c what rounding left)
struct Df {
    float s, c;
};
// acc += a * b: the product and the sum with their rounding errors
__device__ __forceinline__ void df_fma(Df &acc, float a, float b) {
    const float h = __fmul_rn(a, b), e = __fmaf_rn(a, b, -h);
    const float t = __fadd_rn(acc.s, h), z = __fsub_rn(t, acc.s);
    const float err = __fadd_rn(__fsub_rn(acc.s, __fsub_rn(t, z)), __fsub_rn(h, z));
    acc.s = t;
    acc.c = __fadd_rn(acc.c, __fadd_rn(err, e));
}
__device__ __forceinline__ Df df_add(Df x, Df y) {
    const float t = __fadd_rn(x.s, y.s), z = __fsub_rn(t, x.s);
    const float err = __fadd_rn(__fsub_rn(x.s, __fsub_rn(t, z)), __fsub_rn(y.s, z));
    return Df{t, __fadd_rn(__fadd_rn(x.c, y.c), err)};
}
__device__ __forceinline__ Df df_normal(Df x) {   // |c| at most half an ulp of s
    const float t = __fadd_rn(x.s, x.c);
    return Df{t, __fsub_rn(x.c, __fsub_rn(t, x.s))};
}
// x / y rounded to float (a quotient and its correction)
__device__ __forceinline__ float df_div(Df x, Df y) {
    const float q = __fdiv_rn(x.s, y.s);
    const float r = __fadd_rn(__fmaf_rn(-q, y.s, x.s), __fsub_rn(x.c, __fmul_rn(q, y.c)));
    return isfinite(q) ? __fadd_rn(q, __fdiv_rn(r, y.s)) : q;
}
template <int N>
__device__ __forceinline__ Df df_lanes(Df v) {   // over groups of N lanes
#pragma unroll
    for (int o = N / 2; o > 0; o >>= 1) v = df_add(v, Df{__shfl_xor_sync(0xffffffffu, v.s, o), __shfl_xor_sync(0xffffffffu, v.c, o)});
    return v;
}

constexpr int kLenMax = 255;           // off-diagonal entries of a row
constexpr int kOnchipHead = 544;       // bytes of the reduction buffers
// shared memory of a system of n rows whose slices' widths sum to wsum
inline long onchip_bytes(long n, long wsum) { return kOnchipHead + 4 * ((n + 31) & ~31L) + 32 * 6 * wsum; }
// {threads, rows per thread, CTAs per SM, shared memory per CTA}: 16 warps of 128 registers on an SM in
// every shape (32 warps of 64 registers, four rows a thread: 5.2 against 4.8 ms for the 4,096 systems below)
struct OnchipShape {
    int threads, rpt, per_sm;
    long smem;
};
constexpr int kNumShapes = 4;
constexpr OnchipShape kShapes[kNumShapes] = {{512, 8, 1, 226 * 1024}, {256, 8, 2, 112 * 1024}, {128, 8, 4, 55 * 1024}, {64, 8, 8, 27 * 1024}};

// the laid-out systems: rows in sorted order, 32 to a slice
struct OnchipLayout {
    const long *img;         // [S] first entry of a system's image
    const int *slice0;       // [S] its first slice
    const int2 *slice;       // [slices] {first entry / 32 in the system's image, width}
    const unsigned short *orig;   // [rows] the row that sorted row holds
    const int *dpos;         // [rows] position of its diagonal entry, or -1
    const int *pos;          // [entries] positions in vals, -1: padding
    const unsigned short *col;    // [entries] 4 * the sorted row of the column
    double *xs;              // [rows] the solution in sorted order
};

struct BatchArgs {
    int nitems;
    const int *item_sys;     // [nitems * wpb] system ids (-1 padding); large items use slot 0
    const int *item_large;   // [nitems]
    const int *sys_ptr;      // [S + 1]
    const int *pntr, *indx;
    const float *vals;
    const double *b;
    double *x;
    int *iters;              // [S] total inner iterations (may be null)
    double *relres;          // [S] final ||b - Ax|| / ||b|| (may be null)
    double rtol, inner_rtol;
    int max_inner, max_outer;
    int *ticket;             // [2] self-resetting
    int *err;
};

struct WarpGroup {
    __device__ int rank() const { return threadIdx.x & 31; }
    __device__ int size() const { return 32; }
    __device__ void sync() const { __syncwarp(); }
    __device__ double sum(double v) const { return warp_sum(v); }
};

struct CtaGroup {
    double *red;   // >= 33 doubles of shared memory
    __device__ int rank() const { return threadIdx.x; }
    __device__ int size() const { return blockDim.x; }
    __device__ void sync() const { __syncthreads(); }
    __device__ double sum(double v) const {
        v = warp_sum(v);
        const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
        if (lane == 0) red[w] = v;
        __syncthreads();
        if (w == 0) {
            double t = (lane < (int)(blockDim.x >> 5)) ? red[lane] : 0.0;
            t = warp_sum(t);
            if (lane == 0) red[32] = t;
        }
        __syncthreads();
        return red[32];
    }
};

// One system: rows [r0, r0+n) of the batch; sm holds 4 float vectors of n entries.
template <class G>
__device__ void solve_system(const G &g, const BatchArgs &A, int s, float *sm) {
    const int r0 = A.sys_ptr[s], n = A.sys_ptr[s + 1] - r0;
    float *r = sm, *p = sm + n, *q = sm + 2 * n, *d = sm + 3 * n;
    const int t0 = g.rank(), ts = g.size();
    double bb = 0.0;
    for (int i = t0; i < n; i += ts) bb += A.b[r0 + i] * A.b[r0 + i];
    const double bnorm = sqrt(g.sum(bb));
    const double target = A.rtol * bnorm;
    int total = 0;
    double res = 0.0;
    for (int outer = 0;; outer++) {
        // FP64 residual of the stored (FP32) matrix: r = b - A x
        double rr = 0.0;
        for (int i = t0; i < n; i += ts) {
            const int row = r0 + i;
            double acc = A.b[row];
            const int kb = __ldg(A.pntr + row), ke = __ldg(A.pntr + row + 1);
            for (int k = kb; k < ke; k += kBatchUnroll) {
                float vv[kBatchUnroll];
                double xv[kBatchUnroll];
#pragma unroll
                for (int u = 0; u < kBatchUnroll; u++)
                    if (k + u < ke) {
                        vv[u] = __ldg(A.vals + k + u);
                        xv[u] = A.x[__ldg(A.indx + k + u)];
                    }
#pragma unroll
                for (int u = 0; u < kBatchUnroll; u++)
                    if (k + u < ke) acc -= (double)vv[u] * xv[u];
            }
            r[i] = (float)acc;
            d[i] = 0.0f;
            rr += acc * acc;
        }
        res = sqrt(g.sum(rr));
        if (!(res > target) || outer >= A.max_outer || !(res == res)) break;
        // inner FP32 CG on A d = r from d = 0 (solve_cg_core's order, identity preconditioner)
        double rz = 0.0;
        for (int i = t0; i < n; i += ts) {
            p[i] = r[i];
            rz += (double)r[i] * r[i];
        }
        g.sync();
        rz = g.sum(rz);
        const double stop2 = A.inner_rtol * A.inner_rtol * rz;
        for (int it = 0; it < A.max_inner; it++) {
            double pq = 0.0;
            for (int i = t0; i < n; i += ts) {
                const int row = r0 + i;
                const int kb = __ldg(A.pntr + row), ke = __ldg(A.pntr + row + 1);
                float acc = 0.0f;
                // entries kBatchUnroll at a time, their loads issued together (the row's matrix
                // comes from L2: one round trip per group, not per entry); the sum keeps the order
                for (int k = kb; k < ke; k += kBatchUnroll) {
                    float vv[kBatchUnroll];
                    int cc[kBatchUnroll];
#pragma unroll
                    for (int u = 0; u < kBatchUnroll; u++)
                        if (k + u < ke) {
                            vv[u] = __ldg(A.vals + k + u);
                            cc[u] = __ldg(A.indx + k + u);
                        }
#pragma unroll
                    for (int u = 0; u < kBatchUnroll; u++)
                        if (k + u < ke) acc += vv[u] * p[cc[u] - r0];
                }
                q[i] = acc;
                pq += (double)p[i] * acc;
            }
            pq = g.sum(pq);
            const float a = (float)(rz / pq);
            double nr = 0.0;
            for (int i = t0; i < n; i += ts) {
                d[i] += a * p[i];
                float ri = r[i] - a * q[i];
                r[i] = ri;
                nr += (double)ri * ri;
            }
            nr = g.sum(nr);
            total++;
            if (nr < stop2 || !(nr == nr)) break;
            const float beta = (float)(nr / rz);
            for (int i = t0; i < n; i += ts) p[i] = r[i] + beta * p[i];
            rz = nr;
            g.sync();
        }
        for (int i = t0; i < n; i += ts) A.x[r0 + i] += (double)d[i];
        g.sync();
        __threadfence_block();
    }
    if (g.rank() == 0) {
        if (A.iters) A.iters[s] = total;
        if (A.relres) A.relres[s] = bnorm > 0 ? res / bnorm : res;
    }
    g.sync();
}

// A pair of floats has FP32's range.  A matrix whose largest diagonal entry (its largest entry, A being positive
// definite; top: its bits) lies outside [2^-10, 2^20) is solved as 2^-k A, that entry in [1, 2), for 2^k x.  Scales the image
// and the solution; returns the matrix's factor (as two: 2^-k alone may be out of range) and leaves the solution's in *back.
// (A function of its own: inlined, it took the systems that need none of it 4.9 -> 5.0 ms per 4,096.)
template <int T>
__device__ __noinline__ float2 onchip_scale(int top, float *v, int ne, double *xs, int n, double *back) {
    if (!(top > 0 && top < 0x7f800000 && (unsigned)(ilogbf(__int_as_float(top)) + 10) >= 30u)) return make_float2(1.0f, 1.0f);
    const int t = threadIdx.x, k = ilogbf(__int_as_float(top));
    const float s1 = scalbnf(1.0f, -k / 2), s2 = scalbnf(1.0f, -(k - k / 2));
    for (int i = t; i < ne; i += T) v[i] = v[i] * s1 * s2;
    for (int i = t; i < n; i += T) xs[i] *= scalbn(1.0, k);
    if (t == 0) *back = scalbn(1.0, -k);
    __threadfence_block();
    __syncthreads();
    return make_float2(s1, s2);
}
template <int T, int RPT, int MINB>
__global__ void __launch_bounds__(T, MINB)
batch_onchip_kernel(BatchArgs A, OnchipLayout Y, const int *__restrict__ items, int nitems, int *ticket) {
    constexpr int NW = T / 32, U = 8;   // U: entries per round
    extern __shared__ __align__(16) unsigned char osm[];
    Df *red = (Df *)osm;   // [2][NW + 1]
    static_assert(sizeof(Df) * 2 * (NW + 1) <= kOnchipHead && NW <= 32, "head");
    __shared__ double dred[33];
    __shared__ int item, top;
    __shared__ double back;   // the solution's scale
    __shared__ double stop;   // the inner iteration's limit on <r, r>, and as a pair
    __shared__ Df stop_pair;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    int buf = 0;
    // the CTA's sum, the same bits in every thread.  The second stage in one warp: in all of them at
    // once, without the second barrier, its instructions cost more (1630 against 1250 cycles at 32 warps).
    auto sum = [&](Df v) -> Df {
        v = df_lanes<32>(v);
        Df *r = red + buf * (NW + 1);
        buf ^= 1;
        if (lane == 0) r[w] = v;
        __syncthreads();
        if (w == 0) {
            v = df_normal(df_lanes<NW>(r[lane & (NW - 1)]));
            if (lane == 0) r[NW] = v;
        }
        __syncthreads();
        return r[NW];
    };
    const CtaGroup g{dred};
    float *p = (float *)(osm + kOnchipHead);
    for (;;) {
        __syncthreads();
        if (t == 0) {
            item = atomicAdd(ticket, 1);
            top = 0;
            back = 1.0;
        }
        __syncthreads();
        if (item >= nitems) break;
        const int s = items[item], r0 = A.sys_ptr[s], n = A.sys_ptr[s + 1] - r0, ns = (n + 31) >> 5;
        float *v = p + ns * 32;
        const int2 *sl = Y.slice + Y.slice0[s];
        const int2 last = __ldg(sl + ns - 1);
        const int ne = (last.x + last.y) * 32;
        unsigned short *c = (unsigned short *)(v + ne);
        // ---- the system's image: values through their positions, columns as laid out
        {
            const int *pos = Y.pos + Y.img[s];
            const unsigned short *col = Y.col + Y.img[s];
            for (int i = t * 4; i < ne; i += T * 4) {   // ne and the image are multiples of 32 entries
                const int4 q = __ldg((const int4 *)(pos + i));
                const uint2 k = __ldg((const uint2 *)(col + i));
                float4 a;
                a.x = q.x >= 0 ? __ldg(A.vals + q.x) : 0.0f;
                a.y = q.y >= 0 ? __ldg(A.vals + q.y) : 0.0f;
                a.z = q.z >= 0 ? __ldg(A.vals + q.z) : 0.0f;
                a.w = q.w >= 0 ? __ldg(A.vals + q.w) : 0.0f;
                *(float4 *)(v + i) = a;
                *(uint2 *)(c + i) = k;
            }
        }
        // a thread's rows: t, t + T, ... in sorted order; slice j of its warp
        int slice[RPT];   // {first entry / 32, width (8 bits)}
        float diag[RPT];
        double bb = 0.0;
        int big = 0;   // the bits of the largest |diagonal|
#pragma unroll
        for (int j = 0; j < RPT; j++) {
            const int row = t + j * T;
            slice[j] = 0;
            diag[j] = 0.0f;
            if (w + j * NW < ns) {
                const int2 e = __ldg(sl + w + j * NW);
                slice[j] = e.x << 8 | e.y;
                p[row] = 0.0f;   // also the rows past n
            }
            if (row < n) {
                const int d = Y.dpos[r0 + row], o = r0 + Y.orig[r0 + row];
                if (d >= 0) diag[j] = __ldg(A.vals + d);
                big = max(big, __float_as_int(diag[j]) & 0x7fffffff);
                Y.xs[r0 + row] = A.x[o];
                const double bi = A.b[o];
                bb += bi * bi;
            }
        }
        big = __reduce_max_sync(0xffffffffu, big);
        if (lane == 0) atomicMax(&top, big);
        __threadfence_block();
        const double bnorm = sqrt(g.sum(bb));   // its barriers: the image is in
        const float2 sc = onchip_scale<T>(top, v, ne, Y.xs + r0, n, &back);
#pragma unroll
        for (int j = 0; j < RPT; j++) diag[j] = diag[j] * sc.x * sc.y;
        const double target = A.rtol * bnorm;
        int total = 0;
        double res = 0.0;
        for (int outer = 0;; outer++) {
            // FP64 residual of the stored (FP32) matrix: b - A x
            double rr = 0.0, r64[RPT];
#pragma unroll
            for (int j = 0; j < RPT; j++) {
                r64[j] = 0.0;
                if (t + j * T >= n) continue;
                const double *xs = Y.xs + r0;
                double acc = A.b[r0 + Y.orig[r0 + t + j * T]] - (double)diag[j] * xs[t + j * T];
                const int off = (slice[j] >> 8) * 32 + lane, wid = slice[j] & 255;
                const float *vp = v + off;
                const unsigned short *cp = c + off;
                for (int k = 0; k < wid; k += kBatchUnroll) {
                    float vv[kBatchUnroll];
                    double xv[kBatchUnroll];
#pragma unroll
                    for (int u = 0; u < kBatchUnroll; u++)
                        if (k + u < wid) {
                            vv[u] = vp[(k + u) * 32];
                            xv[u] = xs[cp[(k + u) * 32] >> 2];
                        }
#pragma unroll
                    for (int u = 0; u < kBatchUnroll; u++)
                        if (k + u < wid) acc -= (double)vv[u] * xv[u];
                }
                r64[j] = acc;
                rr += acc * acc;
            }
            res = sqrt(g.sum(rr));
            if (!(res > target) || outer >= A.max_outer || !(res == res)) break;
            // the FP32 right-hand side, scaled by a power of two to a norm near 1 (exact, and taken back
            // from the correction): its squares stay far from FP32's range limits
            const int ex = min(max(ilogb(res), -1000), 1000);
            const double down = scalbn(1.0, -ex);
            float r[RPT], d[RPT], q[RPT];
            Df acc{0.0f, 0.0f};
#pragma unroll
            for (int j = 0; j < RPT; j++) {
                r[j] = (float)(r64[j] * down);
                d[j] = 0.0f;
                if (t + j * T < n) p[t + j * T] = r[j];
                df_fma(acc, r[j], r[j]);
            }
            Df rz = sum(acc);
            auto set_stop = [&](double v) {   // (the pair not 0: a residual that vanishes ends the iteration)
                const float h = fmaxf((float)v, 0x1p-126f);
                stop = v;
                stop_pair = Df{h, (float)v >= h ? (float)(v - (double)h) : 0.0f};
            };
            if (t == 0) set_stop(A.inner_rtol * A.inner_rtol * ((double)rz.s + (double)rz.c));
            __syncthreads();
            Df stop2 = stop_pair;
            float unit = 1.0f;   // of d, the residual and the direction
            // inner FP32 CG on A d = r from d = 0 (solve_cg_core's order, identity preconditioner)
            for (int it = 0; it < A.max_inner; it++) {
                acc = Df{0.0f, 0.0f};
#pragma unroll
                for (int j = 0; j < RPT; j++) {
                    q[j] = 0.0f;
                    if (w + j * NW < ns) {
                        const float pr = p[t + j * T];
                        float a = diag[j] * pr;
                        const int off = (slice[j] >> 8) * 32 + lane;
                        const float *vp = v + off;
                        const unsigned short *cp = c + off;
                        // U entries at a time: their columns and values, then the gathers, two
                        // shared-memory round trips for all of them (the width is the same in all lanes)
                        for (int k = slice[j] & 255; k > 0; k -= U, vp += 32 * U, cp += 32 * U) {
                            unsigned cc[U];
                            float vv[U], pv[U];
#pragma unroll
                            for (int u = 0; u < U; u++)
                                if (u < k) cc[u] = cp[32 * u];
#pragma unroll
                            for (int u = 0; u < U; u++)
                                if (u < k) vv[u] = vp[32 * u];
#pragma unroll
                            for (int u = 0; u < U; u++)
                                if (u < k) pv[u] = *(const float *)((const char *)p + cc[u]);
#pragma unroll
                            for (int u = 0; u < U; u++)
                                if (u < k) a += vv[u] * pv[u];
                        }
                        q[j] = a;
                        df_fma(acc, pr, a);   // rows past n: 0
                    }
                }
                const float al = df_div(rz, sum(acc));
                acc = Df{0.0f, 0.0f};
#pragma unroll
                for (int j = 0; j < RPT; j++)
                    if (w + j * NW < ns) {
                        d[j] += al * p[t + j * T];
                        r[j] -= al * q[j];
                        df_fma(acc, r[j], r[j]);
                    }
                const Df nr = sum(acc);   // its barriers: the direction is no longer read
                total++;
                if (nr.s < stop2.s || (nr.s == stop2.s && nr.c < stop2.c) || !(nr.s == nr.s)) break;
                const float beta = df_div(nr, rz);
                rz = nr;
                if (__builtin_expect(nr.s < 0x1p-40f || nr.s > 0x1p60f, 0)) {
                    // another unit (a power of two): <r, r> leaves the range in which its parts' products are exact
                    const float f = nr.s < 1.0f ? 0x1p20f : 0x1p-20f;
                    if (unit < 0x1p-100f) break;   // the rest of d is far below its last bits
                    unit /= f;
                    rz = Df{nr.s * f * f, nr.c * f * f};
                    if (t == 0) set_stop(stop * ((double)f * (double)f));
                    __syncthreads();
                    stop2 = stop_pair;
#pragma unroll
                    for (int j = 0; j < RPT; j++)
                        if (w + j * NW < ns) {
                            r[j] *= f;
                            d[j] *= f;
                            p[t + j * T] *= f;
                        }
                }
#pragma unroll
                for (int j = 0; j < RPT; j++)
                    if (w + j * NW < ns) p[t + j * T] = r[j] + beta * p[t + j * T];
                __syncthreads();
            }
            const double up = scalbn((double)unit, ex);
#pragma unroll
            for (int j = 0; j < RPT; j++)
                if (t + j * T < n) Y.xs[r0 + t + j * T] += (double)d[j] * up;
            __threadfence_block();
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < RPT; j++)
            if (t + j * T < n) A.x[r0 + Y.orig[r0 + t + j * T]] = Y.xs[r0 + t + j * T] * back;
        if (t == 0) {
            if (A.iters) A.iters[s] = total;
            if (A.relres) A.relres[s] = bnorm > 0 ? res / bnorm : res;
        }
    }
    if (t == 0) {
        __threadfence();
        if (atomicAdd(ticket + 1, 1) == (int)gridDim.x - 1) {
            ticket[0] = 0;
            ticket[1] = 0;
        }
    }
}

// Layout, first pass, a CTA per system: off-diagonal entries of its rows, the rows sorted by them
// (longest first, equal ones in their order), the slices' widths.  out[s]: the sum of the widths, or -1
// for a system that cannot be laid out (a row with more than kLenMax, or more than 4096 rows).
__global__ void __launch_bounds__(256) batch_sort_kernel(int S, const int *__restrict__ sys_ptr, const int *__restrict__ pntr,
                                                         const int *__restrict__ indx, const int *__restrict__ slice0,
                                                         unsigned char *len, unsigned short *orig, int2 *slice, int *out) {
    __shared__ int cur[kLenMax + 1], many;
    const int t = threadIdx.x, lane = t & 31;
    for (int s = blockIdx.x; s < S; s += gridDim.x) {
        const int r0 = sys_ptr[s], n = sys_ptr[s + 1] - r0;
        __syncthreads();
        for (int k = t; k <= kLenMax; k += blockDim.x) cur[k] = 0;
        if (t == 0) many = n > 4096;
        __syncthreads();
        for (int i = t; i < n; i += blockDim.x) {
            int m = 0;
            for (int k = pntr[r0 + i]; k < pntr[r0 + i + 1]; k++) m += indx[k] != r0 + i;
            if (m > kLenMax) many = 1;
            len[r0 + i] = (unsigned char)min(m, kLenMax);
            atomicAdd(cur + min(m, kLenMax), 1);
        }
        __syncthreads();
        if (t < 32) {
            if (lane == 0) {
                int run = 0;
                for (int k = kLenMax; k >= 0; k--) {
                    const int c = cur[k];
                    cur[k] = run;
                    run += c;
                }
            }
            __syncwarp();
            for (int i0 = 0; i0 < n; i0 += 32) {
                const int i = i0 + lane, m = i < n ? len[r0 + i] : kLenMax + 1;
                const unsigned same = __match_any_sync(0xffffffffu, m);
                const int rank = __popc(same & ((1u << lane) - 1));
                if (i < n) orig[r0 + cur[m] + rank] = (unsigned short)i;
                __syncwarp();
                if (i < n && rank == 0) cur[m] += __popc(same);
                __syncwarp();
            }
            __threadfence_block();
            __syncwarp();
            int run = 0;
            for (int k0 = 0; 32 * k0 < n; k0 += 32) {   // a slice is as wide as its first row
                const int k = k0 + lane, m = 32 * k < n ? len[r0 + orig[r0 + 32 * k]] : 0;
                int v = m;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += u;
                }
                if (32 * k < n) slice[slice0[s] + k] = make_int2(run + v - m, m);
                run += __shfl_sync(0xffffffffu, v, 31);
            }
            if (lane == 0) out[s] = many ? -1 : run;
        }
    }
}

// second pass, a CTA per laid-out system (img[s] >= 0), a warp per slice.  A row's entries may come in any
// order: for every k the rows of the slice in turn take, of their remaining entries, one in the bank
// of shared memory that the fewest rows before them took, which halves the conflicts of the
// gathers (4,096 systems: 5.64 ms without, 5.40 with).
constexpr int kReorderMax = 48;   // entries of a row up to which it is reordered
__global__ void __launch_bounds__(128) batch_image_kernel(int S, const int *__restrict__ sys_ptr, const int *__restrict__ pntr,
                                                          const int *__restrict__ indx, const int *__restrict__ slice0,
                                                          const int2 *__restrict__ slice, const unsigned short *__restrict__ orig,
                                                          const long *__restrict__ img, int *pos, unsigned short *col, int *dpos) {
    __shared__ unsigned short inv[4096];
    __shared__ unsigned short lc[4][32][kReorderMax];   // a slice's rows: sorted rows of the columns left,
    __shared__ unsigned char lk[4][32][kReorderMax];    // and their places in the row
    __shared__ int taken[4][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int s = blockIdx.x; s < S; s += gridDim.x) {
        if (img[s] < 0) continue;
        const int r0 = sys_ptr[s], n = sys_ptr[s + 1] - r0;
        __syncthreads();
        for (int q = threadIdx.x; q < n; q += blockDim.x) inv[orig[r0 + q]] = (unsigned short)q;
        __syncthreads();
        for (int k = w; 32 * k < n; k += 4) {
            const int2 e = slice[slice0[s] + k];
            const int q = 32 * k + lane;
            const long at = img[s] + (long)e.x * 32 + lane;
            const bool reorder = e.y <= kReorderMax;
            int left = 0, kb = 0;
            if (q < n) {
                const int row = r0 + orig[r0 + q];
                int d = -1;
                kb = pntr[row];
                for (int i = kb; i < pntr[row + 1]; i++) {
                    if (indx[i] == row) {
                        d = i;
                        continue;
                    }
                    const unsigned short c = inv[indx[i] - r0];
                    if (reorder) {
                        lc[w][lane][left] = c;
                        lk[w][lane][left] = (unsigned char)(i - kb);
                    } else {
                        pos[at + 32 * left] = i;
                        col[at + 32 * left] = (unsigned short)(4 * c);
                    }
                    left++;
                }
                dpos[r0 + q] = d;
            }
            __syncwarp();
            if (!reorder) {
                for (; left < e.y; left++) {   // padding: 0 times the row's own entry of the direction
                    pos[at + 32 * left] = -1;
                    col[at + 32 * left] = (unsigned short)(4 * q);
                }
                continue;
            }
            for (int m = 0; m < e.y; m++) {
                taken[w][lane] = 0;
                __syncwarp();
                int place = -1, c = 0;
                for (int r = 0; r < 32; r++) {
                    const int nr = __shfl_sync(0xffffffffu, left, r);
                    if (nr == 0) break;   // rows are sorted: the ones below have none left either
                    const unsigned mine = lane < nr ? (unsigned)taken[w][lc[w][r][lane] & 31] << 8 | lane : 0xffffffffu;
                    const int best = (int)(__reduce_min_sync(0xffffffffu, mine) & 255);
                    const int bc = lc[w][r][best], bk = lk[w][r][best];
                    __syncwarp();
                    if (lane == 0) {
                        taken[w][bc & 31]++;
                        lc[w][r][best] = lc[w][r][nr - 1];
                        lk[w][r][best] = lk[w][r][nr - 1];
                    }
                    __syncwarp();
                    if (lane == r) {
                        place = bk;
                        c = bc;
                        left--;
                    }
                }
                const int lead = __shfl_sync(0xffffffffu, c, 0);   // padding reads what row 0 reads, times 0
                pos[at + 32 * m] = place >= 0 ? kb + place : -1;
                col[at + 32 * m] = (unsigned short)(4 * (place >= 0 ? c : lead));
            }
            __syncwarp();
        }
    }
}

// every column of a system's rows must fall inside that system (block-diagonal batch)
__global__ void batch_check_kernel(int S, const int *__restrict__ sys_ptr, const int *__restrict__ pntr,
                                   const int *__restrict__ indx, int *err) {
    for (int s = blockIdx.x; s < S; s += gridDim.x) {
        const int r0 = sys_ptr[s], r1 = sys_ptr[s + 1];
        for (int row = r0 + threadIdx.x; row < r1; row += blockDim.x)
            for (int k = pntr[row]; k < pntr[row + 1]; k++) {
                int c = indx[k];
                if (c < r0 || c >= r1) { atomicOr(err, DEV_ERR_CSR); break; }
            }
    }
}

static bool same_args(const BatchArgs &a, const BatchArgs &b) {
    return a.nitems == b.nitems && a.item_sys == b.item_sys && a.item_large == b.item_large &&
           a.sys_ptr == b.sys_ptr && a.pntr == b.pntr && a.indx == b.indx && a.vals == b.vals && a.b == b.b &&
           a.x == b.x && a.iters == b.iters && a.relres == b.relres && a.rtol == b.rtol &&
           a.inner_rtol == b.inner_rtol && a.max_inner == b.max_inner && a.max_outer == b.max_outer &&
           a.ticket == b.ticket && a.err == b.err;
}

__global__ void batch_cg_kernel(BatchArgs A) {
    extern __shared__ __align__(16) float bsm[];
    __shared__ double red[33];
    __shared__ int item;
    const int wpb = blockDim.x >> 5, w = threadIdx.x >> 5;
    for (;;) {
        if (threadIdx.x == 0) item = atomicAdd(A.ticket, 1);
        __syncthreads();
        const int it = item;
        __syncthreads();
        if (it >= A.nitems) break;
        if (A.item_large[it]) {
            CtaGroup g{red};
            solve_system(g, A, A.item_sys[it * wpb], bsm);
        } else {
            const int s = A.item_sys[it * wpb + w];
            if (s >= 0) {
                WarpGroup g;
                const int per_warp = kBatchSmem / (int)sizeof(float) / wpb;
                solve_system(g, A, s, bsm + w * per_warp);
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(A.ticket + 1, 1) == (int)gridDim.x - 1) {
            A.ticket[0] = 0;
            A.ticket[1] = 0;
        }
    }
}

}  // namespace hgb

using namespace hgb;

struct hgb_batch {
    hgb_ctx *ctx = nullptr;
    int S = 0, n_total = 0, nnz = 0;
    const int *sys_ptr = nullptr, *pntr = nullptr, *indx = nullptr;
    const float *vals = nullptr;
    std::vector<int> sizes;          // host copy of the system sizes
    std::vector<int> widths;         // sum of every system's slice widths, -1: not laid out
    void *layout = nullptr;          // the on-chip systems' layout (one allocation)
    OnchipLayout lay{};
    // systems solved on chip, by shape (kShapes), largest first; the others are the items below
    int *on_items[kNumShapes] = {};
    int on_count[kNumShapes] = {}, on_grid[kNumShapes] = {};
    cudaStream_t side[kNumShapes] = {};      // the shapes' launches run side by side, the largest first
    cudaEvent_t fork = nullptr, join[kNumShapes] = {};
    hgb_batch_config cfg{256, 256};
    int nitems = 0;
    int *item_sys = nullptr, *item_large = nullptr, *ticket = nullptr;
    // graph of the launches, keyed by the vectors it was captured with
    cudaGraphExec_t exec = nullptr;
    BatchArgs captured{};
};

namespace hgb {

static const void *onchip_kernel(int shape) {
    switch (shape) {
        case 0: return (const void *)batch_onchip_kernel<512, 8, 1>;
        case 1: return (const void *)batch_onchip_kernel<256, 8, 2>;
        case 2: return (const void *)batch_onchip_kernel<128, 8, 4>;
        default: return (const void *)batch_onchip_kernel<64, 8, 8>;
    }
}

// the smallest shape that holds system s, or -1
static int onchip_shape(const hgb_batch *B, int s) {
    if (B->widths[s] < 0) return -1;
    for (int k = kNumShapes - 1; k >= 0; k--)
        if (B->sizes[s] <= kShapes[k].threads * kShapes[k].rpt && onchip_bytes(B->sizes[s], B->widths[s]) <= kShapes[k].smem) return k;
    return -1;
}

// Lays the batch's systems out for the on-chip kernel (once per batch: the pattern is the batch's own).
static int onchip_layout(hgb_batch *B) {
    hgb_ctx *c = B->ctx;
    const int S = B->S;
    B->widths.assign(S, -1);
    std::vector<int> slice0(S + 1, 0);
    for (int s = 0; s < S; s++) slice0[s + 1] = slice0[s] + (B->sizes[s] + 31) / 32;
    const int slices = slice0[S];
    int *dslice0 = nullptr, *dout = nullptr, *dpos = nullptr, *pos = nullptr;
    unsigned char *len = nullptr;
    unsigned short *orig = nullptr, *col = nullptr;
    int2 *slice = nullptr;
    long *img = nullptr;
    double *xs = nullptr;
    std::vector<long> himg(S, -1);
    auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
    auto work = [&]() -> int {
        if (ws_alloc(c, &dslice0, S + 1) || ws_alloc(c, &dout, S) || ws_alloc(c, &len, B->n_total) ||
            ws_alloc(c, &orig, B->n_total) || ws_alloc(c, &slice, slices))
            return cuda_fail(cudaErrorMemoryAllocation, "batch_create");
        HGB_CUDA(cudaMemcpyAsync(dslice0, slice0.data(), sizeof(int) * (S + 1), cudaMemcpyHostToDevice, c->stream));
        const int g = std::min(S, c->num_sms * 8);
        batch_sort_kernel<<<g, 256, 0, c->stream>>>(S, B->sys_ptr, B->pntr, B->indx, dslice0, len, orig, slice, dout);
        HGB_TRY(launch_check("batch_sort_kernel"));
        HGB_CUDA(cudaMemcpyAsync(B->widths.data(), dout, sizeof(int) * S, cudaMemcpyDeviceToHost, c->stream));
        HGB_CUDA(cudaStreamSynchronize(c->stream));
        long entries = 0;
        for (int s = 0; s < S; s++)
            if (onchip_shape(B, s) >= 0) {
                himg[s] = entries;
                entries += 32L * B->widths[s];
            }
        // one allocation: {img, slice0, slice, orig, dpos, pos, col, xs}
        size_t o[8], total = 0;
        const size_t size[8] = {sizeof(long) * S, sizeof(int) * (S + 1), sizeof(int2) * slices, sizeof(short) * (size_t)B->n_total,
                                sizeof(int) * (size_t)B->n_total, sizeof(int) * (size_t)entries, sizeof(short) * (size_t)entries,
                                sizeof(double) * (size_t)B->n_total};
        for (int k = 0; k < 8; k++) {
            o[k] = total;
            total += al(size[k]);
        }
        if (cudaMalloc(&B->layout, total) != cudaSuccess) {
            // no room for it: every system streams its matrix
            cudaGetLastError();
            B->layout = nullptr;
            B->widths.assign(S, -1);
            return HGB_OK;
        }
        char *base = (char *)B->layout;
        img = (long *)(base + o[0]);
        int *ks0 = (int *)(base + o[1]);
        int2 *ksl = (int2 *)(base + o[2]);
        unsigned short *ko = (unsigned short *)(base + o[3]);
        dpos = (int *)(base + o[4]);
        pos = (int *)(base + o[5]);
        col = (unsigned short *)(base + o[6]);
        xs = (double *)(base + o[7]);
        HGB_CUDA(cudaMemcpyAsync(img, himg.data(), size[0], cudaMemcpyHostToDevice, c->stream));
        HGB_CUDA(cudaMemcpyAsync(ks0, dslice0, size[1], cudaMemcpyDeviceToDevice, c->stream));
        HGB_CUDA(cudaMemcpyAsync(ksl, slice, size[2], cudaMemcpyDeviceToDevice, c->stream));
        HGB_CUDA(cudaMemcpyAsync(ko, orig, size[3], cudaMemcpyDeviceToDevice, c->stream));
        batch_image_kernel<<<std::min(S, c->num_sms * 16), 128, 0, c->stream>>>(S, B->sys_ptr, B->pntr, B->indx, ks0, ksl, ko, img,
                                                                               pos, col, dpos);
        HGB_TRY(launch_check("batch_image_kernel"));
        HGB_CUDA(cudaStreamSynchronize(c->stream));
        B->lay = OnchipLayout{img, ks0, ksl, ko, dpos, pos, col, xs};
        return HGB_OK;
    };
    const int st = work();
    ws_free(c, dslice0);
    ws_free(c, dout);
    ws_free(c, len);
    ws_free(c, orig);
    ws_free(c, slice);
    return st;
}

// the on-chip shapes' items, launch grids, streams (once per batch)
static int onchip_plan(hgb_batch *B) {
    hgb_ctx *c = B->ctx;
    std::vector<int> list[kNumShapes];
    for (int s = 0; s < B->S; s++) {
        const int k = onchip_shape(B, s);
        if (k >= 0) list[k].push_back(s);
    }
    int least = 0, greatest = 0;
    HGB_CUDA(cudaDeviceGetStreamPriorityRange(&least, &greatest));
    HGB_CUDA(cudaEventCreateWithFlags(&B->fork, cudaEventDisableTiming));
    for (int k = 0; k < kNumShapes; k++) {
        B->on_count[k] = (int)list[k].size();
        if (list[k].empty()) continue;
        std::stable_sort(list[k].begin(), list[k].end(), [&](int a, int b) { return B->sizes[a] > B->sizes[b]; });
        HGB_CUDA(cudaMalloc(&B->on_items[k], sizeof(int) * list[k].size()));
        HGB_CUDA(cudaMemcpy(B->on_items[k], list[k].data(), sizeof(int) * list[k].size(), cudaMemcpyHostToDevice));
        // a CTA of the first shape needs a whole SM: it has to get one before the small ones
        HGB_CUDA(cudaStreamCreateWithPriority(&B->side[k], cudaStreamNonBlocking, std::min(least, greatest + k)));
        HGB_CUDA(cudaEventCreateWithFlags(&B->join[k], cudaEventDisableTiming));
        const void *f = onchip_kernel(k);
        HGB_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kShapes[k].smem));
        int per_sm = 0;
        HGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, kShapes[k].threads, kShapes[k].smem));
        B->on_grid[k] = std::max(1, std::min(B->on_count[k], c->num_sms * std::max(per_sm, 1)));
    }
    return HGB_OK;
}

static int batch_plan(hgb_batch *B, hgb_batch_config cfg) {
    hgb_ctx *c = B->ctx;
    const int wpb = cfg.block_threads / 32;
    const int warp_cap = kBatchSmem / (int)sizeof(float) / wpb / 4;   // rows per warp system
    const int cta_cap = kBatchSmem / (int)sizeof(float) / 4;
    int warp_max = std::min(cfg.warp_max_n, warp_cap);
    std::vector<int> order;
    for (int s = 0; s < B->S; s++)
        if (onchip_shape(B, s) < 0) order.push_back(s);
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return B->sizes[a] > B->sizes[b]; });
    std::vector<int> isys, ilarge;
    size_t k = 0;
    for (; k < order.size() && B->sizes[order[k]] > warp_max; k++) {
        if (B->sizes[order[k]] > cta_cap) return fail(HGB_ERR_UNSUPPORTED, "batch: system of %d rows > %d", B->sizes[order[k]], cta_cap);
        isys.push_back(order[k]);
        for (int j = 1; j < wpb; j++) isys.push_back(-1);
        ilarge.push_back(1);
    }
    while (k < order.size()) {
        for (int j = 0; j < wpb; j++) isys.push_back(k < order.size() ? order[k++] : -1);
        ilarge.push_back(0);
    }
    cudaFree(B->item_sys);
    cudaFree(B->item_large);
    B->item_sys = B->item_large = nullptr;
    B->nitems = (int)ilarge.size();
    HGB_CUDA(cudaMalloc(&B->item_sys, sizeof(int) * std::max<size_t>(isys.size(), 1)));
    HGB_CUDA(cudaMalloc(&B->item_large, sizeof(int) * std::max<size_t>(ilarge.size(), 1)));
    HGB_CUDA(cudaMemcpy(B->item_sys, isys.data(), sizeof(int) * isys.size(), cudaMemcpyHostToDevice));
    HGB_CUDA(cudaMemcpy(B->item_large, ilarge.data(), sizeof(int) * ilarge.size(), cudaMemcpyHostToDevice));
    B->cfg = cfg;
    if (B->exec) {
        cudaGraphExecDestroy(B->exec);
        B->exec = nullptr;
    }
    (void)c;
    return HGB_OK;
}

static int batch_launch(hgb_batch *B, const BatchArgs &A, cudaStream_t st) {
    hgb_ctx *c = B->ctx;
    int per_sm = 0;
    HGB_CUDA(cudaEventRecord(B->fork, st));
    for (int k = 0; k < kNumShapes; k++) {
        if (B->on_count[k] == 0) continue;
        HGB_CUDA(cudaStreamWaitEvent(B->side[k], B->fork, 0));
        BatchArgs a = A;
        int *ticket = B->ticket + 2 + 2 * k;
        void *args[] = {&a, &B->lay, &B->on_items[k], &B->on_count[k], &ticket};
        HGB_CUDA(cudaLaunchKernel(onchip_kernel(k), dim3(B->on_grid[k]), dim3(kShapes[k].threads), args, kShapes[k].smem, B->side[k]));
        HGB_CUDA(cudaEventRecord(B->join[k], B->side[k]));
        HGB_CUDA(cudaStreamWaitEvent(st, B->join[k], 0));
    }
    if (B->nitems == 0) return HGB_OK;
    HGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batch_cg_kernel, B->cfg.block_threads, kBatchSmem));
    int grid = std::max(1, std::min(B->nitems, c->num_sms * std::max(per_sm, 1)));
    batch_cg_kernel<<<grid, B->cfg.block_threads, kBatchSmem, st>>>(A);
    return launch_check("batch_cg_kernel");
}

static BatchArgs batch_args(hgb_batch *B, const double *b, double *x, double rtol, double inner_rtol, int max_inner,
                            int max_outer, int *iters, double *relres) {
    BatchArgs A{};
    A.nitems = B->nitems;
    A.item_sys = B->item_sys;
    A.item_large = B->item_large;
    A.sys_ptr = B->sys_ptr;
    A.pntr = B->pntr;
    A.indx = B->indx;
    A.vals = B->vals;
    A.b = b;
    A.x = x;
    A.iters = iters;
    A.relres = relres;
    A.rtol = rtol;
    A.inner_rtol = inner_rtol;
    A.max_inner = max_inner;
    A.max_outer = max_outer;
    A.ticket = B->ticket;
    A.err = B->ctx->err;
    return A;
}

}  // namespace hgb

extern "C" {

int hgb_batch_create(hgb_ctx *c, int num_systems, const int *sys_ptr, int n_total, int nnz, const int *pntr,
                     const int *indx, const float *vals, hgb_batch **out) {
    if (!out) return fail(HGB_ERR_ARG, "batch_create: null output");
    *out = nullptr;
    if (!c || num_systems <= 0 || n_total <= 0 || nnz < 0 || !sys_ptr || !pntr || !indx || !vals)
        return fail(HGB_ERR_ARG, "batch_create: bad arguments");
    DeviceGuard g(c->device);
    HGB_TRY(csr_check(c, n_total, n_total, nnz, pntr, indx));
    std::vector<int> sp(num_systems + 1);
    HGB_CUDA(cudaMemcpy(sp.data(), sys_ptr, sizeof(int) * (num_systems + 1), cudaMemcpyDeviceToHost));
    if (sp[0] != 0 || sp[num_systems] != n_total) return fail(HGB_ERR_ARG, "batch_create: sys_ptr must span [0, n_total]");
    hgb_batch *B = new hgb_batch();
    B->ctx = c;
    B->S = num_systems;
    B->n_total = n_total;
    B->nnz = nnz;
    B->sys_ptr = sys_ptr;
    B->pntr = pntr;
    B->indx = indx;
    B->vals = vals;
    B->sizes.resize(num_systems);
    for (int s = 0; s < num_systems; s++) {
        B->sizes[s] = sp[s + 1] - sp[s];
        if (B->sizes[s] <= 0) { delete B; return fail(HGB_ERR_ARG, "batch_create: empty system %d", s); }
    }
    int st = HGB_OK;
    batch_check_kernel<<<std::min(num_systems, c->num_sms * 8), 128, 0, c->stream>>>(num_systems, sys_ptr, pntr, indx, c->err);
    st = collect_dev_error(c);
    if (st) {
        delete B;
        return fail(st, "batch_create: a column falls outside its system's rows");
    }
    const size_t tickets = sizeof(int) * 2 * (1 + kNumShapes);
    if (cudaMalloc(&B->ticket, tickets) || cudaMemset(B->ticket, 0, tickets)) st = cuda_fail(cudaGetLastError(), "batch_create");
    if (!st) st = onchip_layout(B);
    if (!st) st = onchip_plan(B);
    if (!st) st = cudaFuncSetAttribute(batch_cg_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBatchSmem) ? HGB_ERR_CUDA : HGB_OK;
    if (!st) st = batch_plan(B, B->cfg);
    if (st) {
        hgb_batch_destroy(B);
        return st;
    }
    *out = B;
    return HGB_OK;
}

int hgb_batch_set_config(hgb_batch *B, const hgb_batch_config *cfg) {
    if (!B || !cfg) return fail(HGB_ERR_ARG, "batch_set_config: bad arguments");
    if (cfg->block_threads != 128 && cfg->block_threads != 256 && cfg->block_threads != 512)
        return fail(HGB_ERR_ARG, "batch: block_threads must be 128, 256 or 512");
    if (cfg->warp_max_n < 0) return fail(HGB_ERR_ARG, "batch: warp_max_n < 0");
    DeviceGuard g(B->ctx->device);
    return batch_plan(B, *cfg);
}

int hgb_batch_get_config(hgb_batch *B, hgb_batch_config *cfg) {
    if (!B || !cfg) return fail(HGB_ERR_ARG, "batch_get_config: bad arguments");
    *cfg = B->cfg;
    return HGB_OK;
}

int hgb_batch_cg_solve(hgb_batch *B, const double *b, double *x, double rtol, double inner_rtol, int max_inner,
                       int max_outer, int *iters, double *relres) {
    if (!B || !b || !x || !(rtol > 0) || !(inner_rtol > 0) || max_inner < 1 || max_outer < 0)
        return fail(HGB_ERR_ARG, "batch_cg_solve: bad arguments");
    hgb_ctx *c = B->ctx;
    DeviceGuard g(c->device);
    BatchArgs A = batch_args(B, b, x, rtol, inner_rtol, max_inner, max_outer, iters, relres);
    // the persistent launches are captured once into a graph and replayed while the
    // vectors and controls stay the same
    bool same = B->exec && same_args(A, B->captured);
    if (!same) {
        if (B->exec) {
            cudaGraphExecDestroy(B->exec);
            B->exec = nullptr;
        }
        CaptureStream cs(c);
        cudaGraph_t graph = nullptr;
        HGB_CUDA(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
        int st = batch_launch(B, A, c->stream);
        cudaError_t ce = cudaStreamEndCapture(c->stream, &graph);
        if (st) return st;
        if (ce != cudaSuccess) return cuda_fail(ce, "batch capture");
        cudaError_t ie = cudaGraphInstantiate(&B->exec, graph, 0);
        cudaGraphDestroy(graph);
        if (ie != cudaSuccess) return cuda_fail(ie, "batch graph instantiate");
        B->captured = A;
    }
    {
        CaptureStream cs(c);
        HGB_CUDA(cudaGraphLaunch(B->exec, c->stream));
    }
    return collect_dev_error(c);
}

int hgb_batch_autotune(hgb_batch *B, const double *b, double *x, double rtol, const char *cache_path,
                       hgb_batch_config *best) {
    if (!B || !b || !x) return fail(HGB_ERR_ARG, "batch_autotune: bad arguments");
    hgb_ctx *c = B->ctx;
    DeviceGuard g(c->device);
    if (B->nitems == 0) {   // every system is on chip: the configuration changes nothing
        if (best) *best = B->cfg;
        return HGB_OK;
    }
    // signature: number of systems and the streamed ones' size histogram in powers of two
    std::ostringstream sig;
    int hist[16] = {0};
    for (int s = 0; s < B->S; s++) {
        if (onchip_shape(B, s) >= 0) continue;
        int k = 0;
        while ((1 << (k + 1)) <= B->sizes[s] && k < 15) k++;
        hist[k]++;
    }
    sig << "streamed_of_S" << B->S << "_rt" << rtol;
    for (int k = 0; k < 16; k++) if (hist[k]) sig << "_" << k << ":" << hist[k];
    if (cache_path) {
        std::ifstream in(cache_path);
        std::string key;
        int bt, wm;
        while (in >> key >> bt >> wm) {
            if (key == sig.str()) {
                hgb_batch_config cfg{bt, wm};
                HGB_TRY(hgb_batch_set_config(B, &cfg));
                if (best) *best = cfg;
                return HGB_OK;
            }
        }
    }
    const int blocks[] = {128, 256, 512};
    const int warp_max[] = {0, 64, 128, 256, 512};
    double best_ms = 1e30;
    hgb_batch_config bcfg = B->cfg;
    cudaEvent_t e0, e1;
    HGB_CUDA(cudaEventCreate(&e0));
    HGB_CUDA(cudaEventCreate(&e1));
    int st = HGB_OK;
    for (int bt : blocks) {
        for (int wm : warp_max) {
            int cap = kBatchSmem / (int)sizeof(float) / (bt / 32) / 4;
            if (wm > cap) continue;
            hgb_batch_config cfg{bt, wm};
            if ((st = hgb_batch_set_config(B, &cfg))) break;
            float best_here = 1e30f;
            for (int rep = 0; rep < 2 && !st; rep++) {
                if (cudaMemsetAsync(x, 0, sizeof(double) * B->n_total, c->stream)) { st = HGB_ERR_CUDA; break; }
                cudaEventRecord(e0, c->stream);
                st = hgb_batch_cg_solve(B, b, x, rtol, 1e-4, 1000, 20, nullptr, nullptr);
                cudaEventRecord(e1, c->stream);
                cudaEventSynchronize(e1);
                float ms = 0;
                cudaEventElapsedTime(&ms, e0, e1);
                best_here = std::min(best_here, ms);
            }
            if (st) break;
            if (best_here < best_ms) {
                best_ms = best_here;
                bcfg = cfg;
            }
        }
        if (st) break;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (st) return st;
    HGB_TRY(hgb_batch_set_config(B, &bcfg));
    if (best) *best = bcfg;
    if (cache_path) {
        std::ofstream o(cache_path, std::ios::app);
        o << sig.str() << " " << bcfg.block_threads << " " << bcfg.warp_max_n << "\n";
    }
    return HGB_OK;
}

int hgb_batch_destroy(hgb_batch *B) {
    if (!B) return HGB_OK;
    DeviceGuard g(B->ctx->device);
    if (B->exec) cudaGraphExecDestroy(B->exec);
    cudaFree(B->item_sys);
    cudaFree(B->item_large);
    cudaFree(B->ticket);
    for (int k = 0; k < kNumShapes; k++) {
        cudaFree(B->on_items[k]);
        if (B->side[k]) cudaStreamDestroy(B->side[k]);
        if (B->join[k]) cudaEventDestroy(B->join[k]);
    }
    if (B->fork) cudaEventDestroy(B->fork);
    cudaFree(B->layout);
    delete B;
    return HGB_OK;
}

}  // extern "C"
