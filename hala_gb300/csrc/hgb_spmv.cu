// CSR SpMV and SpMM for sm_103a.  One warp takes 32 consecutive rows (a tile) at a time: it copies the
// tile's whole vals / indx range into its own shared-memory buffer with coalesced 16-byte cp.async (no
// handshake between warps), then every lane sums its row from shared memory, gathering x from
// global memory (L1 / L2).  The copies of the next kStages - 1 tiles and the row pointers of the tile
// after them are in flight while a tile is summed.  Tiles of more than CAP entries read their rows
// directly, the longest of them by the whole warp (spmv_wide_row).
//
// Two arithmetic modes, chosen per context (hgb_ctx_set_spmv_mode):
//  - exact: each row summed in column order with separately rounded multiply and add, the
//    arithmetic of the reference's sparse_gemv_array<T,'N'> (sparse/hala_sparse_utils.hpp:104-112),
//    so FP64 results are bit-identical to the reference CPU path.  That is two FP64 operations per
//    entry; sm_103's FP64 pipe is narrow (a warp-wide FP64 instruction holds an SMSP's FP64 unit
//    for 64 cycles), so the exact FP64 product is bound by the FP64 pipe, not by HBM.
//  - fused (the default): the same column order with one fused multiply-add per entry; a product
//    with alpha = 1 and beta = 0 skips the scaling.  Results differ from the reference's by the
//    rounding of the individual products (a few ulps of the row sum).
#include "hgb_internal.cuh"
#include "hgb_kernels.cuh"
#include "hgb_complex.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <string>
#include <vector>

namespace hgb {

static bool aligned16(const void *p) { return ((uintptr_t)p & 15u) == 0; }

constexpr int kWarpBlock = 256;   // 8 warps per CTA
constexpr int kStages = 2;        // tiles per warp in shared memory; three or four measured no gain
constexpr int kMmCols = 5;        // columns summed per pass over a tile at most
constexpr int kCapShort = 256, kCapLong = 384;   // entries of a staged tile (spmv_long_rows)
constexpr int kWideMin = 64;      // entries from which a row of a tile that is not staged may be summed by its warp

// CTAs per SM and x gathers in flight per lane and column, by vector type, columns per pass and
// tile size.  More CTAs leave less of the 256 KB for L1, which holds the gathered part of x and the
// rows that are read directly, and fewer registers for gathers; fewer CTAs leave HBM idle.  Measured
// (us; 128^3 7-point FP64 / FP32, graph Laplacians of 680k rows FP64 / FP32, 5 columns on 95x97x96 FP64 / FP32):
//   FP64, 256 entries: 3 CTAs of 8 gathers 45.2; of 4 gathers 47.8; 2 CTAs: 61.5; 4: 83.9 (spills); 6: 115.
//   FP32, 256 entries: 4 CTAs of 8 gathers 28.5 (BF16 values 24.7), of 7 31.8; 5 of 4 28.9 (30.8), of 7 44.8 (spills); 6 of 4
//   31.8 (31.6); 3 of 8 36.3.
//   384 entries (rows of 9, which 256 would send to the direct path): FP64 2 CTAs 30.8, 3: 35.2; FP32 3 CTAs of
//   4 gathers 16.9, of 8 20.2, 2 of 4 18.5.
//   columns: FP64 3 CTAs with one gather per column 66.6, with two and passes of 3 + 2 columns 78.7; FP32 3 CTAs
//   with two 28.8, 4 with three 39.0.  Three FP32 columns (and passes of six) run 4 CTAs of three gathers: a 5-point 369 x 408
//   grid, whose 4,705 tiles are two for some warps of 3 CTAs, 6.2 us and six columns 8.2, with 3 CTAs of four 8.2 and 10.3 (768 x
//   700: 12.4 and 18.6, both ways).  Four columns would gain there (8.2 -> 6.2), and lose on 768 x 700 (14.4 -> 16.4).
// One shape for all, 4 gathers, passes of 4 columns with one: 55.4 / 28.9 (25.0), 33.2 / 26.7, 108.6 / 43.1.
template <typename X, int NC, int CAP>
struct TileShape {
    static constexpr bool f64 = sizeof(X) == 8, wide = CAP > kCapShort;
    static constexpr int ctas = NC == 1 ? (f64 ? (wide ? 2 : 3) : (wide ? 3 : 4)) : (wide ? 2 : (NC == (f64 ? 2 : 3) ? 4 : 3));
    static constexpr int gathers = NC == 1 ? (wide ? 4 : 8) : (f64 ? (NC == 2 ? 2 : 1) : (NC == 2 ? 6 : (NC == 3 ? (wide ? 4 : 3) : 12 / NC)));
};

// acc += v * x in the mode's rounding
template <bool EXACT>
__device__ __forceinline__ double spmv_acc(double acc, double v, double x) {
    return EXACT ? add_rn(acc, mul_rn(v, x)) : __fma_rn(v, x, acc);
}
template <bool EXACT>
__device__ __forceinline__ float spmv_acc(float acc, float v, float x) {
    return EXACT ? add_rn(acc, mul_rn(v, x)) : __fmaf_rn(v, x, acc);
}
// How a product ends: y = acc (alpha 1, beta 0), alpha acc, or alpha acc + beta y.  Chosen on the host: an FP64
// comparison per row would hold the FP64 unit as long as a multiply-add.
enum SpmvEnd : int { END_PLAIN = 0, END_SCALED = 1, END_FULL = 2 };
template <typename X>
static SpmvEnd spmv_end(X alpha, X beta) {
    return beta != X(0) ? END_FULL : (alpha == X(1) ? END_PLAIN : END_SCALED);
}
// (EXACT: alpha acc, with beta y added, separately rounded; 1 times acc is acc)
template <bool EXACT, typename X>
__device__ __forceinline__ X spmv_out(int end, X alpha, X acc, X beta, const X *yp) {
    if (end == END_PLAIN) return acc;
    if (end == END_SCALED) return mul_rn(alpha, acc);
    if (EXACT) return add_rn(mul_rn(alpha, acc), mul_rn(beta, *yp));
    return spmv_acc<false>(mul_rn(beta, *yp), alpha, acc);
}

// A warp-uniform choice that stays a branch for FP64: a predicated-off FP64 instruction would hold the
// unit like any other.
__device__ __forceinline__ bool spmv_uniform(bool c, double) {
    int v = c;
    asm volatile("" : "+r"(v));
    return v;
}
__device__ __forceinline__ bool spmv_uniform(bool c, float) { return c; }

// The fused <x, y> (DOT): 0 none; 1 the grid reduction into *dot_out (the last CTA adds the
// parts); 2 each CTA's part to partials[blockIdx.x], summed by the consuming kernel (in one order
// in every CTA), which keeps the serial last-CTA step out of the product.
template <int DOT>
__device__ __forceinline__ void spmv_dot_epilogue(double d, double *partials, unsigned *counter, double *dot_out) {
    double dsum[1] = {d};
    if (DOT == 1) {
        grid_sum<1>(dsum, partials, counter, [&](double (&v)[1]) { *dot_out = v[0]; });
    } else if (DOT == 2) {
        block_sum<1>(dsum);
        if (threadIdx.x == 0) partials[blockIdx.x] = dsum[0];
    }
}

// A long row among short ones (in a tile that is not staged): alone in its lane it is bound by the latency of column
// then x, a few entries at a time.  spmv_wide_row takes 32 of its entries at once, with the next 32 and the
// columns after them in flight, and every lane adds them in column order (the products of EXACT are formed before,
// one per lane), so the sum is the single lane's bit for bit, at the FP64 unit's 64 cycles per entry.  The rows of a tile
// then come one after another: spmv_wide takes a row while it has a third (FP64) or an eighth (FP32) of the entries
// left, by the cost of an entry alone in its lane (about 190 cycles) and here (64; FP32 about 25).
// Such tiles wait for the end of the kernel, in a function of their own: inlined, or at their place among the
// staged tiles, they cost the staged FP64 product 45.8 -> 49 to 54 us.  Even so the test and the call cost the staged
// products registers (128^3 FP64 45.2 -> 45.6 us, FP32 28.5 -> 32.9), so they are compiled in (WIDE) for the matrices that
// may have such rows (spmv_may_be_wide).
// Rows of 7 with 0.2 % of 3000, FP64 / FP32: 100k rows 646 / 285 -> 302 / 109 us; of 300, 400k rows 115 / 79 -> 76 / 36.
// Four FP64 columns at 100k rows: 1637 -> 1174.  FP32 columns keep the lanes' own sums.
template <typename X>
__device__ __forceinline__ bool spmv_wide(int longest, int left) {
    return longest >= kWideMin && longest >= left / (sizeof(X) == 8 ? 3 : 8);
}
template <typename V, bool EXACT>
__device__ __forceinline__ typename Val<V>::X spmv_wide_row(const V *vp, const int *ip, unsigned len, const typename Val<V>::X *x) {
    using X = typename Val<V>::X;
    const unsigned lane = threadIdx.x & 31;
    auto at = [&](unsigned j) { return min(j + lane, len - 1); };   // past the end: the last entry, not summed
    X acc = X(0), v = Val<V>::get(__ldg(vp + at(0))), xv = __ldg(x + __ldg(ip + at(0)));
    int col = __ldg(ip + at(32));
    for (unsigned j = 0; j < len; j += 32) {
        const X v1 = Val<V>::get(__ldg(vp + at(j + 32))), x1 = __ldg(x + col);
        col = __ldg(ip + at(j + 64));
        if (EXACT) xv = mul_rn(v, xv);
        const int few = (int)min(len - j, 32u);
#pragma unroll 4
        for (int q = 0; q < few; q++) {
            const X xq = __shfl_sync(0xffffffffu, xv, q);
            acc = EXACT ? add_rn(acc, xq) : spmv_acc<false>(acc, __shfl_sync(0xffffffffu, v, q), xq);
        }
        v = v1;
        xv = x1;
    }
    return acc;
}

template <typename V, int CAP, bool DOT, bool EXACT>
__device__ __noinline__ DotAcc<typename Val<V>::X>
spmv_wide_tiles(int tb, int te, int n_rows, const int *__restrict__ pntr, const int *__restrict__ indx,
                const V *__restrict__ vals, int nrhs, int end_mode, typename Val<V>::X alpha,
                const typename Val<V>::X *__restrict__ x, long ldx, typename Val<V>::X beta,
                typename Val<V>::X *__restrict__ y, long ldy, DotAcc<typename Val<V>::X> dacc) {
    using X = typename Val<V>::X;
    const int lane = threadIdx.x & 31;
    for (int k = tb; k < te; k++) {
        const int row = k * 32 + lane;
        const int ps = __ldg(pntr + min(row, n_rows)), pe = __ldg(pntr + min(row, n_rows - 1) + 1);
        const int total = __shfl_sync(0xffffffffu, pe, 31) - __shfl_sync(0xffffffffu, ps, 0);
        if (total <= CAP || !spmv_wide<X>(__reduce_max_sync(0xffffffffu, pe - ps), total)) continue;
        for (int m = 0; m < nrhs; m++) {
            const X *xc = x + (long)m * ldx;
            X acc = X(0);
            int n = pe - ps, longest = __reduce_max_sync(0xffffffffu, n), left = total;
            while (spmv_wide<X>(longest, left)) {
                const int r = __ffs(__ballot_sync(0xffffffffu, n == longest)) - 1;
                const int base = __shfl_sync(0xffffffffu, ps, r);
                const X sum = spmv_wide_row<V, EXACT>(vals + base, indx + base, (unsigned)longest, xc);
                if (lane == r) {
                    acc = sum;
                    n = 0;
                }
                left -= longest;
                longest = __reduce_max_sync(0xffffffffu, n);
            }
            for (int j0 = 0; j0 < n; j0 += 4) {
                X xv[4], vv[4];
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (j0 + q < n) {
                        vv[q] = Val<V>::get(__ldg(vals + ps + j0 + q));
                        xv[q] = __ldg(xc + __ldg(indx + ps + j0 + q));
                    }
#pragma unroll
                for (int q = 0; q < 4; q++)
                    if (j0 + q < n) acc = spmv_acc<EXACT>(acc, vv[q], xv[q]);
            }
            if (row < n_rows) {
                X *yp = y + (long)m * ldy + row;
                const X out = spmv_out<EXACT>(end_mode, alpha, acc, beta, yp);
                *yp = out;
                if (DOT) dacc.add(__ldg(x + row), out);
            }
        }
    }
    return dacc;
}

// Y = alpha * A X + beta * Y for nrhs column-major columns (x column c at x + c * ldx), cols <= NC of them per
// pass over a staged tile (the matrix is read once); optionally <x, y> (one column, square A; DOT as
// spmv_dot_epilogue).  Every column is summed in column order in the mode's rounding, so each column
// equals the single-column product bit for bit.
template <typename V, int NC, int CAP, int DOT, bool EXACT, bool WIDE>
__global__ void __launch_bounds__(kWarpBlock, TileShape<typename Val<V>::X, NC, CAP>::ctas)
spmv_tile_kernel(int n_rows, const int *__restrict__ pntr, const int *__restrict__ indx, const V *__restrict__ vals,
                 int nrhs, int cols, int end_mode, typename Val<V>::X alpha, const typename Val<V>::X *__restrict__ x,
                 long ldx, typename Val<V>::X beta, typename Val<V>::X *__restrict__ y, long ldy, double *partials,
                 unsigned *counter, double *dot_out, const int *skip) {
    using X = typename Val<V>::X;
    constexpr int EV = 16 / (int)sizeof(V);   // values per 16-byte unit
    constexpr int SV = CAP + 2 * EV, SI = CAP + 8, ST = kStages;
    static_assert(CAP % 8 == 0, "every buffer starts on a 16-byte boundary");
    if (skip && *skip) return;
    extern __shared__ __align__(16) unsigned char spmv_smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    V *const s_vals = (V *)spmv_smem + wib * ST * SV;
    int *const s_idx = (int *)((V *)spmv_smem + (kWarpBlock / 32) * ST * SV) + wib * ST * SI;
    const int nnz = __ldg(pntr + n_rows);
    const int ntiles = (int)(((long)n_rows + 31) / 32);
    const int nwarps = gridDim.x * (kWarpBlock / 32);
    const int per = (ntiles + nwarps - 1) / nwarps;
    const int tb = (blockIdx.x * (kWarpBlock / 32) + wib) * per;
    const int te = min(ntiles, tb + per);
    int wide = te;    // tb once a tile of this warp is left for the end (spmv_wide_tiles)
    DotAcc<X> dacc;   // fused <x, y> (per-thread partial)

    // lane's row pointers of tile k (loads only; nothing waits on them yet)
    auto load_ptrs = [&](int k, int &ps, int &pe) {
        // unsigned: the row behind the last tile may be 2^31 (a clamp to the last tile: 128^3 FP32 28.4 -> 32.0 us)
        const unsigned row = (unsigned)min(k, ntiles) * 32u + lane, rows = n_rows;
        ps = __ldg(pntr + min(row, rows));
        pe = __ldg(pntr + min(row + 1, rows));
    };
    // tile k's copy into buffer buf when it fits (one commit per call)
    auto stage = [&](int k, int ps, int pe, int buf) {
        const int base = __shfl_sync(0xffffffffu, ps, 0), end = __shfl_sync(0xffffffffu, pe, 31);
        if (k < te && end - base <= CAP) {
            V *sv = s_vals + buf * SV;
            int *si = s_idx + buf * SI;
            const int av = base & ~(EV - 1), ai = base & ~3;
            for (int g = av + lane * EV; g < end; g += 32 * EV) {
                if (g + EV <= nnz) cp_async16(sv + (g - av), vals + g);
                else
                    for (int q = 0; q < EV && g + q < end; q++) sv[g - av + q] = vals[g + q];
            }
            for (int g = ai + lane * 4; g < end; g += 32 * 4) {
                if (g + 4 <= nnz) cp_async16(si + (g - ai), indx + g);
                else
                    for (int q = 0; q < 4 && g + q < end; q++) si[g - ai + q] = indx[g + q];
            }
        }
        cp_async_commit();
    };

    if (tb < te) {
        int ps[ST + 1], pe[ST + 1];   // row pointers of tiles k ... k + ST
#pragma unroll
        for (int s = 0; s < ST; s++) load_ptrs(tb + s, ps[s], pe[s]);
#pragma unroll
        for (int s = 0; s < ST - 1; s++) stage(tb + s, ps[s], pe[s], s);
        int buf = 0, fill = ST - 1;
        for (int k = tb; k < te; k++) {
            stage(k + ST - 1, ps[ST - 1], pe[ST - 1], fill);
            load_ptrs(k + ST, ps[ST], pe[ST]);
            cp_async_wait<ST - 1>();   // tile k has landed
            __syncwarp();
            int row = k * 32 + lane;
            const int first = __shfl_sync(0xffffffffu, ps[0], 0), end = __shfl_sync(0xffffffffu, pe[0], 31);
            int cnt = pe[0] - ps[0];
            int most = __reduce_max_sync(0xffffffffu, cnt);
            if (WIDE && __builtin_expect(end - first > CAP && spmv_wide<X>(most, end - first), 0)) {   // no entries, no row to write
                wide = tb;
                row = n_rows;
                cnt = most = 0;
            }
            for (int c0 = 0; c0 < (NC == 1 ? 1 : nrhs); c0 += cols) {
                const int nc = NC == 1 ? 1 : min(cols, nrhs - c0);
                const X *xc = x + (long)c0 * ldx;
                X acc[NC];
#pragma unroll
                for (int m = 0; m < NC; m++) acc[m] = X(0);
                // the row's entries, GW at a time, from vp / ip (its first entry in the buffer or in memory), in step
                // across the warp; not for several columns of a direct tile, whose long rows leave few lanes active
                auto sum = [&](const V *vp, const int *ip, auto staged) {
                    constexpr bool in_step = decltype(staged)::value || NC == 1;
                    // FP64 values stay in shared memory until they are multiplied: registers for gathers
                    constexpr bool late = decltype(staged)::value && sizeof(X) == 8;
                    constexpr int GW = TileShape<X, NC, CAP>::gathers;
                    const int upto = in_step ? most : cnt;
                    for (int j0 = 0; j0 < upto; j0 += GW) {
                        X xv[GW][NC], vv[GW];
#pragma unroll
                        for (int q = 0; q < GW; q++)
                            if (j0 + q < cnt) {
                                V v;
                                int col;
                                if constexpr (decltype(staged)::value) {
                                    v = vp[j0 + q];
                                    col = ip[j0 + q];
                                } else {
                                    v = __ldg(vp + j0 + q);
                                    col = __ldg(ip + j0 + q);
                                }
                                if (!late) vv[q] = Val<V>::get(v);
                                const X *xp = xc + col;
#pragma unroll
                                for (int m = 0; m < NC; m++)
                                    if (m < nc) xv[q][m] = __ldg(xp + (long)m * ldx);
                            }
#pragma unroll
                        for (int q = 0; q < GW; q++)
                            if (!in_step || spmv_uniform(j0 + q < most, X(0))) {
#pragma unroll
                                for (int m = 0; m < NC; m++)
                                    if (NC == 1 || !in_step || spmv_uniform(m < nc, X(0)))
                                        if (j0 + q < cnt) acc[m] = spmv_acc<EXACT>(acc[m], late ? Val<V>::get(vp[j0 + q]) : vv[q], xv[q][m]);
                            }
                    }
                };
                if (end - first <= CAP)
                    sum(s_vals + buf * SV + (ps[0] - (first & ~(EV - 1))), s_idx + buf * SI + (ps[0] - (first & ~3)),
                        std::true_type());
                else
                    sum(vals + ps[0], indx + ps[0], std::false_type());
                if (row < n_rows) {
#pragma unroll
                    for (int m = 0; m < NC; m++)
                        if (m < nc) {
                            X *yp = y + (long)(c0 + m) * ldy + row;
                            const X out = spmv_out<EXACT>(end_mode, alpha, acc[m], beta, yp);
                            *yp = out;
                            if (DOT) dacc.add(__ldg(x + row), out);
                        }
                }
            }
            __syncwarp();   // the buffer is refilled next
            fill = buf;
            buf = buf + 1 == ST ? 0 : buf + 1;
#pragma unroll
            for (int s = 0; s < ST; s++) {
                ps[s] = ps[s + 1];
                pe[s] = pe[s + 1];
            }
        }
    }
    cp_async_wait<0>();
    if (WIDE && wide < te)   // the tiles that were left out
        dacc = spmv_wide_tiles<V, CAP, DOT != 0, EXACT>(wide, te, n_rows, pntr, indx, vals, NC == 1 ? 1 : nrhs, end_mode, alpha, x, ldx,
                                                        beta, y, ldy, dacc);
    if (DOT) spmv_dot_epilogue<DOT>(dacc.get(), partials, counter, dot_out);
}
template <typename V, int CAP>
constexpr size_t spmv_smem_bytes() {
    return (size_t)(kWarpBlock / 32) * kStages * ((CAP + 2 * (16 / sizeof(V))) * sizeof(V) + (CAP + 8) * sizeof(int));
}

// Arrays that are not 16-byte aligned cannot be staged with cp.async: one row per thread,
// grid-stride, the row's vals/indx and x gathers (8 at a time) straight from global memory
// through L1.  Same arithmetic as spmv_tile_kernel.
template <typename V, int DOT, bool EXACT>
__global__ void __launch_bounds__(256)
spmv_direct_kernel(int n_rows, const int *__restrict__ pntr, const int *__restrict__ indx,
                   const V *__restrict__ vals, int end_mode, typename Val<V>::X alpha,
                   const typename Val<V>::X *__restrict__ x, typename Val<V>::X beta, typename Val<V>::X *__restrict__ y,
                   double *partials, unsigned *counter, double *dot_out, const int *skip) {
    using X = typename Val<V>::X;
    if (skip && *skip) return;
    DotAcc<X> dacc;   // fused <x, y> (per-thread partial)
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += gridDim.x * blockDim.x) {
        const int ps = __ldg(pntr + r), pe = __ldg(pntr + r + 1);
        X acc = X(0);
        for (int j0 = ps; j0 < pe; j0 += 8) {
            X xv[8], vv[8];
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (j0 + k < pe) {
                    vv[k] = Val<V>::get(__ldg(vals + j0 + k));
                    xv[k] = __ldg(x + __ldg(indx + j0 + k));
                }
#pragma unroll
            for (int k = 0; k < 8; k++)
                if (j0 + k < pe) acc = spmv_acc<EXACT>(acc, vv[k], xv[k]);
        }
        const X out = spmv_out<EXACT>(end_mode, alpha, acc, beta, y + r);
        y[r] = out;
        if (DOT) dacc.add(__ldg(x + r), out);
    }
    if (DOT) spmv_dot_epilogue<DOT>(dacc.get(), partials, counter, dot_out);
}


// transposed product by atomic scatter (stateless path): y[c] += (alpha * x[i]) * v_ic
template <typename V>
__global__ void spmv_t_atomic_kernel(int n_rows, const int *__restrict__ pntr, const int *__restrict__ indx,
                                     const V *__restrict__ vals, typename Val<V>::X alpha,
                                     const typename Val<V>::X *__restrict__ x, typename Val<V>::X *y) {
    using X = typename Val<V>::X;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_rows; i += gridDim.x * blockDim.x) {
        X ax = mul_rn(alpha, x[i]);
        for (int p = __ldg(pntr + i); p < __ldg(pntr + i + 1); p++)
            atomicAdd(y + __ldg(indx + p), mul_rn(ax, Val<V>::get(__ldg(vals + p))));
    }
}

template <typename X>
__global__ void scale_or_zero_kernel(long n, X beta, X *y) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        y[i] = (beta == X(0)) ? X(0) : mul_rn(beta, y[i]);
}

// transposed product through the cached transpose: one thread per column, entries in ascending
// original row, which is the accumulation order of sparse_gemv_array<'T'> (utils:113-118).
// FUSE_DOT additionally reduces <x', y> with x' = the vector y is paired with (dot_x, indexed by
// column), for the CG on the transposed operator.
// Bound by the FP64 unit (separately rounded operations, the oracle's) and the latency of the chain
// pointers -> map / rows -> values / x: the scaling by alpha, and the comparisons with alpha and beta, are
// left out where end_mode says that they do nothing; three entries' loads are in flight per lane, in 32 registers, so
// that an SM holds 64 warps (512^2 5-point FP64: 12.4 -> 10.3 us; 97x96^2 7-point FP32: 17.0 -> 14.2; five or eight
// entries in flight in fewer warps: 10.3 to 14.4 and 14.4 to 16.4).  The loop is warp-uniform (spmv_uniform).
template <typename V, bool FUSE_DOT>
__global__ void __launch_bounds__(256, 8)
spmv_t_cached_kernel(int n_cols, const int *__restrict__ pntrT, const int *__restrict__ rowT,
                     const int *__restrict__ mapT, const V *__restrict__ vals, int end_mode,
                     typename Val<V>::X alpha, const typename Val<V>::X *__restrict__ x,
                     typename Val<V>::X beta, typename Val<V>::X *__restrict__ y,
                     const typename Val<V>::X *__restrict__ dot_x, double *partials,
                     unsigned *counter, double *dot_out, const int *skip) {
    using X = typename Val<V>::X;
    constexpr int G = 3;
    if (skip && *skip) return;
    DotAcc<X> dacc;   // fused <x, y> (per-thread partial)
    for (int cb = blockIdx.x * blockDim.x + (threadIdx.x & ~31); cb < n_cols; cb += gridDim.x * blockDim.x) {
        const int c = cb + (threadIdx.x & 31);
        const int ps = __ldg(pntrT + min(c, n_cols)), cnt = __ldg(pntrT + min(c + 1, n_cols)) - ps;
        const int most = __reduce_max_sync(0xffffffffu, cnt);
        X acc = X(0);
        if (end_mode == END_FULL && c < n_cols) acc = mul_rn(beta, y[c]);
        for (int j0 = 0; j0 < most; j0 += G) {
            int at[G];
            X xv[G], vv[G];
#pragma unroll
            for (int q = 0; q < G; q++)
                if (j0 + q < cnt) {
                    at[q] = __ldg(mapT + ps + j0 + q);
                    xv[q] = __ldg(x + __ldg(rowT + ps + j0 + q));
                }
#pragma unroll
            for (int q = 0; q < G; q++)
                if (j0 + q < cnt) vv[q] = Val<V>::get(__ldg(vals + at[q]));
            if (end_mode != END_PLAIN) {
#pragma unroll
                for (int q = 0; q < G; q++)
                    if (spmv_uniform(j0 + q < most, X(0)))
                        if (j0 + q < cnt) xv[q] = mul_rn(alpha, xv[q]);
            }
#pragma unroll
            for (int q = 0; q < G; q++)
                if (spmv_uniform(j0 + q < most, X(0)))
                    if (j0 + q < cnt) acc = add_rn(acc, mul_rn(xv[q], vv[q]));
        }
        if (c < n_cols) {
            y[c] = acc;
            if (FUSE_DOT) dacc.add(dot_x[c], acc);
        }
    }
    if (FUSE_DOT) {
        double dsum[1] = {dacc.get()};
        grid_sum<1>(dsum, partials, counter, [&](double (&v)[1]) { *dot_out = v[0]; });
    }
}

// ------------------------------------------------------------- CSR validation ----------
__global__ void csr_check_kernel(int n_rows, int n_cols, int nnz, const int *__restrict__ pntr,
                                 const int *__restrict__ indx, int *err, int *longest) {
    __shared__ int most;
    if (threadIdx.x == 0) most = 0;
    __syncthreads();
    int len = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_rows; i += gridDim.x * blockDim.x) {
        int a = pntr[i], b = pntr[i + 1];
        if (a < 0 || b < a || b > nnz) { atomicOr(err, DEV_ERR_CSR); continue; }
        len = max(len, b - a);
        int prev = -1;
        for (int p = a; p < b; p++) {
            int c = indx[p];
            if (c <= prev || c >= n_cols) { atomicOr(err, DEV_ERR_CSR); break; }
            prev = c;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && (pntr[0] != 0 || pntr[n_rows] != nnz)) atomicOr(err, DEV_ERR_CSR);
    if (!longest) return;
    atomicMax(&most, len);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(longest, most);
}

// ------------------------------------------------------------- scan / transpose -------
__global__ void scan_blocks_kernel(const int *__restrict__ in, int *__restrict__ out, int n, int *block_tot) {
    // exclusive scan of 1024-element chunks (one per CTA of 1024 threads)
    __shared__ int sh[1024];
    int i = blockIdx.x * 1024 + threadIdx.x;
    int v = (i < n) ? in[i] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
        int t = (threadIdx.x >= o) ? sh[threadIdx.x - o] : 0;
        __syncthreads();
        sh[threadIdx.x] += t;
        __syncthreads();
    }
    if (i < n) out[i] = sh[threadIdx.x] - v;
    if (threadIdx.x == 1023) block_tot[blockIdx.x] = sh[1023];
}

__global__ void __launch_bounds__(1024) scan_tot_kernel(int *tot, int nb, int *grand) {
    // exclusive scan of the block totals by one CTA, 1024 at a time
    __shared__ int wsum[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int run = 0;
    for (int b0 = 0; b0 < nb; b0 += 1024) {
        const int b = b0 + threadIdx.x, t = b < nb ? tot[b] : 0;
        int v = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += u;
        }
        if (lane == 31) wsum[w] = v;
        __syncthreads();
        int before = 0, all = 0;
        for (int k = 0; k < 32; k++) {
            if (k < w) before += wsum[k];
            all += wsum[k];
        }
        if (b < nb) tot[b] = run + before + v - t;
        run += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *grand = run;
}

__global__ void scan_add_kernel(int *out, int n, const int *tot) {
    int i = blockIdx.x * 1024 + threadIdx.x;
    if (i < n) out[i] += tot[blockIdx.x];
}

__global__ void count_cols_kernel(int nnz, const int *__restrict__ indx, int *cnt) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < nnz; p += gridDim.x * blockDim.x)
        atomicAdd(cnt + indx[p], 1);
}

__global__ void fill_transpose_kernel(int n_rows, const int *__restrict__ pntr, const int *__restrict__ indx,
                                      const int *__restrict__ pntrT, int *cursor, int *rowT, int *mapT) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_rows; i += gridDim.x * blockDim.x)
        for (int p = pntr[i]; p < pntr[i + 1]; p++) {
            int c = indx[p];
            int slot = pntrT[c] + atomicAdd(cursor + c, 1);
            rowT[slot] = i;
            mapT[slot] = p;
        }
}

__global__ void sort_segments_kernel(int n, const int *__restrict__ ptr, int *key, int *val) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        int a = ptr[r], b = ptr[r + 1];
        for (int i = a + 1; i < b; i++) {   // insertion sort: segments are short
            int k = key[i], v = val[i], j = i - 1;
            while (j >= a && key[j] > k) {
                key[j + 1] = key[j];
                val[j + 1] = val[j];
                j--;
            }
            key[j + 1] = k;
            val[j + 1] = v;
        }
    }
}

int exclusive_scan(hgb_ctx *c, const int *in, int *out, int n, int *total_dev, int *scratch) {
    // scratch: at least ceil(n/1024) ints
    int nb = (n + 1023) / 1024;
    if (nb == 0) return HGB_OK;
    scan_blocks_kernel<<<nb, 1024, 0, c->stream>>>(in, out, n, scratch);
    scan_tot_kernel<<<1, 1024, 0, c->stream>>>(scratch, nb, total_dev);
    scan_add_kernel<<<nb, 1024, 0, c->stream>>>(out, n, scratch);
    return launch_check("exclusive_scan");
}

int csr_check(hgb_ctx *c, int n_rows, int n_cols, int nnz, const int *pntr, const int *indx, int *longest) {
    if (longest) *longest = 0;
    if (n_rows <= 0) return HGB_OK;
    int *most = longest ? (int *)c->result : nullptr;
    if (most) HGB_CUDA(cudaMemsetAsync(most, 0, sizeof(int), c->stream));
    csr_check_kernel<<<std::min((n_rows + 255) / 256, c->num_sms * 8), 256, 0, c->stream>>>(n_rows, n_cols, nnz,
                                                                                           pntr, indx, c->err, most);
    HGB_TRY(launch_check("csr_check_kernel"));
    if (most) HGB_CUDA(cudaMemcpyAsync(c->host_result, most, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    HGB_TRY(collect_dev_error(c));
    if (longest) *longest = *(const int *)c->host_result;
    return HGB_OK;
}

int build_transpose(hgb_ctx *c, int n_rows, int n_cols, int nnz, const int *pntr, const int *indx,
                    Transpose &T) {
    T.n = n_cols;
    size_t nb = (size_t)(n_cols + 1 + 1023) / 1024 + 1;
    HGB_CUDA(cudaMalloc(&T.pntr, sizeof(int) * (size_t)(n_cols + 1)));
    HGB_CUDA(cudaMalloc(&T.row, sizeof(int) * (size_t)std::max(nnz, 1)));
    HGB_CUDA(cudaMalloc(&T.map, sizeof(int) * (size_t)std::max(nnz, 1)));
    int *cnt = nullptr, *scratch = nullptr;
    HGB_CUDA(cudaMalloc(&cnt, sizeof(int) * (size_t)(n_cols + 1)));
    HGB_CUDA(cudaMalloc(&scratch, sizeof(int) * (nb + 1)));
    int st = HGB_OK;
    do {
        if (cudaMemsetAsync(cnt, 0, sizeof(int) * (size_t)(n_cols + 1), c->stream) != cudaSuccess) { st = HGB_ERR_CUDA; break; }
        int g = std::max(1, std::min((nnz + 255) / 256, c->num_sms * 8));
        count_cols_kernel<<<g, 256, 0, c->stream>>>(nnz, indx, cnt);
        st = exclusive_scan(c, cnt, T.pntr, n_cols + 1, scratch + nb, scratch);
        if (st) break;
        if (cudaMemsetAsync(cnt, 0, sizeof(int) * (size_t)(n_cols + 1), c->stream) != cudaSuccess) { st = HGB_ERR_CUDA; break; }
        int gr = std::max(1, std::min((n_rows + 255) / 256, c->num_sms * 8));
        fill_transpose_kernel<<<gr, 256, 0, c->stream>>>(n_rows, pntr, indx, T.pntr, cnt, T.row, T.map);
        int gc = std::max(1, std::min((n_cols + 255) / 256, c->num_sms * 8));
        sort_segments_kernel<<<gc, 256, 0, c->stream>>>(n_cols, T.pntr, T.row, T.map);
        st = launch_check("build_transpose");
        if (!st && cudaStreamSynchronize(c->stream) != cudaSuccess) st = cuda_fail(cudaGetLastError(), "build_transpose");
    } while (0);
    cudaFree(cnt);
    cudaFree(scratch);
    return st;
}

void Transpose::release() {
    cudaFree(pntr);
    cudaFree(row);
    cudaFree(map);
    pntr = row = map = nullptr;
}

// Tiles of rows of 7 entries fit kCapShort; where rows average more than 7.5, kCapLong keeps those up to 12
// staged.  (Tiles cut into chunks, or longer buffers, were slower than the direct reads for longer rows: the lanes
// whose row is not in the chunk idle.)
static bool spmv_long_rows(int n_rows, long nnz) { return 2 * nnz > 15L * n_rows; }

// The staged kernel's launch: a persistent grid of the resident CTAs of every SM (occupancy queried once per
// kernel and device).
template <typename V, int NC, int CAP, int DOT, bool EXACT, bool WIDE>
static int spmv_tile_launch(hgb_ctx *c, int n_rows, const int *pntr, const int *indx, const V *vals, int nrhs, int cols,
                            typename Val<V>::X alpha, const typename Val<V>::X *x, long ldx, typename Val<V>::X beta,
                            typename Val<V>::X *y, long ldy, double *partials, unsigned *counter, double *dot_out,
                            const int *skip, int *nparts) {
    constexpr size_t smem = spmv_smem_bytes<V, CAP>();
    constexpr int most = TileShape<typename Val<V>::X, NC, CAP>::ctas;
    auto kernel = spmv_tile_kernel<V, NC, CAP, DOT, EXACT, WIDE>;
    static std::atomic<int> occ_dev[64];
    if (c->device < 0 || c->device >= 64) return fail(HGB_ERR_UNSUPPORTED, "spmv: device ordinal %d", c->device);
    int occ = occ_dev[c->device].load();
    if (!occ) {
        HGB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        HGB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                      std::min(100, (int)(most * (smem + 1024) * 100 / (228 * 1024)) + 1)));
        HGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kernel, kWarpBlock, smem));
        occ = std::min(std::max(occ, 1), most);
        occ_dev[c->device] = occ;
    }
    const long tiles = ((long)n_rows + 31) / 32;
    const int g = (int)std::max<long>(1, std::min<long>((tiles + 7) / 8, std::min(c->num_sms * occ, kMaxReduceBlocks)));
    if (nparts) *nparts = g;
    kernel<<<g, kWarpBlock, smem, c->stream>>>(n_rows, pntr, indx, vals, nrhs, cols, spmv_end(alpha, beta), alpha, x, ldx, beta,
                                               y, ldy, partials, counter, dot_out, skip);
    return launch_check("spmv_tile_kernel");
}

// Whether a row may be long enough to be summed by its warp (spmv_wide).  The pattern check of a matrix handle knows the
// longest row; the entries without a handle do not: in FP64 they take the test along (128^3 45.2 -> 45.6 us; without it
// 100k rows of 7 with 0.2 % of 3000 take 646 us instead of 302), in FP32 and BF16, where it costs more (28.5 -> 32.9 and
// 24.7 -> 32.9) and the rows' own lanes lose less (285 instead of 109), they do not.
template <typename V>
static bool spmv_may_be_wide(CsrSize size) { return size.longest < 0 ? sizeof(V) == 8 : size.longest >= kWideMin; }

template <typename V, int DOT, bool EXACT>
static int spmv_n_launch_mode(hgb_ctx *c, int n_rows, CsrSize size, const int *pntr, const int *indx, const V *vals,
                              typename Val<V>::X alpha, const typename Val<V>::X *x, typename Val<V>::X beta,
                              typename Val<V>::X *y, double *dot_out, const int *skip, int *nparts) {
    // DOT 2: the per-CTA parts of <x, y> stay in the context's parts slots (their count to *nparts)
    double *partials = DOT == 2 ? c->partials + kSpmvPartsOffset : (DOT == 1 ? c->partials : nullptr);
    unsigned *counter = DOT == 1 ? c->counter : nullptr;
    if (aligned16(vals) && aligned16(indx)) {
#define HGB_SPMV(CAP, WIDE)                                                                                                    \
    spmv_tile_launch<V, 1, CAP, DOT, EXACT, WIDE>(c, n_rows, pntr, indx, vals, 1, 1, alpha, x, 0, beta, y, 0, partials, counter, \
                                                  dot_out, skip, nparts)
        if (spmv_long_rows(n_rows, size.nnz)) return spmv_may_be_wide<V>(size) ? HGB_SPMV(kCapLong, true) : HGB_SPMV(kCapLong, false);
        return spmv_may_be_wide<V>(size) ? HGB_SPMV(kCapShort, true) : HGB_SPMV(kCapShort, false);
#undef HGB_SPMV
    }
    const int g = std::min((n_rows + 255) / 256, std::min(c->num_sms * 8, kMaxReduceBlocks));
    if (nparts) *nparts = g;
    spmv_direct_kernel<V, DOT, EXACT><<<g, 256, 0, c->stream>>>(n_rows, pntr, indx, vals, spmv_end(alpha, beta), alpha, x, beta, y,
                                                                   partials, counter, dot_out, skip);
    return launch_check("spmv_direct_kernel");
}

template <typename V>
int spmv_n_launch(hgb_ctx *c, int n_rows, CsrSize size, const int *pntr, const int *indx, const V *vals,
                  typename Val<V>::X alpha, const typename Val<V>::X *x, typename Val<V>::X beta,
                  typename Val<V>::X *y, double *dot_out, const int *skip, int *nparts) {
    if (nparts) *nparts = 0;
    if (n_rows <= 0) return HGB_OK;
    const bool exact = c->spmv_mode == HGB_SPMV_EXACT;
    if (nparts)
        return exact ? spmv_n_launch_mode<V, 2, true>(c, n_rows, size, pntr, indx, vals, alpha, x, beta, y, nullptr, skip, nparts)
                     : spmv_n_launch_mode<V, 2, false>(c, n_rows, size, pntr, indx, vals, alpha, x, beta, y, nullptr, skip, nparts);
    if (dot_out)
        return exact ? spmv_n_launch_mode<V, 1, true>(c, n_rows, size, pntr, indx, vals, alpha, x, beta, y, dot_out, skip, nullptr)
                     : spmv_n_launch_mode<V, 1, false>(c, n_rows, size, pntr, indx, vals, alpha, x, beta, y, dot_out, skip, nullptr);
    return exact ? spmv_n_launch_mode<V, 0, true>(c, n_rows, size, pntr, indx, vals, alpha, x, beta, y, nullptr, skip, nullptr)
                 : spmv_n_launch_mode<V, 0, false>(c, n_rows, size, pntr, indx, vals, alpha, x, beta, y, nullptr, skip, nullptr);
}

template <typename V>
int spmm_n_launch(hgb_ctx *c, int n_rows, CsrSize size, const int *pntr, const int *indx, const V *vals, int nrhs,
                  typename Val<V>::X alpha, const typename Val<V>::X *x, long ldx, typename Val<V>::X beta,
                  typename Val<V>::X *y, long ldy) {
    if (n_rows <= 0 || nrhs <= 0) return HGB_OK;
    if (!aligned16(vals) || !aligned16(indx)) {   // no staging: the single-column products
        for (int k = 0; k < nrhs; k++)
            HGB_TRY(spmv_n_launch<V>(c, n_rows, size, pntr, indx, vals, alpha, x + (long)k * ldx, beta, y + (long)k * ldy,
                                     nullptr));
        return HGB_OK;
    }
    const bool exact = c->spmv_mode == HGB_SPMV_EXACT;
    const int passes = (nrhs + kMmCols - 1) / kMmCols, cols = (nrhs + passes - 1) / passes;   // columns split evenly
    // FP32 columns keep the lanes' own sums (spmv_wide_row)
#define HGB_SPMM3(NC, CAP, EXACT, WIDE)                                                                             \
    spmv_tile_launch<V, NC, CAP, 0, EXACT, WIDE>(c, n_rows, pntr, indx, vals, nrhs, cols, alpha, x, ldx, beta, y, ldy, nullptr, \
                                           nullptr, nullptr, nullptr, nullptr)
#define HGB_SPMM2(NC, CAP, EXACT)                                                                                   \
    (spmv_may_be_wide<V>(size) ? HGB_SPMM3(NC, CAP, EXACT, (NC == 1 || sizeof(V) == 8)) : HGB_SPMM3(NC, CAP, EXACT, false))
#define HGB_SPMM(NC)                                                                               \
    (spmv_long_rows(n_rows, size.nnz) ? (exact ? HGB_SPMM2(NC, kCapLong, true) : HGB_SPMM2(NC, kCapLong, false)) \
                                 : (exact ? HGB_SPMM2(NC, kCapShort, true) : HGB_SPMM2(NC, kCapShort, false)))
    switch (cols) {
        case 1: return HGB_SPMM(1);
        case 2: return HGB_SPMM(2);
        case 3: return HGB_SPMM(3);
        case 4: return HGB_SPMM(4);
        default: return HGB_SPMM(kMmCols);
    }
#undef HGB_SPMM3
#undef HGB_SPMM2
#undef HGB_SPMM
}

template int spmv_n_launch<double>(hgb_ctx *, int, CsrSize, const int *, const int *, const double *, double,
                                   const double *, double, double *, double *, const int *, int *);
template int spmv_n_launch<float>(hgb_ctx *, int, CsrSize, const int *, const int *, const float *, float,
                                  const float *, float, float *, double *, const int *, int *);
template int spmv_n_launch<uint16_t>(hgb_ctx *, int, CsrSize, const int *, const int *, const uint16_t *, float,
                                     const float *, float, float *, double *, const int *, int *);
template int spmm_n_launch<double>(hgb_ctx *, int, CsrSize, const int *, const int *, const double *, int, double,
                                   const double *, long, double, double *, long);
template int spmm_n_launch<float>(hgb_ctx *, int, CsrSize, const int *, const int *, const float *, int, float,
                                  const float *, long, float, float *, long);
template int spmm_n_launch<uint16_t>(hgb_ctx *, int, CsrSize, const int *, const int *, const uint16_t *, int, float,
                                     const float *, long, float, float *, long);

template <typename V>
int spmv_t_launch(hgb_ctx *c, int n_rows, int n_cols, const int *pntr, const int *indx, const V *vals,
                  typename Val<V>::X alpha, const typename Val<V>::X *x, typename Val<V>::X beta,
                  typename Val<V>::X *y, const Transpose *T) {
    using X = typename Val<V>::X;
    if (n_cols <= 0) return HGB_OK;
    int gc = std::max(1, std::min((n_cols + 255) / 256, c->num_sms * 8));
    if (T) {
        spmv_t_cached_kernel<V, false><<<gc, 256, 0, c->stream>>>(n_cols, T->pntr, T->row, T->map, vals, spmv_end(alpha, beta), alpha, x,
                                                                 beta, y, nullptr, nullptr, nullptr, nullptr, nullptr);
        return launch_check("spmv_t_cached_kernel");
    }
    scale_or_zero_kernel<X><<<gc, 256, 0, c->stream>>>(n_cols, beta, y);
    if (n_rows > 0) {
        int gr = std::max(1, std::min((n_rows + 255) / 256, c->num_sms * 8));
        spmv_t_atomic_kernel<V><<<gr, 256, 0, c->stream>>>(n_rows, pntr, indx, vals, alpha, x, y);
    }
    return launch_check("spmv_t_atomic_kernel");
}

template int spmv_t_launch<double>(hgb_ctx *, int, int, const int *, const int *, const double *, double,
                                   const double *, double, double *, const Transpose *);
template int spmv_t_launch<float>(hgb_ctx *, int, int, const int *, const int *, const float *, float,
                                  const float *, float, float *, const Transpose *);

}  // namespace hgb

using namespace hgb;

struct hgb_csr {
    hgb_ctx *ctx;
    int n_rows, n_cols, nnz;
    int longest = -1;   // entries of the longest row
    const int *pntr, *indx;
    const void *vals;
    hgb_dtype dtype;
    Transpose T;
    bool has_T = false;
};

namespace hgb {
template <typename T>
__global__ void pattern_grad_kernel(int n_rows, const int *__restrict__ pntr, const int *__restrict__ indx, T alpha,
                                    const T *__restrict__ lam, const T *__restrict__ u, T *__restrict__ grad) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_rows; i += gridDim.x * blockDim.x) {
        const T li = alpha * lam[i];
        for (int p = pntr[i]; p < pntr[i + 1]; p++) grad[p] = li * u[indx[p]];
    }
}

int csr_ensure_transpose(hgb_csr *A) {
    if (A->has_T) return HGB_OK;
    DeviceGuard g(A->ctx->device);
    HGB_TRY(build_transpose(A->ctx, A->n_rows, A->n_cols, A->nnz, A->pntr, A->indx, A->T));
    A->has_T = true;
    return HGB_OK;
}

template <typename V>
int spmv_t_fused_launch(hgb_csr *A, typename Val<V>::X alpha, const typename Val<V>::X *x, typename Val<V>::X beta,
                        typename Val<V>::X *y, const typename Val<V>::X *dot_x, double *dot_out, const int *skip) {
    hgb_ctx *c = A->ctx;
    if (!A->has_T) return fail(HGB_ERR_ARG, "transposed product before the transpose was built");
    const int n = A->n_cols;
    if (n <= 0) return HGB_OK;
    int gc = std::max(1, std::min((n + 255) / 256, std::min(c->num_sms * 8, kMaxReduceBlocks)));
    if (dot_out)
        spmv_t_cached_kernel<V, true><<<gc, 256, 0, c->stream>>>(n, A->T.pntr, A->T.row, A->T.map, (const V *)A->vals,
                                                                spmv_end(alpha, beta), alpha, x, beta, y, dot_x, c->partials, c->counter, dot_out, skip);
    else
        spmv_t_cached_kernel<V, false><<<gc, 256, 0, c->stream>>>(n, A->T.pntr, A->T.row, A->T.map, (const V *)A->vals,
                                                                 spmv_end(alpha, beta), alpha, x, beta, y, nullptr, nullptr, nullptr, nullptr, skip);
    return launch_check("spmv_t_cached_kernel");
}
template int spmv_t_fused_launch<double>(hgb_csr *, double, const double *, double, double *, const double *, double *, const int *);
template int spmv_t_fused_launch<float>(hgb_csr *, float, const float *, float, float *, const float *, double *, const int *);

const int *csr_pntr(const hgb_csr *A) { return A->pntr; }
const int *csr_indx(const hgb_csr *A) { return A->indx; }
const void *csr_vals(const hgb_csr *A) { return A->vals; }
int csr_rows(const hgb_csr *A) { return A->n_rows; }
int csr_cols(const hgb_csr *A) { return A->n_cols; }
int csr_nnz(const hgb_csr *A) { return A->nnz; }
CsrSize csr_size(const hgb_csr *A) { return CsrSize{A->nnz, A->longest}; }
hgb_dtype csr_dtype(const hgb_csr *A) { return A->dtype; }
hgb_ctx *csr_ctx(const hgb_csr *A) { return A->ctx; }
}  // namespace hgb

static int check_spmv_args(hgb_ctx *c, char trans, int n_rows, int n_cols, int nnz, const int *pntr,
                           const int *indx, const void *vals, const void *x, const void *y) {
    if (!c) return fail(HGB_ERR_ARG, "spmv: null context");
    if (n_rows < 0 || n_cols < 0 || nnz < 0) return fail(HGB_ERR_ARG, "spmv: negative size");
    if (trans != 'N' && trans != 'n' && trans != 'T' && trans != 't' && trans != 'C' && trans != 'c')
        return fail(HGB_ERR_ARG, "spmv: trans '%c'", trans);
    if (n_rows > 0 && !pntr) return fail(HGB_ERR_ARG, "spmv: null pntr");
    if (nnz > 0 && (!indx || !vals)) return fail(HGB_ERR_ARG, "spmv: null indx/vals");
    bool nt = (trans == 'N' || trans == 'n');
    if ((nt ? n_rows : n_cols) > 0 && !y) return fail(HGB_ERR_ARG, "spmv: null y");
    if ((nt ? n_cols : n_rows) > 0 && !x && nnz > 0) return fail(HGB_ERR_ARG, "spmv: null x");
    return HGB_OK;
}

extern "C" {

int hgb_spmv_f64(hgb_ctx *c, char trans, int n_rows, int n_cols, int nnz, const int *pntr, const int *indx,
                 const double *vals, double alpha, const double *x, double beta, double *y) {
    HGB_TRY(check_spmv_args(c, trans, n_rows, n_cols, nnz, pntr, indx, vals, x, y));
    DeviceGuard g(c->device);
    if (trans == 'N' || trans == 'n') return spmv_n_launch<double>(c, n_rows, CsrSize{nnz}, pntr, indx, vals, alpha, x, beta, y, nullptr, nullptr);
    return spmv_t_launch<double>(c, n_rows, n_cols, pntr, indx, vals, alpha, x, beta, y, nullptr);
}

int hgb_spmv_f32(hgb_ctx *c, char trans, int n_rows, int n_cols, int nnz, const int *pntr, const int *indx,
                 const float *vals, float alpha, const float *x, float beta, float *y) {
    HGB_TRY(check_spmv_args(c, trans, n_rows, n_cols, nnz, pntr, indx, vals, x, y));
    DeviceGuard g(c->device);
    if (trans == 'N' || trans == 'n') return spmv_n_launch<float>(c, n_rows, CsrSize{nnz}, pntr, indx, vals, alpha, x, beta, y, nullptr, nullptr);
    return spmv_t_launch<float>(c, n_rows, n_cols, pntr, indx, vals, alpha, x, beta, y, nullptr);
}

int hgb_spmv_bf16f32(hgb_ctx *c, char trans, int n_rows, int n_cols, int nnz, const int *pntr,
                     const int *indx, const uint16_t *vals, float alpha, const float *x, float beta, float *y) {
    HGB_TRY(check_spmv_args(c, trans, n_rows, n_cols, nnz, pntr, indx, vals, x, y));
    if (trans != 'N' && trans != 'n') return fail(HGB_ERR_UNSUPPORTED, "spmv_bf16f32: only trans 'N'");
    DeviceGuard g(c->device);
    return spmv_n_launch<uint16_t>(c, n_rows, CsrSize{nnz}, pntr, indx, vals, alpha, x, beta, y, nullptr, nullptr);
}

int hgb_csr_create(hgb_ctx *c, int n_rows, int n_cols, int nnz, const int *pntr, const int *indx,
                   const void *vals, hgb_dtype dtype, hgb_csr **out) {
    if (!out) return fail(HGB_ERR_ARG, "csr_create: null output");
    *out = nullptr;
    HGB_TRY(check_spmv_args(c, 'N', n_rows, n_cols, nnz, pntr, indx, vals, pntr, pntr));
    if (dtype != HGB_F64 && dtype != HGB_F32 && dtype != HGB_BF16 && dtype != HGB_C128 && dtype != HGB_C64)
        return fail(HGB_ERR_ARG, "csr_create: dtype");
    DeviceGuard g(c->device);
    int longest = 0;
    HGB_TRY(csr_check(c, n_rows, n_cols, nnz, pntr, indx, &longest));
    hgb_csr *A = new hgb_csr();
    A->longest = longest;
    A->ctx = c;
    A->n_rows = n_rows;
    A->n_cols = n_cols;
    A->nnz = nnz;
    A->pntr = pntr;
    A->indx = indx;
    A->vals = vals;
    A->dtype = dtype;
    *out = A;
    return HGB_OK;
}

int hgb_csr_gemv(hgb_csr *A, char trans, double alpha, const void *x, double beta, void *y) {
    if (!A) return fail(HGB_ERR_ARG, "csr_gemv: null matrix");
    hgb_ctx *c = A->ctx;
    HGB_TRY(check_spmv_args(c, trans, A->n_rows, A->n_cols, A->nnz, A->pntr, A->indx, A->vals, x, y));
    DeviceGuard g(c->device);
    bool nt = (trans == 'N' || trans == 'n');
    if (A->dtype == HGB_C128 || A->dtype == HGB_C64) {
        const double a[2] = {alpha, 0.0}, b[2] = {beta, 0.0};
        return hgb_csr_gemv_z(A, trans, a, x, b, y);
    }
    if (nt) {
        switch (A->dtype) {
            case HGB_F64: return spmv_n_launch<double>(c, A->n_rows, csr_size(A), A->pntr, A->indx, (const double *)A->vals, alpha, (const double *)x, beta, (double *)y, nullptr, nullptr);
            case HGB_F32: return spmv_n_launch<float>(c, A->n_rows, csr_size(A), A->pntr, A->indx, (const float *)A->vals, (float)alpha, (const float *)x, (float)beta, (float *)y, nullptr, nullptr);
            default: return spmv_n_launch<uint16_t>(c, A->n_rows, csr_size(A), A->pntr, A->indx, (const uint16_t *)A->vals, (float)alpha, (const float *)x, (float)beta, (float *)y, nullptr, nullptr);
        }
    }
    if (A->dtype == HGB_BF16) return fail(HGB_ERR_UNSUPPORTED, "csr_gemv: transpose of a bf16 matrix");
    if (!A->has_T) {
        HGB_TRY(build_transpose(c, A->n_rows, A->n_cols, A->nnz, A->pntr, A->indx, A->T));
        A->has_T = true;
    }
    if (A->dtype == HGB_F64)
        return spmv_t_launch<double>(c, A->n_rows, A->n_cols, A->pntr, A->indx, (const double *)A->vals, alpha, (const double *)x, beta, (double *)y, &A->T);
    return spmv_t_launch<float>(c, A->n_rows, A->n_cols, A->pntr, A->indx, (const float *)A->vals, (float)alpha, (const float *)x, (float)beta, (float *)y, &A->T);
}

int hgb_csr_gemv_z(hgb_csr *A, char trans, const double *alpha, const void *x, const double *beta, void *y) {
    if (!A || !alpha || !beta) return fail(HGB_ERR_ARG, "csr_gemv_z: bad arguments");
    if (A->dtype != HGB_C128 && A->dtype != HGB_C64) return fail(HGB_ERR_ARG, "csr_gemv_z: a complex matrix");
    hgb_ctx *c = A->ctx;
    HGB_TRY(check_spmv_args(c, trans, A->n_rows, A->n_cols, A->nnz, A->pntr, A->indx, A->vals, x, y));
    DeviceGuard g(c->device);
    const bool nt = (trans == 'N' || trans == 'n');
    if (!nt && !A->has_T) {
        HGB_TRY(build_transpose(c, A->n_rows, A->n_cols, A->nnz, A->pntr, A->indx, A->T));
        A->has_T = true;
    }
    const Transpose *T = nt ? nullptr : &A->T;
    if (A->dtype == HGB_C128)
        return zspmv<double>(c, trans, A->n_rows, A->n_cols, A->pntr, A->indx, A->vals, alpha, x, beta, y, T);
    const float a[2] = {(float)alpha[0], (float)alpha[1]}, b[2] = {(float)beta[0], (float)beta[1]};
    return zspmv<float>(c, trans, A->n_rows, A->n_cols, A->pntr, A->indx, A->vals, a, x, b, y, T);
}

int hgb_spmv_c128(hgb_ctx *c, char trans, int n_rows, int n_cols, int nnz, const int *pntr, const int *indx,
                  const void *vals, const double *alpha, const void *x, const double *beta, void *y) {
    HGB_TRY(check_spmv_args(c, trans, n_rows, n_cols, nnz, pntr, indx, vals, x, y));
    if (!alpha || !beta) return fail(HGB_ERR_ARG, "spmv_c128: null scalar");
    DeviceGuard g(c->device);
    return zspmv<double>(c, trans, n_rows, n_cols, pntr, indx, vals, alpha, x, beta, y, nullptr);
}

int hgb_spmv_c64(hgb_ctx *c, char trans, int n_rows, int n_cols, int nnz, const int *pntr, const int *indx,
                 const void *vals, const float *alpha, const void *x, const float *beta, void *y) {
    HGB_TRY(check_spmv_args(c, trans, n_rows, n_cols, nnz, pntr, indx, vals, x, y));
    if (!alpha || !beta) return fail(HGB_ERR_ARG, "spmv_c64: null scalar");
    DeviceGuard g(c->device);
    return zspmv<float>(c, trans, n_rows, n_cols, pntr, indx, vals, alpha, x, beta, y, nullptr);
}

int hgb_csr_gemv_dot(hgb_csr *A, const void *x, void *y, double *dot_out) {
    if (!A || !dot_out) return fail(HGB_ERR_ARG, "csr_gemv_dot: bad arguments");
    if (A->dtype == HGB_C128 || A->dtype == HGB_C64) return fail(HGB_ERR_UNSUPPORTED, "csr_gemv_dot: real matrices");
    if (A->n_rows != A->n_cols) return fail(HGB_ERR_ARG, "csr_gemv_dot: square matrix required");
    hgb_ctx *c = A->ctx;
    DeviceGuard g(c->device);
    switch (A->dtype) {
        case HGB_F64: return spmv_n_launch<double>(c, A->n_rows, csr_size(A), A->pntr, A->indx, (const double *)A->vals, 1.0, (const double *)x, 0.0, (double *)y, dot_out, nullptr);
        case HGB_F32: return spmv_n_launch<float>(c, A->n_rows, csr_size(A), A->pntr, A->indx, (const float *)A->vals, 1.0f, (const float *)x, 0.0f, (float *)y, dot_out, nullptr);
        default: return spmv_n_launch<uint16_t>(c, A->n_rows, csr_size(A), A->pntr, A->indx, (const uint16_t *)A->vals, 1.0f, (const float *)x, 0.0f, (float *)y, dot_out, nullptr);
    }
}

int hgb_csr_pattern_grad(hgb_csr *A, double alpha, const void *lam, const void *u, void *grad) {
    if (!A || !lam || !u || !grad) return fail(HGB_ERR_ARG, "csr_pattern_grad: bad arguments");
    if (A->dtype != HGB_F64 && A->dtype != HGB_F32) return fail(HGB_ERR_UNSUPPORTED, "csr_pattern_grad: F64 or F32 matrices");
    hgb_ctx *c = A->ctx;
    DeviceGuard g(c->device);
    if (A->n_rows == 0) return HGB_OK;
    int gr = std::max(1, std::min((A->n_rows + 255) / 256, c->num_sms * 8));
    if (A->dtype == HGB_F64)
        pattern_grad_kernel<double><<<gr, 256, 0, c->stream>>>(A->n_rows, A->pntr, A->indx, alpha, (const double *)lam, (const double *)u, (double *)grad);
    else
        pattern_grad_kernel<float><<<gr, 256, 0, c->stream>>>(A->n_rows, A->pntr, A->indx, (float)alpha, (const float *)lam, (const float *)u, (float *)grad);
    return launch_check("pattern_grad_kernel");
}

int hgb_csr_destroy(hgb_csr *A) {
    if (!A) return HGB_OK;
    DeviceGuard g(A->ctx->device);
    if (A->has_T) A->T.release();
    delete A;
    return HGB_OK;
}

}  // extern "C"
