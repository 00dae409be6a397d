// Strip-scheduled sparse triangular solve for sm_103a.
//
// A sweep is a wavefront: on a natural-ordered grid its length is the number of levels (382 on
// 128^3), and the time is levels x (time of one step) + hand-overs x (time of one hand-over); the
// bytes (about 48 per row) are a tenth of it.  So everything that a step does not have to wait
// for is off its path, and a hand-over is one store.  Measured (GB300, both sweeps): 128^3 with BF16
// or FP32 store 168 us (a step about 130 ns, a hand-over 0.25 us inside a cluster and 1.2 us between
// clusters), FP64 361 us (a step 280-400 ns: six to nine dependent FP64 operations of 62 cycles);
// 512^2 FP32 209 us (1023 levels).  With steps of 128 rows between barriers and every value of
// another block through a ring: 322, 576 and 4550 us.
//
// A strip of consecutive rows (hgb_bsplan.cu) is solved a step at a time, a step being at most 32 rows
// of one local level, one row per lane.  The steps of a strip go round kBsK warps: while one warp
// is in the part of its step that depends on the step before (a named barrier, the loads of the
// strip's own values, the arithmetic, the store of the result), the others store their results to
// memory, offer them, and prepare their next steps.  A value that comes from elsewhere is its own
// ready flag: all values that a CTA's rows read have a slot in its shared memory, and the slots of
// values from other strips start with a pending pattern (a signalling NaN, which arithmetic never
// produces) and are polled there until the value is in, before the step's turn; the products and the
// leading sum that need only such values are formed before it too.  Inside a CTA the strip that
// owns a row stores it into its slot; between the CTAs of a thread-block cluster the owner stores it
// into the reader's slot (distributed shared memory), each slot being written once per sweep, so
// that nothing can be overwritten or dropped.  Across clusters the owner stores it into the reader's
// mailbox in memory, which has an entry per slot: a strip's mail lies in the order in which the strip
// uses it, and one warp per strip polls it with 16-byte loads, copies it to the slots and puts the
// pending pattern back for the next launch.  (Polling the scattered solution entries instead, even
// in windows sorted by row, limited the sweep behind each cluster boundary: 128^3, FP32, 360 ns per
// step against 137 before it.)
//
// The row packets (codes, values, diagonal terms) of a warp's steps lie in the order in which it reads
// them.  Lane 0 copies them a step at a time into a ring in shared memory (cp.async.bulk on an
// mbarrier); the right-hand side is gathered by per-lane cp.async RA of the warp's steps ahead, from
// row numbers that travel with the packets RA steps before.
//
// Rows keep the reference's accumulation order (sparse/hala_sparse_utils.hpp: apply_ilu_array,
// sparse_trsv_array), products and sums separately rounded, so results are bit-identical to the
// sequential loops.  Padding entries subtract 0 * 0, which changes no sum and quiets a signalling
// NaN of the right-hand side, so that no result looks pending.  Blocks are handed out by an atomic
// ticket per cluster in solve order, so a wait is only ever on rows of running or finished CTAs, and
// each wait is bounded.
#include "hgb_internal.cuh"
#include "hgb_kernels.cuh"
#include "hgb_bsolve.cuh"

#include <algorithm>
#include <climits>
#include <mutex>
#include <new>
#include <vector>

namespace hgb {

constexpr int kBsMaxCluster = 16;  // largest thread-block cluster (above 8: non-portable sizes)

// the diagonal of a sweep: unit, divided by, or multiplied by the FP32 reciprocal of an FP64 pivot
enum : int { BS_UNIT = 0, BS_DIV = 1, BS_RECIP = 2 };

// A row's values from its value pieces (pieces are the step's row count apart):
//   FP64 {v0, v1} {v2, RN(1/d)} {d, 0} (no third piece in a unit sweep);  FP32 {v0, v1, v2, dv}
// (a BF16 store is expanded: the same values).
template <typename X> struct BsRow;
template <> struct BsRow<double> {
    double v[3], d, dinv;
    template <int DIAG> __device__ __forceinline__ void load(const int4 *p, int stride) {
        const double2 a = *(const double2 *)p, b = *(const double2 *)(p + stride);
        v[0] = a.x;
        v[1] = a.y;
        v[2] = b.x;
        dinv = b.y;
        d = 0.0;
        if (DIAG != BS_UNIT) d = *(const double *)(p + 2 * stride);
    }
};
template <> struct BsRow<float> {
    float v[3], d;
    template <int DIAG> __device__ __forceinline__ void load(const int4 *p, int) {
        const float4 a = *(const float4 *)p;
        v[0] = a.x;
        v[1] = a.y;
        v[2] = a.z;
        d = a.w;
    }
};

// a / d correctly rounded, from the stored y = RN(1/d): q0 = RN(a y), r = a - d q0 (exact with
// FMA), q = RN(q0 + r y) equals RN(a / d) (Markstein, IBM J. Res. Dev. 34(1), 1990) when no step
// overflows or underflows.  Operands with |exponent| >= 500, zeros, infinities and NaNs take the
// division instead; for such a d the packet stores y = 0.  The guards are integer tests (the FP64
// pipe of sm_103 is slow).
__host__ __device__ constexpr bool bs_markstein_range(unsigned biased_exp) { return biased_exp - 523u < 1000u; }
template <int DIAG>
__device__ __forceinline__ double bs_divide(double a, const BsRow<double> &r) {
    const unsigned ea = ((unsigned)__double2hiint(a) >> 20) & 0x7FFu;
    if (bs_markstein_range(ea) && __double_as_longlong(r.dinv) != 0) {
        const double q0 = __dmul_rn(a, r.dinv);
        const double rem = __fma_rn(-r.d, q0, a);
        return __fma_rn(rem, r.dinv, q0);
    }
    return __ddiv_rn(a, r.d);
}
template <int DIAG>
__device__ __forceinline__ float bs_divide(float a, const BsRow<float> &r) {
    return DIAG == BS_RECIP ? __fmul_rn(a, r.d) : __fdiv_rn(a, r.d);
}

struct BsArgs {
    int nblk, cl, nflag;
    const int4 *blk, *strip;
    const unsigned char *packets;
    const int2 *watch;
    void *mail;
    const int *ext_codes;
    const void *ext_vals;
    int *ticket;
    int *err;
    const int *skip;
};

__device__ __forceinline__ unsigned bs_cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned bs_cluster_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void bs_cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void bs_cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t bs_peer(uint32_t local, unsigned rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ void bs_peer_store(uint32_t a, int v) {
    asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// a solution value into a peer's slot: strong (relaxed, cluster scope), the peer polls it
__device__ __forceinline__ void bs_offer(uint32_t a, double v) {
    asm volatile("st.relaxed.cluster.shared::cluster.b64 [%0], %1;" ::"r"(a), "l"(__double_as_longlong(v)) : "memory");
}
__device__ __forceinline__ void bs_offer(uint32_t a, float v) {
    asm volatile("st.relaxed.cluster.shared::cluster.b32 [%0], %1;" ::"r"(a), "r"(__float_as_uint(v)) : "memory");
}
// slots: strong loads and stores (peers and the CTA's other warps access them without a barrier)
__device__ __forceinline__ double bs_slot(uint32_t a, double) {
    unsigned long long v;
    asm volatile("ld.relaxed.cluster.shared::cta.b64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return __longlong_as_double((long long)v);
}
__device__ __forceinline__ float bs_slot(uint32_t a, float) {
    unsigned v;
    asm volatile("ld.relaxed.cluster.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return __uint_as_float(v);
}
__device__ __forceinline__ void bs_set_slot(uint32_t a, double v) {
    asm volatile("st.relaxed.cluster.shared::cta.b64 [%0], %1;" ::"r"(a), "l"(__double_as_longlong(v)) : "memory");
}
__device__ __forceinline__ void bs_set_slot(uint32_t a, float v) {
    asm volatile("st.relaxed.cluster.shared::cta.b32 [%0], %1;" ::"r"(a), "r"(__float_as_uint(v)) : "memory");
}

// packet copies
__device__ __forceinline__ void bs_mbar_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bs_copy_chunk(uint32_t dst, const void *src, unsigned bytes, uint32_t bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool bs_mbar_done(uint32_t bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// one element of the right-hand side, into this lane's ring entry
__device__ __forceinline__ void bs_copy_rhs(uint32_t dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void bs_copy_rhs(uint32_t dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// An entry of a mailbox that no row writes: another signalling NaN
template <typename X> struct BsVoid;
template <> struct BsVoid<double> {
    static constexpr unsigned long long bits = 0x7FF4DEADBEEF0002ull;
    __device__ static bool is(double v) { return (unsigned long long)__double_as_longlong(v) == bits; }
    __device__ static double value() { return __longlong_as_double((long long)bits); }
};
template <> struct BsVoid<float> {
    static constexpr unsigned bits = 0x7FA5A5A6u;
    __device__ static bool is(float v) { return __float_as_uint(v) == bits; }
    __device__ static float value() { return __uint_as_float(bits); }
};
// a 16-byte unit of a mailbox; its elements are strong loads, each its own ready flag
template <typename X> struct BsUnit;
template <> struct BsUnit<double> {
    double x[2];
    __device__ __forceinline__ void load(const int4 *p) {
        unsigned long long a, b;
        asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
        x[0] = __longlong_as_double((long long)a);
        x[1] = __longlong_as_double((long long)b);
    }
    __device__ __forceinline__ bool pending() const { return Pending<double>::is(x[0]) || Pending<double>::is(x[1]); }
    __device__ __forceinline__ void reset(int4 *p) const {
        const double q = Pending<double>::value();
        *(double2 *)p = make_double2(BsVoid<double>::is(x[0]) ? x[0] : q, BsVoid<double>::is(x[1]) ? x[1] : q);
    }
};
template <> struct BsUnit<float> {
    float x[4];
    __device__ __forceinline__ void load(const int4 *p) {
        asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3])
                     : "l"(p)
                     : "memory");
    }
    __device__ __forceinline__ bool pending() const {
        return Pending<float>::is(x[0]) || Pending<float>::is(x[1]) || Pending<float>::is(x[2]) || Pending<float>::is(x[3]);
    }
    __device__ __forceinline__ void reset(int4 *p) const {
        float r[4];
#pragma unroll
        for (int e = 0; e < 4; e++) r[e] = BsVoid<float>::is(x[e]) ? x[e] : Pending<float>::value();
        *(float4 *)p = make_float4(r[0], r[1], r[2], r[3]);
    }
};

// Polls of a slot run at shared-memory speed for a few thousand rounds (a hand-over takes a few), then
// sleep; the bound is about a second.  A wait that runs out, here or in any other warp of the
// launch, sets DEV_ERR_TIMEOUT and gives NaN, so that all dependents end too.
constexpr int kBsPollFast = 4096, kBsPollLimit = 1 << 23;
__device__ __noinline__ bool bs_poll_pause(int spins, int *err) {
    if (spins > kBsPollFast) __nanosleep(64);
    if (spins > kBsPollLimit || ((spins & 1023) == 0 && (*(volatile int *)err & DEV_ERR_TIMEOUT))) {
        atomicOr(err, DEV_ERR_TIMEOUT);
        return false;
    }
    return true;
}
__device__ __forceinline__ bool bs_pending(double v) { return (unsigned)__double2hiint(v) == (unsigned)(Pending<double>::bits >> 32); }
__device__ __forceinline__ bool bs_pending(float v) { return __float_as_uint(v) == Pending<float>::bits; }
template <typename X>
__device__ __forceinline__ X bs_nan() { return Pending<X>::canon(Pending<X>::value()); }

// the value of a slot, polled until it is in (v: its first reading)
template <typename X>
__device__ __forceinline__ X bs_wait_slot(uint32_t a, X v, int *err) {
    int spins = 0;
    while (bs_pending(v)) {
        if ((++spins & 255) == 0 || spins > kBsPollFast)
            if (!bs_poll_pause(spins, err)) return bs_nan<X>();
        v = bs_slot(a, X(0));
    }
    return v;
}
// Holds a value where it is computed: without it the compiler moves the arithmetic from before a step's
// turn behind it, or computes both sides of a (warp-uniform) choice and selects.
__device__ __forceinline__ void bs_pin(double &v) { asm volatile("" : "+d"(v)); }
__device__ __forceinline__ void bs_pin(float &v) { asm volatile("" : "+f"(v)); }
// one product taken into the sum
template <int MODE, typename X>
__device__ __forceinline__ X bs_term(X acc, X m) {
    return MODE == 0 ? sub_rn(acc, m) : add_rn(acc, m);
}
// hand-over from a step to the next one of its strip: the producer warp arrives, the consumer waits
__device__ __forceinline__ void bs_step_done(int id) { asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void bs_step_wait(int id) { asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory"); }

// MODE 0: x_i = (b_i - sum_k v_k x_k) [/ d_i]  (apply_ilu_array's order);
// MODE 1: x_i = (alpha b_i - (sum_k v_k x_k)) [/ d_i]  (sparse_trsv_array's order).
// LOOK: look for the values from other strips before a step's turn (always in FP64; in FP32 not for the
// patterns of 3D grids, where they are never in that early: 180 us per 128^3 BF16-store application
// without, 204 with; the 512^2 one 260 without, 232 with).
// EXT: some row of the plan lists its entries in the ext arrays (a form of its own: without it all sweeps took 6 to 12 %
// longer, 128^3 FP32 194 us a pair against 184, 512^2 254 against 228, FP64 596 against 528).
template <typename X, int MODE, int DIAG, bool LOOK, bool EXT>
__global__ void __launch_bounds__(kBsThreads, 1)
bsolve_kernel(BsArgs A, X alpha, const X *in, X *out, X *pend) {
    constexpr int XS = sizeof(X), W = kBsW, K = kBsK, D = bs_d(XS), RA = bs_ra(XS);
    constexpr int NU = DIAG != BS_UNIT, NP = bs_np(XS, NU), CB = bs_chunk_bytes(XS, NU), CTA = kBsThreads, QE = 16 / XS;
    static_assert(W * K <= 16, "a named barrier per solver warp");
    static_assert(RA < D, "the first right-hand sides come from landed chunks");
    static_assert(CB % 16 == 0, "bulk copies");
    if (A.skip && *A.skip) return;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) unsigned long long bars[W * K][D];
    __shared__ int blk_sh;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    const unsigned rank = bs_cluster_rank(), ncl = bs_cluster_size();
    if ((int)ncl != A.cl) {   // the plan's offers assume clusters of A.cl CTAs
        if (t == 0) atomicOr(A.err, DEV_ERR_CSR);
        return;
    }
    bs_cluster_arrive();   // a peer's shared memory is written only after this CTA has started
    const int sw = warp < W * K ? warp : 0;   // solver warp
    unsigned char *ring = smem + (size_t)sw * (D * CB);
    X *rhs = (X *)(smem + (size_t)(W * K) * (D * CB)) + sw * (RA * 32) + lane;
    X *slots = (X *)(smem + bs_ring_bytes(XS, NU));
    const uint32_t sbase = smem_addr(slots), rhs_a = smem_addr(rhs), ring_a = smem_addr(ring), bar_a = smem_addr(&bars[sw][0]);
    if (warp < W * K && lane == 0) {
        for (int k = 0; k < D; k++) bs_mbar_init(bar_a + 8 * k);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    // the ring position that the warp's next chunk takes, and the parity of its barrier
    int wslot = 0;
    unsigned wpar = 0;
    for (int round = 0;; round++) {
        // clusters take tickets; rank r of the cluster with ticket q solves block q * ncl + r.  The
        // first barrier: every CTA of the cluster runs and is done with the previous round (its slots and its
        // peers' are read); the second: the ticket and the pending slots are visible to all.
        __syncwarp();
        if (round) bs_cluster_arrive();
        bs_cluster_wait();
        if (t == 0 && rank == 0) {
            const int q = atomicAdd(A.ticket, 1);
            for (unsigned r = 0; r < ncl; r++) bs_peer_store(bs_peer(smem_addr(&blk_sh), r), q);
        }
        for (int i = t; i < A.nflag; i += CTA) slots[i] = i == 0 ? X(0) : Pending<X>::value();
        __syncwarp();
        bs_cluster_arrive();
        bs_cluster_wait();
        const int q = blk_sh;
        if (q * (int)ncl >= A.nblk) break;   // the same for the whole cluster
        const int b = q * (int)ncl + (int)rank;
        if (b >= A.nblk) continue;           // the last cluster may have spare ranks

        if (warp >= W * K) {
            // ---- mail warp of strip mw: every lane goes through its units of the strip's mail (32 apart, two
            // at a time) and moves on as soon as all values of a unit are in; beside them through its share
            // of the block's watches
            const int mw = warp - W * K;
            const int4 bf = __ldg(A.blk + 4 * b + 1), seg = __ldg(A.blk + 4 * b + 2 + (mw >> 1));
            const int first = (mw & 1) ? seg.z : seg.x, end = bf.z < 0 ? 0 : ((mw & 1) ? seg.w : seg.y);
            int4 *box = (int4 *)A.mail + bf.z;
            int u[2] = {first + lane, first + 32 + lane}, wi = 32 * mw + lane;
            int2 f = wi < bf.y ? __ldg(A.watch + bf.x + wi) : make_int2(0, 0);
            for (int spins = 1; __any_sync(0xFFFFFFFFu, u[0] < end || u[1] < end || wi < bf.y); spins++) {
                BsUnit<X> v[2];
                X w = X(0);
                bool moved = false;
#pragma unroll
                for (int j = 0; j < 2; j++)
                    if (u[j] < end) v[j].load(box + u[j]);
                if (wi < bf.y) w = ld_relaxed(out + f.x);
#pragma unroll
                for (int j = 0; j < 2; j++)
                    if (u[j] < end && !v[j].pending()) {
#pragma unroll
                        for (int e = 0; e < QE; e++)
                            if (!BsVoid<X>::is(v[j].x[e])) bs_set_slot(sbase + (u[j] * QE + e) * XS, v[j].x[e]);
                        v[j].reset(box + u[j]);
                        u[j] += 64;
                        moved = true;
                    }
                if (wi < bf.y && !Pending<X>::is(w)) {
                    bs_set_slot(sbase + f.y * XS, w);
                    wi += 32 * W;
                    if (wi < bf.y) f = __ldg(A.watch + bf.x + wi);
                    moved = true;
                }
                if (!__any_sync(0xFFFFFFFFu, moved)) {
                    __nanosleep(20);
                    if ((spins & 255) == 0 && __any_sync(0xFFFFFFFFu, !bs_poll_pause(spins, A.err))) {
                        // given up: NaN for all that is left, so that the solver warps end too
                        for (int j = 0; j < 2; j++)
                            for (; u[j] < end; u[j] += 64) {
                                BsUnit<X> r;
                                r.load(box + u[j]);
                                for (int e = 0; e < QE; e++)
                                    if (!BsVoid<X>::is(r.x[e])) bs_set_slot(sbase + (u[j] * QE + e) * XS, bs_nan<X>());
                            }
                        for (; wi < bf.y; wi += 32 * W) bs_set_slot(sbase + __ldg(A.watch + bf.x + wi).y * XS, bs_nan<X>());
                        break;
                    }
                }
            }
            continue;
        }

        // ---- solver warps: warp k of group g takes the steps k, k + K, ... of strip g (a block has at most W)
        const int4 bi = __ldg(A.blk + 4 * b);
        const int g = warp / K, k = warp % K;
        if (g < bi.y) {
            const int4 sd = __ldg(A.strip + 2 * ((bi.x + g) * K + k)), sz = __ldg(A.strip + 2 * ((bi.x + g) * K + k) + 1);
            const int ns = sd.y, nch = (ns - k + K - 1) / K;   // steps of the strip, and this warp's
            const X *inb = in + sd.x;
            X *outb = out + sd.x, *pendb = pend ? pend + sd.x : nullptr;
            const unsigned char *src = A.packets + (size_t)sd.z * 16;   // next chunk to copy (lane 0)
            if (lane == 0) {
                const int words[4] = {sz.x, sz.y, sz.z, sz.w};
                int islot = wslot;
#pragma unroll
                for (int c = 0; c < D; c++)
                    if (c < nch) {
                        const unsigned bytes = ((unsigned)words[c >> 1] >> (16 * (c & 1)) & 0xFFFFu) * 16;
                        bs_copy_chunk(ring_a + islot * CB, src, bytes, bar_a + 8 * islot);
                        src += bytes;
                        islot = islot + 1 == D ? 0 : islot + 1;
                    }
            }
            auto wait_chunk = [&](int slot, unsigned par) {
                int spins = 0;
                while (!bs_mbar_done(bar_a + 8 * slot, par))
                    if (++spins > kSpinLimit) {   // a copy in flight always lands: not met in practice
                        atomicOr(A.err, DEV_ERR_TIMEOUT);
                        break;
                    }
            };
            // ---- the first RA right-hand sides: their rows are in the first chunks' packets
            {
                int slot = wslot;
                unsigned par = wpar;
                for (int c = 0; c < RA; c++) {
                    if (c < nch) {
                        wait_chunk(slot, par);
                        const int cnt = *(const int *)(ring + slot * CB) & 0xFF;
                        if (lane < cnt)
                            bs_copy_rhs(rhs_a + c * 32 * XS, inb + *(const unsigned short *)(ring + slot * CB + 16 + lane * 16 + 8));
                        slot = slot + 1 == D ? 0 : slot + 1;
                        if (slot == 0) par ^= 1;
                    }
                    cp_async_commit();
                }
            }
            int rslot = 0;   // right-hand-side ring entry of the current step
            for (int c = 0; c < nch; c++) {
                const int s = c * K + k;
                // ---- the step's packet: {rows | flags, rows RA ahead, units of the chunk D ahead, 0}, first
                // pieces, value pieces, row numbers RA ahead
                wait_chunk(wslot, wpar);
                const unsigned char *base = ring + wslot * CB;
                const int4 h = *(const int4 *)base;
                const int cnt = h.x & 0xFF;
                const bool act = lane < cnt;
                int4 p = make_int4(0, kBsNoSlot << 16, 0, 0);   // an idle lane reads the zero slot
                if (act) p = *(const int4 *)(base + 16 + lane * 16);
                BsRow<X> rw;
                rw.template load<DIAG>((const int4 *)(base + 16) + cnt + min(lane, cnt - 1), cnt);
                int ahead = 0;
                if (lane < h.y) ahead = *(const unsigned short *)(base + 16 + cnt * (NP * 16) + lane * 2);
                asm volatile("cp.async.wait_group %0;" ::"n"(RA - 1) : "memory");
                const X xin = rhs[rslot * 32];
                const bool ext = (p.w & kBsExt) != 0;
                const unsigned c0 = ext ? 0 : (unsigned)p.x & 0xFFFF, c1 = ext ? 0 : (unsigned)p.x >> 16,
                               c2 = ext ? 0 : (unsigned)p.y & 0xFFFF;
                const uint32_t a0 = sbase + c0 * XS, a1 = sbase + c1 * XS, a2 = sbase + c2 * XS;
                const unsigned slot = (unsigned)p.y >> 16;
                const uint32_t slot_a = sbase + slot * XS;
                const bool push = act && (p.w & kBsPush), post = act && (p.w & kBsMail);
                uint32_t offer_a = 0;
                if (push) offer_a = bs_peer(sbase + ((unsigned)p.z >> 16) * XS, rank + (p.w & 0xFF));
                X *mail = nullptr;
                if (post) mail = (X *)A.mail + (long)__ldg(A.blk + 4 * (b + (p.w & 0xFF)) + 1).z * QE + ((unsigned)p.z >> 16);
                const bool early0 = h.x & kBsEarly0, early2 = h.x & kBsEarly2, no2 = h.x & kBsNo2;   // uniform
                X ax = X(0);
                if (MODE == 1) ax = mul_rn(alpha, xin);
                // rows with their entries in the ext arrays: the first ones' codes and values, of all rows' count
                constexpr int PE = XS == 8 ? 2 : 4;   // registers: four in FP64 cost a grid with a few long rows 7.1 -> 7.6 ms
                int nd = 0, most = 0, ecode[PE];
                X evalue[PE];
                auto load_ext = [&](int q0) {
#pragma unroll
                    for (int u = 0; u < PE; u++)
                        if (q0 + u < nd) {
                            const long e = (long)p.x + (long)(q0 + u) * cnt;
                            ecode[u] = __ldg(A.ext_codes + e);
                            evalue[u] = __ldg((const X *)A.ext_vals + e);
                        }
                };
                if (EXT && (h.x & kBsStepExt)) {
                    nd = ext && act ? p.y & 0xFFFF : 0;
                    most = __reduce_max_sync(0xFFFFFFFFu, nd);
                    load_ext(0);
                }
                // ---- before the step's turn: whether all values that come from other strips and blocks (far) are
                // in, so that its turn need not poll; FP64: the arithmetic that needs no others, an operation taking 64 cycles
                X acc = (MODE == 0) ? xin : X(0), m2 = X(0);
                bool early = false;
                if (LOOK) {
                    const X x0 = bs_slot(p.w & kBsFar ? a0 : sbase, X(0)), x1 = bs_slot(p.w & kBsFar << 1 ? a1 : sbase, X(0)),
                            x2 = bs_slot(p.w & kBsFar << 2 ? a2 : sbase, X(0));
                    early = !__any_sync(0xFFFFFFFFu, bs_pending(x0) || bs_pending(x1) || bs_pending(x2));
                    if (XS == 8) {
                        HGB_UNIFORM_IF(early && early0) {
                            acc = bs_term<MODE>(acc, mul_rn(rw.v[0], x0));
                            bs_pin(acc);
                        }
                        HGB_UNIFORM_IF(early && early2 && !no2) {
                            m2 = mul_rn(rw.v[2], x2);
                            bs_pin(m2);
                        }
                    }
                }
                // ---- its turn: the strip's own values are in; the far ones are polled.  The warp polls as one:
                // lanes that left a loop one by one would run the rest of the step apart.
                if (s > 0) bs_step_wait(g * K + (k + K - 1) % K);
                X x0 = bs_slot(a0, X(0)), x1 = bs_slot(a1, X(0)), x2 = bs_slot(a2, X(0));
                if (!early)
                    for (int spins = 1; __any_sync(0xFFFFFFFFu, bs_pending(x0) || bs_pending(x1) || bs_pending(x2)); spins++) {
                        if ((spins & 255) == 0 || spins > kBsPollFast) {
                            if (__any_sync(0xFFFFFFFFu, !bs_poll_pause(spins, A.err))) {
                                if (bs_pending(x0)) x0 = bs_nan<X>();
                                if (bs_pending(x1)) x1 = bs_nan<X>();
                                if (bs_pending(x2)) x2 = bs_nan<X>();
                                break;
                            }
                        }
                        x0 = bs_slot(a0, X(0));
                        x1 = bs_slot(a1, X(0));
                        x2 = bs_slot(a2, X(0));
                    }
                if (XS == 8) {
                    X m1 = mul_rn(rw.v[1], x1);
                    bs_pin(m1);
                    HGB_UNIFORM_IF(!early || !early0) {
                        acc = bs_term<MODE>(acc, mul_rn(rw.v[0], x0));
                        bs_pin(acc);
                    }
                    HGB_UNIFORM_IF((!early || !early2) && !no2) {
                        m2 = mul_rn(rw.v[2], x2);
                        bs_pin(m2);
                    }
                    acc = bs_term<MODE>(acc, m1);
                    HGB_UNIFORM_IF(!no2) {
                        acc = bs_term<MODE>(acc, m2);
                        bs_pin(acc);
                    }
                } else {
                    acc = bs_term<MODE>(acc, mul_rn(rw.v[0], x0));
                    acc = bs_term<MODE>(acc, mul_rn(rw.v[1], x1));
                    acc = bs_term<MODE>(acc, mul_rn(rw.v[2], x2));
                }
                if (EXT && (h.x & kBsStepExt)) {   // PE entries at a time, the next ones' loads in flight
                    for (int q0 = 0; q0 < most; q0 += PE) {
                        X xk[PE], vk[PE];
                        int cd[PE];
#pragma unroll
                        for (int u = 0; u < PE; u++)
                            if (q0 + u < nd) {
                                cd[u] = ecode[u];
                                vk[u] = evalue[u];
                                xk[u] = cd[u] >= 0 ? bs_slot(sbase + cd[u] * XS, X(0)) : ld_relaxed(out + (-cd[u] - 1));
                            }
                        load_ext(q0 + PE);
#pragma unroll
                        for (int u = 0; u < PE; u++)
                            if (q0 + u < nd) {
                                if (cd[u] >= 0) xk[u] = bs_wait_slot(sbase + cd[u] * XS, xk[u], A.err);
                                else if (Pending<X>::is(xk[u])) xk[u] = wait_value(out + (-cd[u] - 1), A.err);
                                acc = bs_term<MODE>(acc, mul_rn(vk[u], xk[u]));
                            }
                    }
                    __syncwarp();
                }
                if (MODE == 1) acc = sub_rn(ax, acc);
                if (DIAG != BS_UNIT) acc = bs_divide<DIAG>(act ? acc : X(1), rw);   // idle lanes: no slow division
                if (slot != kBsNoSlot) bs_set_slot(slot_a, acc);
                if (push) bs_offer(offer_a, acc);
                if (post) st_relaxed(mail, acc);
                __syncwarp();
                if (s + 1 < ns) bs_step_done(g * K + k);
                // ---- after it
                if (act) {
                    const int row = p.z & 0xFFFF;
                    st_relaxed(outb + row, acc);
                    if (p.w & kBsReset) pendb[row] = Pending<X>::value();
                }
                if (lane < h.y) bs_copy_rhs(rhs_a + rslot * 32 * XS, inb + ahead);
                cp_async_commit();
                rslot = rslot + 1 == RA ? 0 : rslot + 1;
                __syncwarp();   // every lane has read this chunk
                if (h.z && lane == 0) {
                    const unsigned bytes = (unsigned)h.z * 16;
                    bs_copy_chunk(ring_a + wslot * CB, src, bytes, bar_a + 8 * wslot);
                    src += bytes;
                }
                wslot = wslot + 1 == D ? 0 : wslot + 1;
                if (wslot == 0) wpar ^= 1;
            }
            cp_async_wait<0>();
        }
    }
    // the last CTA to leave resets the ticket for the next launch
    if (t == 0) {
        __threadfence();
        if (atomicAdd(A.ticket + 1, 1) == (int)gridDim.x - 1) {
            A.ticket[0] = 0;
            A.ticket[1] = 0;
        }
    }
}

__device__ __forceinline__ double bs_store_value(const double *s, int p) { return s[p]; }
__device__ __forceinline__ float bs_store_value(const float *s, int p) { return s[p]; }
__device__ __forceinline__ float bs_store_value(const uint16_t *s, int p) { return __uint_as_float((unsigned)s[p] << 16); }

struct BsPackArgs {
    int nchunks, lower, rev, nonunit;
    const int4 *chunk, *step, *pk;
    const int *pntr, *diag;
    const double *piv;
    unsigned char *packets;
    const int4 *blk;
    void *mail;
};

// The packet buffer from the plan: a warp per chunk writes its header, its step's first pieces, the
// value pieces (from the pattern's positions) and the rows of the step that it names.
template <typename V, typename X>
__global__ void __launch_bounds__(256) bs_pack_kernel(BsPackArgs A, const V *__restrict__ vals) {
    const int lane = threadIdx.x & 31, np = bs_np(sizeof(X), A.nonunit);
    for (int c = blockIdx.x * 8 + (threadIdx.x >> 5); c < A.nchunks; c += gridDim.x * 8) {
        const int4 ch = __ldg(A.chunk + c), st = __ldg(A.step + ch.y);
        const int rb = ch.w, cnt = st.y & 0xFF;
        int4 sa = make_int4(0, 0, 0, 0);
        if (st.z >= 0) sa = __ldg(A.step + st.z);
        const int cnta = sa.y & 0xFF;
        int4 *at = (int4 *)(A.packets + (size_t)ch.x * 16);
        if (lane == 0) *at = make_int4(st.y, cnta, ch.z, 0);
        at++;
        if (lane < cnt) {
            const int4 p = __ldg(A.pk + st.x + lane);
            const int row = rb + (p.z & 0xFFFF), d = __ldg(A.diag + row);
            const int a = A.lower ? __ldg(A.pntr + row) : d + 1, e = A.lower ? d : __ldg(A.pntr + row + 1);
            X v[3] = {X(0), X(0), X(0)};
            if (!(p.w & kBsExt))
                for (int k = 0; k < 3 && k < e - a; k++) v[k] = bs_store_value(vals, A.rev ? e - 1 - k : a + k);
            at[lane] = p;
            if (p.w & kBsMail)   // the entry that this row mails to waits for it
                ((X *)A.mail)[(long)__ldg(A.blk + 4 * (st.w + (p.w & 0xFF)) + 1).z * (16 / (int)sizeof(X)) + ((unsigned)p.z >> 16)] =
                    Pending<X>::value();
            if constexpr (sizeof(X) == 8) {
                const double dv = !A.nonunit ? 1.0 : (A.piv ? A.piv[row] : bs_store_value(vals, d));
                const bool fast = bs_markstein_range(((unsigned)__double2hiint(dv) >> 20) & 0x7FFu);
                ((double2 *)at)[cnt + lane] = make_double2(v[0], v[1]);
                ((double2 *)at)[2 * cnt + lane] = make_double2(v[2], fast ? 1.0 / dv : 0.0);   // correctly rounded
                if (A.nonunit) ((double2 *)at)[3 * cnt + lane] = make_double2(dv, 0.0);
            } else {
                const float dv = !A.nonunit ? 1.0f : (A.piv ? (float)(1.0 / A.piv[row]) : bs_store_value(vals, d));
                ((float4 *)at)[cnt + lane] = make_float4(v[0], v[1], v[2], dv);
            }
        }
        unsigned short *ra = (unsigned short *)(at + cnt * np);
        if (lane < cnta) ra[lane] = (unsigned short)(__ldg(A.pk + sa.x + lane).z & 0xFFFF);
    }
}

template <typename V, typename X>
__global__ void bs_gather_kernel(long n, const int *__restrict__ map, const V *__restrict__ src, X *__restrict__ dst) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const int m = map[i];
        dst[i] = (m >= 0) ? bs_store_value(src, m) : X(0);
    }
}

// mailboxes: all void at first; after a launch that failed, every entry that is not void pending again
template <typename X>
__global__ void bs_mail_kernel(long n, X *mail, int init) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        if (init) mail[i] = BsVoid<X>::value();
        else if (!BsVoid<X>::is(mail[i])) mail[i] = Pending<X>::value();
    }
}
static int bs_mail(hgb_ctx *c, const BlockSolve &S, int init) {
    if (S.mail_n == 0) return HGB_OK;
    const int g = (int)std::max<long>(1, std::min<long>((S.mail_n + 255) / 256, c->num_sms * 8));
    if (S.xsize == 8) bs_mail_kernel<double><<<g, 256, 0, c->stream>>>(S.mail_n, (double *)S.mail, init);
    else bs_mail_kernel<float><<<g, 256, 0, c->stream>>>(S.mail_n, (float *)S.mail, init);
    return launch_check("bs_mail_kernel");
}

void BlockSolve::release() {
    cudaFree(base);
    *this = BlockSolve();
}

// Co-resident thread-block clusters of cl sweep CTAs (queried once per device, element size and
// cluster size, with the largest shared memory).  One CTA per SM fits.
static int bs_clusters_fit(hgb_ctx *c, int cl, int xsize) {
    static int cache[64][2][kBsMaxCluster + 1];
    static bool init[64][2][kBsMaxCluster + 1];
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    const int xi = xsize == 8;
    if (c->device < 0 || c->device >= 64 || cl < 1 || cl > kBsMaxCluster) return 0;
    if (init[c->device][xi][cl]) return cache[c->device][xi][cl];
    auto fits = [&](auto kernel) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBsSmemMax) != cudaSuccess ||
            (cl > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
            cudaGetLastError();
            return 0;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(cl * 16);
        cfg.blockDim = dim3(kBsThreads);
        cfg.dynamicSmemBytes = kBsSmemMax;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cl;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return n;
    };
    DeviceGuard g(c->device);
    const int n = xi ? fits(bsolve_kernel<double, 0, BS_DIV, true, true>) : fits(bsolve_kernel<float, 0, BS_DIV, false, true>);
    cache[c->device][xi][cl] = n;
    init[c->device][xi][cl] = true;
    return n;
}

// Cluster size.  Every hop between clusters goes through L2 and the mail warps, a hop inside a
// cluster through distributed shared memory; and a block whose cluster is not co-resident starts
// only when another cluster has finished all its blocks.  So: the largest size (up to 16, sizes
// above 8 being non-portable) at which the clusters of all nblk blocks are co-resident; failing
// that, the largest of 8, 4, 2 that fits.
static int bs_cluster_plan(hgb_ctx *c, int nblk, int xsize) {
    if (nblk < 2) return 1;
    for (int cl = std::min(kBsMaxCluster, nblk); cl > 1; cl--)
        if ((long)bs_clusters_fit(c, cl, xsize) * cl >= nblk) return cl;
    for (int cl = 8; cl > 1; cl /= 2)
        if (bs_clusters_fit(c, cl, xsize) >= 1) return cl;
    return 1;
}

int bsolve_plan_pair(hgb_ctx *c, int n, int nnz, const int *pntr, const int *indx, const int *diag, int nonunit_a,
                     int nonunit_b, int rev_b, int xsize, BsPlanPair **out) {
    (void)nnz;
    *out = nullptr;
    BsPlanPair *P = nullptr;
    try {
        P = new BsPlanPair();
        const BsSweepKind kind[2] = {{1, 0, nonunit_a}, {0, rev_b, nonunit_b}};
        BsPlan *plan[2] = {&P->A, &P->B};
        const int st = bs_plan_sweeps(n, pntr, indx, diag, xsize, [&](int nblk) { return bs_cluster_plan(c, nblk, xsize); }, 2,
                                      kind, plan);
        if (st) {
            delete P;
            return st;
        }
    } catch (const std::exception &e) {
        delete P;
        return fail(HGB_ERR_ALLOC, "triangular plan: %s", e.what());
    }
    *out = P;
    return HGB_OK;
}

void bsolve_plan_pair_free(BsPlanPair *P) { delete P; }

// parts of one device allocation, each on a 256-byte boundary
struct BsParts {
    size_t total = 0;
    size_t add(size_t bytes) {
        const size_t at = total;
        total += (bytes + 255) & ~(size_t)255;
        return at;
    }
};
template <typename A>
static int upload(hgb_ctx *c, void *dst, const A &src) {
    if (!src.empty()) HGB_CUDA(cudaMemcpyAsync(dst, src.data(), sizeof(*src.data()) * src.size(), cudaMemcpyHostToDevice, c->stream));
    return HGB_OK;
}

template <typename V, typename X>
static int bs_pack(hgb_ctx *c, const BsPackArgs &A, const void *svals, long next, const int *ext_map, void *ext_vals) {
    const int g = std::max(1, std::min((A.nchunks + 7) / 8, c->num_sms * 8));
    bs_pack_kernel<V, X><<<g, 256, 0, c->stream>>>(A, (const V *)svals);
    if (next) {
        const int ge = (int)std::max<long>(1, std::min<long>((next + 255) / 256, c->num_sms * 8));
        bs_gather_kernel<V, X><<<ge, 256, 0, c->stream>>>(next, ext_map, (const V *)svals, (X *)ext_vals);
    }
    return launch_check("bs_pack_kernel");
}

int bsolve_load(hgb_ctx *c, const BsPlan &P, BlockSolve &S, const int *pntr, const int *diag, const void *svals,
                int vsize, const double *piv) {
    S.release();
    S.n = P.n;
    S.nblk = P.nblk;
    S.cl = P.cl;
    S.nslots = P.nslots;
    S.nflag = P.nflag;
    S.xsize = P.xsize;
    S.nonunit = P.nonunit;
    S.deep = P.deep;
    S.ext = !P.ext_map.empty();
    S.dv_recip = (piv != nullptr && P.xsize == 4) ? 1 : 0;
    BsParts dev, tmp;   // what stays, and what only the packing needs
    const size_t o_blk = dev.add(sizeof(int4) * P.blk.size()), o_strip = dev.add(sizeof(int4) * P.strip.size()),
                 o_watch = dev.add(sizeof(int2) * P.watch.size()), o_codes = dev.add(sizeof(int) * P.ext_codes.size()),
                 o_vals = dev.add((size_t)P.xsize * P.ext_map.size()), o_pack = dev.add((size_t)P.units * 16),
                 o_mail = dev.add((size_t)P.mail_units * 16), o_ticket = dev.add(sizeof(int) * 2);
    const size_t t_chunk = tmp.add(sizeof(int4) * P.chunk.size()), t_step = tmp.add(sizeof(int4) * P.step.size()),
                 t_pk = tmp.add(sizeof(int4) * P.pk.size()), t_map = tmp.add(sizeof(int) * P.ext_map.size());
    HGB_CUDA(cudaMalloc(&S.base, dev.total));
    S.blk = (int4 *)(S.base + o_blk);
    S.strip = (int4 *)(S.base + o_strip);
    S.watch = (int2 *)(S.base + o_watch);
    S.ext_codes = (int *)(S.base + o_codes);
    S.ext_vals = S.base + o_vals;
    S.packets = S.base + o_pack;
    S.mail = S.base + o_mail;
    S.ticket = (int *)(S.base + o_ticket);
    S.mail_n = P.mail_units * (16 / P.xsize);
    S.mail_epoch = c->error_epoch;
    unsigned char *w = nullptr;
    if (ws_alloc(c, &w, tmp.total)) return cuda_fail(cudaErrorMemoryAllocation, "triangular plan");
    auto load = [&]() -> int {
        HGB_TRY(upload(c, w + t_chunk, P.chunk));
        HGB_TRY(upload(c, w + t_step, P.step));
        HGB_TRY(upload(c, w + t_pk, P.pk));
        HGB_TRY(upload(c, w + t_map, P.ext_map));
        HGB_TRY(upload(c, S.blk, P.blk));
        HGB_TRY(upload(c, S.strip, P.strip));
        HGB_TRY(upload(c, S.watch, P.watch));
        HGB_TRY(upload(c, S.ext_codes, P.ext_codes));
        HGB_CUDA(cudaMemsetAsync(S.ticket, 0, sizeof(int) * 2, c->stream));
        HGB_TRY(bs_mail(c, S, 1));
        const BsPackArgs A{(int)P.chunk.size(), P.lower, P.rev, P.nonunit, (int4 *)(w + t_chunk), (int4 *)(w + t_step),
                           (int4 *)(w + t_pk), pntr, diag, piv, S.packets, S.blk, S.mail};
        const long next = (long)P.ext_map.size();
        const int *ext_map = (const int *)(w + t_map);
        if (vsize == 8) return bs_pack<double, double>(c, A, svals, next, ext_map, S.ext_vals);
        if (vsize == 4) return bs_pack<float, float>(c, A, svals, next, ext_map, S.ext_vals);
        return bs_pack<uint16_t, float>(c, A, svals, next, ext_map, S.ext_vals);
    };
    const int st = load();
    ws_free(c, w);
    return st;
}

template <typename X, int MODE, int DIAG, bool LOOK, bool EXT>
static int bs_launch_form(hgb_ctx *c, const BlockSolve &S, const BsArgs &A, X alpha, const X *in, X *out, X *pend) {
    constexpr int XS = sizeof(X), CTA = kBsThreads;
    const size_t smem = bs_ring_bytes(XS, DIAG != BS_UNIT) + (size_t)S.nslots * XS;
    if (smem > (size_t)kBsSmemMax) return fail(HGB_ERR_UNSUPPORTED, "bsolve: %d slots per block", S.nslots);
    auto kernel = bsolve_kernel<X, MODE, DIAG, LOOK, EXT>;
    // per device: the kernel's attributes; per (device, cluster size, shared memory): how many clusters
    // are co-resident
    struct FitKey { int dev, cl; size_t smem; int n; };
    static std::vector<FitKey> fit_cache;
    static bool attr_set[64];
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    if (c->device < 0 || c->device >= 64) return fail(HGB_ERR_UNSUPPORTED, "bsolve: device ordinal %d", c->device);
    if (!attr_set[c->device]) {
        HGB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBsSmemMax));
        // clusters above 8 CTAs are planned only where the occupancy query accepted them with this
        // attribute set; a refusal here leaves the portable sizes working
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
            cudaGetLastError();
        attr_set[c->device] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = S.cl;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(CTA);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters_max = 0;
    for (const FitKey &k : fit_cache)
        if (k.dev == c->device && k.cl == S.cl && k.smem == smem) clusters_max = k.n;
    if (clusters_max == 0) {
        cfg.gridDim = dim3(S.cl * 16);
        HGB_CUDA(cudaOccupancyMaxActiveClusters(&clusters_max, kernel, &cfg));
        if (clusters_max < 1) return fail(HGB_ERR_UNSUPPORTED, "bsolve: no cluster of %d CTAs fits", S.cl);
        fit_cache.push_back(FitKey{c->device, S.cl, smem, clusters_max});
    }
    const int runs = (S.nblk + S.cl - 1) / S.cl;
    cfg.gridDim = dim3(S.cl * std::max(1, std::min(runs, clusters_max)));
    HGB_CUDA(cudaLaunchKernelEx(&cfg, kernel, A, alpha, in, out, pend));
    return launch_check("bsolve_kernel");
}

template <typename X, int MODE, int DIAG>
static int bs_launch_one(hgb_ctx *c, const BlockSolve &S, const BsArgs &A, X alpha, const X *in, X *out, X *pend) {
    if constexpr (sizeof(X) == 4)
        if (S.deep)
            return S.ext ? bs_launch_form<X, MODE, DIAG, false, true>(c, S, A, alpha, in, out, pend)
                         : bs_launch_form<X, MODE, DIAG, false, false>(c, S, A, alpha, in, out, pend);
    return S.ext ? bs_launch_form<X, MODE, DIAG, true, true>(c, S, A, alpha, in, out, pend)
                 : bs_launch_form<X, MODE, DIAG, true, false>(c, S, A, alpha, in, out, pend);
}

template <typename X>
int bsolve_launch(hgb_ctx *c, BlockSolve &S, int mode, X alpha, const X *in, X *out, X *pend, const int *skip) {
    if (S.n == 0) return HGB_OK;
    if (S.mail_epoch != c->error_epoch) {   // an earlier launch failed: it may have left mail behind
        HGB_TRY(bs_mail(c, S, 0));
        S.mail_epoch = c->error_epoch;
    }
    if (S.xsize != (int)sizeof(X) || !S.packets) return fail(HGB_ERR_ARG, "bsolve: values not loaded for this store");
    const BsArgs A{S.nblk, S.cl, S.nflag, S.blk, S.strip, S.packets, S.watch, S.mail, S.ext_codes, S.ext_vals, S.ticket, c->err, skip};
    const int diag = !S.nonunit ? BS_UNIT : (S.dv_recip ? BS_RECIP : BS_DIV);
    if (diag == BS_UNIT)
        return mode == 0 ? bs_launch_one<X, 0, BS_UNIT>(c, S, A, alpha, in, out, pend)
                         : bs_launch_one<X, 1, BS_UNIT>(c, S, A, alpha, in, out, pend);
    if constexpr (sizeof(X) == 4)
        if (diag == BS_RECIP)
            return mode == 0 ? bs_launch_one<X, 0, BS_RECIP>(c, S, A, alpha, in, out, pend)
                             : bs_launch_one<X, 1, BS_RECIP>(c, S, A, alpha, in, out, pend);
    return mode == 0 ? bs_launch_one<X, 0, BS_DIV>(c, S, A, alpha, in, out, pend)
                     : bs_launch_one<X, 1, BS_DIV>(c, S, A, alpha, in, out, pend);
}

template int bsolve_launch<double>(hgb_ctx *, BlockSolve &, int, double, const double *, double *, double *, const int *);
template int bsolve_launch<float>(hgb_ctx *, BlockSolve &, int, float, const float *, float *, float *, const int *);

}  // namespace hgb
