// Strip-scheduled triangular solve (hgb_bsolve.cu): the plan of one sweep and its entry points.
#pragma once

#include "hgb_internal.cuh"

#include <functional>
#include <memory>
#include <vector>

namespace hgb {

// Shape of the sweep kernel per solution type (xsize bytes).  A CTA solves up to kBsW strips at a time;
// the steps of a strip go round kBsK warps, so that a warp has kBsK step times for the part of a
// step that does not wait for the step before.  A mail warp per strip brings in
// values from other clusters.  (20 warps in all: a 21st would take the registers of four.)  Each solver warp has a ring of D
// packet chunks (a chunk is one step) and loads right-hand sides RA of its steps ahead: (D - 1) kBsK
// and RA kBsK steps of about 150 (FP32) or 400 (FP64) cycles against an L2 latency of 700.
constexpr int kBsW = 4, kBsK = 4;
constexpr int kBsThreads = 32 * (kBsW * kBsK + kBsW);
__host__ __device__ constexpr int bs_d(int xsize) { return xsize == 8 ? 2 : 4; }
__host__ __device__ constexpr int bs_ra(int xsize) { return xsize == 8 ? 1 : 3; }
// 16-byte pieces of a packet: the row's codes, then the values and the diagonal terms
__host__ __device__ constexpr int bs_np(int xsize, int nonunit) { return xsize == 8 ? (nonunit ? 4 : 3) : 2; }
__host__ __device__ constexpr int bs_chunk_bytes(int xsize, int nonunit) { return 16 + 32 * bs_np(xsize, nonunit) * 16 + 64; }
// shared memory besides the value slots: the packet rings and the right-hand-side rings
__host__ __device__ constexpr int bs_ring_bytes(int xsize, int nonunit) {
    return kBsW * kBsK * (bs_d(xsize) * bs_chunk_bytes(xsize, nonunit) + bs_ra(xsize) * 32 * xsize);
}
constexpr int kBsSmemMax = 227 * 1024 - 1024;   // of one CTA; 1 KB for the kernel's static shared memory
__host__ __device__ constexpr int bs_slots_max(int xsize, int nonunit) {
    return (kBsSmemMax - bs_ring_bytes(xsize, nonunit)) / xsize;
}
constexpr int kBsNoSlot = 0xFFFF;
constexpr int kBsMaxStrip = 16384;   // rows of a strip (the packets count them in 16 bits)
// packet flags (first piece, .w): bits 0-7 blocks to the one whose slot (first piece, .z, high half) takes
// the row's value, in shared memory (push) or through its mailbox (mail)
constexpr int kBsExt = 1 << 8, kBsReset = 1 << 9, kBsPush = 1 << 10;
constexpr int kBsMail = 1 << 14;
constexpr int kBsFar = 1 << 11;   // << k: entry k comes from another strip or block
// step flags (bits 8.. of a step's word, after its rows): some row lists its entries in the ext
// arrays; entry 0 / entry 2 of every other row is far (or padding); no row has an entry 2
constexpr int kBsStepExt = 1 << 8, kBsEarly0 = 1 << 9, kBsEarly2 = 1 << 10, kBsNo2 = 1 << 11;

// A host array whose elements start undefined: the pages of a large one are first touched by the threads
// that fill it.
template <typename T>
struct BsArray {
    std::unique_ptr<T[]> p;
    size_t count = 0;
    void resize(size_t n) {
        p.reset(new T[n]);
        count = n;
    }
    T *data() { return p.get(); }
    const T *data() const { return p.get(); }
    size_t size() const { return count; }
    bool empty() const { return count == 0; }
    T &operator[](size_t i) { return p[i]; }
    const T &operator[](size_t i) const { return p[i]; }
};

// The schedule of one sweep as the host plans it (structure only).
struct BsPlan {
    // deep: the pattern of a 3D grid (hgb_bsplan.cu)
    int n = 0, nblk = 0, cl = 1, nslots = 0, nflag = 0, nonunit = 0, lower = 1, rev = 0, xsize = 8, deep = 0;
    long units = 0;                 // 16-byte units of the packet buffer
    long path = 0;                  // length of the sweep in steps, hand-overs included (hgb_bsplan.cu)
    int levels = 0;                 // levels of the strip with the most: the pattern has no fewer
    std::vector<int4> blk;          // [4 nblk] {first strip, strips, flagged slots, slots} {first watch, watches, mailbox or
                                    // -1, 0} {per strip: first and end mail unit}; units of 16 bytes
    long mail_units = 0;
    std::vector<int4> strip;        // [2 kBsK nstrips], per warp of a strip: {lowest row, steps of the strip, first
                                    // unit, 0} {units of its first chunks, 16 bits each}
    std::vector<int4> chunk;        // [steps], warp by warp: {first unit, step, units of the chunk D ahead, lowest row}
    std::vector<int4> step;         // [steps] {first packet, rows | flags, step whose rows it names or -1, block}
    BsArray<int4> pk;               // [packets] the first piece of every packet
    std::vector<int2> watch;        // {global row, slot}, by block in the order of their first use
    std::vector<int> ext_codes, ext_map;
    BsArray<int> pk_of_row;     // packet of every row
    std::vector<unsigned char> watched;   // rows that other blocks read through memory
};

// The two sweeps of one preconditioner: A the lower triangle (ascending rows), B the upper one.
struct BsPlanPair {
    BsPlan A, B;
};

// Device copy of a plan with the values in the packets.
struct BlockSolve {
    int n = 0, nblk = 0, cl = 1, nslots = 0, nflag = 0, xsize = 8, nonunit = 0, dv_recip = 0, deep = 0, ext = 0;
    unsigned char *base = nullptr;   // the one allocation that holds all of the below
    int4 *blk = nullptr, *strip = nullptr;
    unsigned char *packets = nullptr;
    int2 *watch = nullptr;
    void *mail = nullptr;           // mailboxes of the blocks that read values from other clusters
    long mail_n = 0;                // their elements
    unsigned mail_epoch = 0;        // context error epoch at their last reset
    int *ext_codes = nullptr;
    void *ext_vals = nullptr;
    int *ticket = nullptr;
    void release();
};

// Sweeps of one pattern, planned together; the two of a pair (two sweeps) reset each other's watched
// entries.  lower: ascending rows; cluster_of(blocks): CTAs per thread-block cluster.
struct BsSweepKind {
    int lower, rev, nonunit;
};
int bs_plan_sweeps(int n, const int *pntr, const int *indx, const int *diag, int xsize, const std::function<int(int)> &cluster_of,
                   int sweeps, const BsSweepKind *kind, BsPlan **plan);
// Plans both sweeps from HOST arrays.  nonunit_a / nonunit_b: the sweep divides by its diagonal;
// rev_b: the upper sweep visits a row's entries in descending column order.  xsize: bytes of a
// solution element (8 or 4).
int bsolve_plan_pair(hgb_ctx *c, int n, int nnz, const int *pntr, const int *indx, const int *diag, int nonunit_a,
                     int nonunit_b, int rev_b, int xsize, BsPlanPair **out);
// Uploads a plan and packs the values (store precision vsize; piv: FP64 pivots of a lower-precision
// store, whose reciprocals the packets carry).  pntr, diag: device arrays of the planned pattern.
int bsolve_load(hgb_ctx *c, const BsPlan &P, BlockSolve &S, const int *pntr, const int *diag, const void *svals,
                int vsize, const double *piv);
void bsolve_plan_pair_free(BsPlanPair *P);
// out = op(in).  pend: the buffer whose entries, where the pair's other sweep watches them, go back
// to the pending pattern.  It may be in.
template <typename X>
int bsolve_launch(hgb_ctx *c, BlockSolve &S, int mode, X alpha, const X *in, X *out, X *pend, const int *skip);

}  // namespace hgb
