// The host's plan of a strip-scheduled triangular sweep (hgb_bsolve.cu runs it).
//
// Rows are cut, in solve order, into strips (kBsK warps solve a strip, its steps in turn) and runs of up to kBsW strips
// into blocks (one CTA).  Inside a strip the rows are grouped by their level over the dependencies that stay in
// the strip, each level cut into steps of at most 32 rows, one row per lane.  Every value that a
// block's rows read has a slot in the CTA's shared memory:
//  - slot 0 holds 0 (the padding of rows with fewer than three entries);
//  - flagged slots hold the pending pattern until their value arrives: rows of this block that other
//    strips of it read, and the distinct rows of earlier blocks (the halo), numbered in the order
//    of their first use, so that the lanes of a step read consecutive slots;
//  - the other rows take a slot of their strip from their step to their last use in the strip (a
//    free list in first-in first-out order), so a strip needs a few dozen of them.
// A halo slot is filled by the CTA that solves the row: straight, if that CTA is in the same
// thread-block cluster (push), else through the block's mailbox, an array in memory with an entry per
// slot, which the block's mail warps poll (mail).  A row has one such target; another block that needs
// it polls the solution itself (a watched row).  Rows with more than three entries, and rows of which an entry
// found no halo slot, list their entries in the ext arrays (a negative code polls the solution).
//
// The blocks are planned in parallel host threads; the result does not depend on their number.
#include "hgb_internal.cuh"
#include "hgb_bsolve.cuh"

#include <algorithm>
#include <atomic>
#include <climits>
#include <exception>
#include <functional>
#include <mutex>
#include <thread>

namespace hgb {

// The host threads of one planning call: started once, they take the items of every phase in turn (a
// start costs more than a phase of a small matrix).
class HostTeam {
    std::vector<std::thread> th;
    std::function<void(int)> work;
    std::atomic<int> next{0}, items{0}, busy{0}, phase{0};
    std::exception_ptr failed;
    std::mutex mu;
    void take() {
        try {
            for (int i; (i = next.fetch_add(1)) < items.load();) work(i);
        } catch (...) {
            next = INT_MAX / 2;
            std::lock_guard<std::mutex> lock(mu);
            failed = std::current_exception();
        }
    }

  public:
    explicit HostTeam(long rows) {
        const int nt = (int)std::min<long>({(long)std::thread::hardware_concurrency(), 16L, rows / 16384 + 1});
        try {
            for (int k = 1; k < nt; k++)
                th.emplace_back([this] {
                    for (int seen = 0;;) {
                        int p;
                        while ((p = phase.load()) == seen) std::this_thread::yield();
                        if (p < 0) return;
                        seen = p;
                        take();
                        busy.fetch_sub(1);
                    }
                });
        } catch (const std::exception &) {   // no more threads, or no memory for them: those that run take the work
        }
    }
    ~HostTeam() {
        phase = -1;
        for (auto &t : th) t.join();
    }
    // f(0) .. f(n - 1), in any order and thread
    void run(int n, std::function<void(int)> f) {
        work = std::move(f);
        next = 0;
        items = n;
        busy = (int)th.size();
        phase.fetch_add(1);
        take();
        while (busy.load()) std::this_thread::yield();
        if (failed) std::rethrow_exception(failed);
    }
};

namespace {

struct Rows {   // a row's strictly lower / upper entries, in solve order of the rows
    int n, lower;
    const int *pntr, *indx, *diag;
    int row_of(int pos) const { return lower ? pos : n - 1 - pos; }
    int pos_of(int row) const { return lower ? row : n - 1 - row; }
    void deps(int row, int &a, int &e) const {
        a = lower ? pntr[row] : diag[row] + 1;
        e = lower ? diag[row] : pntr[row + 1];
    }
};

struct Halo {
    int row, slot, key;
};
struct Use {   // a step (a sample of them) that reads a row of an earlier block, and its begin on its strip's clock
    int row, strip, begin;
};
struct Lag {
    int strip, offset;   // a strip starts at least so long after that one
};

struct BlockOut {
    int nflag = 0, nslots = 0, seg[kBsW + 1] = {};   // seg: first halo slot of every strip
    long units = 0;
    std::vector<int4> strip, chunk, step;
    std::vector<int> ext_codes, ext_map, direct;
    std::vector<Halo> halo;
    std::vector<Use> use;             // by strip
    int span[kBsW] = {};              // the strips' clocks at their ends
    int late[kBsW][kBsW];             // of strip k behind strip s of the block (INT_MIN: does not read it)
    int levels = 0;                   // of its strip with the most
};

struct Scratch {   // one thread's working arrays
    std::vector<int> lev, cnt, start, order, step_of, last, flag, tslot, next, head, time, clock, window, touched;
    std::vector<int> strip_steps, step_base, free_q;
};

}  // namespace

// Strip length.  The rows of a strip's steps should fill a warp: 32 grid lines of the pattern.  The
// line is read off the entries' distances: the largest one at most half the bandwidth (the
// second stride of a 3D grid), or the bandwidth itself where that is the stride of a 2D grid.
// Where the bandwidth is a whole number of lines (a grid plane), strips are cut evenly inside it, so
// that every plane has the same ones: strips of several planes and a part run up to twice as long (15 x 13 x 13:
// 87 steps against 54; planes of fewer than ten lines leave a strip's steps too few rows: 96 x 8 x 40 153 against
// 190).  No strip has more than kBsMaxStrip rows: a packet holds its row's place in the strip in 16 bits, and a
// strip's own rows have to fit the slots.
static void bs_strips(int n, int bw, int d2, std::vector<int> &cut, int &T, bool &deep) {
    constexpr int kMaxT = kBsMaxStrip, kMinT = 512, kMinLines = 10;
    deep = d2 >= 8;
    const int u = deep ? d2 : std::max(bw, 1);
    cut.assign(1, 0);
    if (bw == 0) {
        T = 4096;
    } else {
        T = u > kMaxT ? kMaxT : (int)std::min<long>(32L * u, (long)(kMaxT / u) * u);
        if (T < kMinT) T = (kMinT + T - 1) / T * T;
        if (deep && u <= kMaxT && bw % u == 0 && bw / u >= kMinLines && bw <= n) {
            const int ny = bw / u, k = (bw + T - 1) / T, lines = (ny + k - 1) / k;
            T = lines * u;
            for (long p = 0; p < n; p += bw)
                for (int l = 0; l < ny; l += lines) {
                    const long e = p + (long)std::min(ny, l + lines) * u;
                    if (cut.back() < n) cut.push_back((int)std::min<long>(e, n));
                }
            return;
        }
    }
    for (long p = T; p < n; p += T) cut.push_back((int)p);
    cut.push_back(n);
}

// Clock of the plan, in steps of rows of up to three entries (0.14 us in FP32, 0.35 in FP64): a step with rows of kx entries in
// the ext arrays (0.17 us an entry, 0.2) ...
static int bs_step_cost(int xsize, int kx) { return kx == 0 ? 1 : (xsize == 8 ? 1 + (4 * kx + 3) / 7 : 1 + (6 * kx + 4) / 5); }
// ... and a hand-over inside a cluster, and across
static int bs_hop_cost(int xsize, bool near) { return xsize == 8 ? (near ? 1 : 4) : (near ? 2 : 9); }
constexpr int kPathSample = 16;   // every so many steps of a strip are looked at for the strips that it waits for

// One block: its strips' steps, slots, chunks and packets (into pk from position P0 on).  Where the block's own
// rows take more than cap slots, only B.nslots is set.
static void bs_plan_block(const Rows &R, int rev, int np, int xsize, int cap, int bw, const int *cut, int s0, int s1,
                          int4 *pk, int *pk_of_row, int *done, BlockOut &B, Scratch &S) {
    const int P0 = cut[s0], P1 = cut[s1], rows = P1 - P0, ns = s1 - s0;
    const int RA = bs_ra(xsize), D = bs_d(xsize);
    S.lev.resize(rows);
    S.order.resize(rows);
    S.step_of.resize(rows);
    S.last.assign(rows, -1);
    S.flag.assign(rows, 0);
    S.tslot.assign(rows, -1);
    S.strip_steps.assign(ns + 1, 0);
    S.step_base.clear();   // first row (in order) of every step, over the block's strips
    // ---- levels and steps of every strip
    for (int k = 0; k < ns; k++) {
        const int p0 = cut[s0 + k], p1 = cut[s0 + k + 1], o = p0 - P0;
        S.cnt.clear();
        for (int p = p0; p < p1; p++) {
            int a, e, lv = 0;
            R.deps(R.row_of(p), a, e);
            for (int q = a; q < e; q++) {
                const int pj = R.pos_of(R.indx[q]);
                if (pj >= p0) lv = std::max(lv, S.lev[pj - P0] + 1);
            }
            S.lev[p - P0] = lv;
            if ((int)S.cnt.size() <= lv) S.cnt.resize(lv + 1, 0);
            S.cnt[lv]++;
        }
        const int nl = (int)S.cnt.size();
        B.levels = std::max(B.levels, nl);
        S.start.assign(nl + 1, 0);
        for (int l = 0; l < nl; l++) S.start[l + 1] = S.start[l] + S.cnt[l];
        int steps = 0;
        S.head.assign(nl, 0);   // first step of a level
        for (int l = 0; l < nl; l++) {
            S.head[l] = steps;
            for (int q = 0; q < S.cnt[l]; q += 32, steps++) S.step_base.push_back(o + S.start[l] + q);
        }
        S.cnt.assign(S.start.begin(), S.start.end() - 1);
        for (int p = p0; p < p1; p++) {
            const int l = S.lev[p - P0], at = S.cnt[l]++;
            S.order[o + at] = p;
            S.step_of[p - P0] = S.head[l] + (at - S.start[l]) / 32;
        }
        S.strip_steps[k + 1] = S.strip_steps[k] + steps;
    }
    S.step_base.push_back(rows);
    const int nsteps = S.strip_steps[ns];
    // a step ends where the next one begins, also at the end of a strip: the rows of a strip's last
    // step reach to the next strip's first row
    auto step_rows = [&](int st) { return S.step_base[st + 1] - S.step_base[st]; };
    // ---- who reads what inside the block
    for (int k = 0; k < ns; k++) {
        const int p0 = cut[s0 + k], p1 = cut[s0 + k + 1];
        for (int p = p0; p < p1; p++) {
            int a, e;
            R.deps(R.row_of(p), a, e);
            for (int q = a; q < e; q++) {
                const int pj = R.pos_of(R.indx[q]);
                if (pj >= p0) S.last[pj - P0] = std::max(S.last[pj - P0], S.step_of[p - P0]);
                else if (pj >= P0) S.flag[pj - P0] = 1;
            }
        }
    }
    // ---- flagged rows of the block in the order of their steps, then the strips' own slots
    int nf = 0, ntemp = 0;
    for (int q = 0; q < rows; q++) {
        const int r = S.order[q] - P0;
        if (S.flag[r]) S.flag[r] = ++nf;
    }
    for (int k = 0; k < ns; k++) {
        S.next.resize(rows);
        const int f = S.strip_steps[k], steps = S.strip_steps[k + 1] - f;
        S.head.assign(steps, -1);   // rows by the step of their last use
        S.free_q.clear();
        size_t fq = 0;
        for (int st = 0; st < steps; st++) {
            for (int q = S.step_base[f + st]; q < S.step_base[f + st + 1]; q++) {
                const int r = S.order[q] - P0, lu = S.last[r];
                if (S.flag[r] || lu < 0) continue;
                S.tslot[r] = fq < S.free_q.size() ? S.free_q[fq++] : ntemp++;
            }
            for (int q = S.step_base[f + st + 1] - 1; q >= S.step_base[f + st]; q--) {   // lists in lane order
                const int r = S.order[q] - P0;
                if (S.tslot[r] < 0) continue;
                S.next[r] = S.head[S.last[r]];
                S.head[S.last[r]] = r;
            }
            for (int r = S.head[st]; r >= 0; r = S.next[r]) S.free_q.push_back(S.tslot[r]);
        }
    }
    B.nslots = 1 + nf + ntemp;
    if (B.nslots > cap) return;   // its own rows do not fit: the sweep is cut into smaller blocks
    // ---- the halo in the order of its first use; the steps' times order the fetches
    S.window.resize(std::max<size_t>(S.window.size(), std::min(P0, bw)), 0);   // by distance from the block
    S.touched.clear();
    S.time.assign(nsteps, 0);
    S.clock.assign(nsteps, 0);   // end of every step, on its strip's clock (bs_step_cost)
    std::fill(&B.late[0][0], &B.late[0][0] + kBsW * kBsW, INT_MIN);
    int nh = 0;
    for (int k = 0; k < ns; k++) {
        const int p0 = cut[s0 + k];
        // a strip's halo starts a 16-byte unit of the mailbox: a unit with values of two strips would
        // hold the first values of one until the last ones of the other are in (without room for that, the
        // strip has no halo slots of its own)
        while ((1 + nf + nh) % (16 / xsize) && 1 + nf + nh + ntemp < cap) {
            B.halo.push_back({-1, 1 + nf + nh, INT_MAX});
            nh++;
        }
        B.seg[k] = (1 + nf + nh + 16 / xsize - 1) / (16 / xsize) * (16 / xsize);
        for (int st = S.strip_steps[k]; st < S.strip_steps[k + 1]; st++) {
            int t = st > S.strip_steps[k] ? S.time[st - 1] + 1 : 0, kx = 0;
            const int begin = st > S.strip_steps[k] ? S.clock[st - 1] : 0;
            const bool sample = (st - S.strip_steps[k]) % kPathSample == 0;
            for (int pass = 0; pass < 2; pass++) {   // the step's time, then its halo
                for (int q = S.step_base[st]; q < S.step_base[st + 1]; q++) {
                    int a, e;
                    R.deps(R.row_of(S.order[q]), a, e);
                    bool ext = e - a > 3;
                    for (int i = a; i < e; i++) {
                        const int pj = R.pos_of(R.indx[i]);
                        if (pj >= p0) continue;
                        if (pj >= P0) {
                            if (pass == 0) {
                                int s = 0;
                                while (cut[s0 + s + 1] <= pj) s++;
                                const int from = S.strip_steps[s] + S.step_of[pj - P0];
                                t = std::max(t, S.time[from] + 1);
                                if (sample) B.late[k][s] = std::max(B.late[k][s], S.clock[from] + 1 - begin);
                            }
                        } else if (pass == 1) {
                            int &w = S.window[P0 - 1 - pj];
                            if (w == 0) {
                                S.touched.push_back(P0 - 1 - pj);
                                if (1 + nf + nh + ntemp < cap) {
                                    w = 1 + nf + nh++;
                                    B.halo.push_back({R.indx[i], w, t});
                                } else {
                                    w = -1;
                                    B.direct.push_back(R.indx[i]);
                                }
                            } else if (w > 0) {
                                Halo &h = B.halo[w - 1 - nf];
                                h.key = std::min(h.key, t);
                            }
                            if (sample) B.use.push_back({R.indx[i], k, begin});
                            ext = ext || w < 0;
                        }
                    }
                    if (pass == 1 && ext) kx = std::max(kx, e - a);
                }
                if (pass == 0) S.time[st] = t;
            }
            S.clock[st] = begin + bs_step_cost(xsize, kx);
            for (int q = S.step_base[st]; q < S.step_base[st + 1]; q++) done[S.order[q]] = S.clock[st];
            B.span[k] = S.clock[st];
        }
    }
    for (int k = ns; k <= kBsW; k++) B.seg[k] = (1 + nf + nh + 16 / xsize - 1) / (16 / xsize) * (16 / xsize);
    B.nflag = 1 + nf + nh;
    B.nslots = B.nflag + ntemp;
    auto code_of = [&](int pj) {
        if (pj < P0) return S.window[P0 - 1 - pj];
        const int r = pj - P0;
        return S.flag[r] ? S.flag[r] : B.nflag + S.tslot[r];
    };
    // ---- packets and steps
    for (int k = 0; k < ns; k++) {
        const int p0 = cut[s0 + k], p1 = cut[s0 + k + 1], f = S.strip_steps[k], steps = S.strip_steps[k + 1] - f;
        const int rb = R.lower ? p0 : R.n - p1;
        for (int st = f; st < f + steps; st++) {
            const int nr = step_rows(st), eb = (int)B.ext_codes.size();
            int kx = 0, early0 = kBsEarly0, early2 = kBsEarly2, no2 = kBsNo2;
            for (int i = 0; i < nr; i++) {
                int far = 0;
                const int p = S.order[S.step_base[st] + i], row = R.row_of(p);
                int a, e, cd[3] = {0, 0, 0};
                R.deps(row, a, e);
                bool ext = e - a > 3;
                for (int q = a; q < e && !ext; q++) {
                    const int ix = rev ? e - 1 - (q - a) : q;
                    const int pj = R.pos_of(R.indx[ix]);
                    cd[q - a] = code_of(pj);
                    ext = cd[q - a] < 0;
                    if (pj < p0) far |= kBsFar << (q - a);
                }
                if (ext) {   // column-major over the step's rows: entry q of row i at eb + q * nr + i
                    if (e - a > kx) {
                        kx = e - a;
                        B.ext_codes.resize(eb + (size_t)kx * nr, 0);
                        B.ext_map.resize(eb + (size_t)kx * nr, -1);
                    }
                    for (int q = 0; q < e - a; q++) {
                        const int ix = rev ? e - 1 - q : a + q;
                        const int code = code_of(R.pos_of(R.indx[ix]));
                        B.ext_codes[eb + (size_t)q * nr + i] = code >= 0 ? code : -(R.indx[ix] + 1);
                        B.ext_map[eb + (size_t)q * nr + i] = ix;
                    }
                    cd[0] = (eb + i) & 0xFFFF;
                    cd[1] = (unsigned)(eb + i) >> 16;
                    cd[2] = e - a;
                } else {
                    if (cd[0] && !(far & kBsFar)) early0 = 0;
                    if (cd[2] && !(far & kBsFar << 2)) early2 = 0;
                    if (e - a > 2) no2 = 0;
                }
                const int r = p - P0;
                const int slot = S.flag[r] ? S.flag[r] : (S.tslot[r] >= 0 ? B.nflag + S.tslot[r] : kBsNoSlot);
                const int q = P0 + S.step_base[st] + i;
                pk[q] = make_int4((int)((unsigned)cd[0] | (unsigned)cd[1] << 16), (int)((unsigned)cd[2] | (unsigned)slot << 16),
                                  row - rb, ext ? kBsExt : far);
                pk_of_row[row] = q;
            }
            const int ahead = st - f + RA * kBsK < steps ? st + RA * kBsK : -1;
            B.step.push_back(make_int4(P0 + S.step_base[st], nr | (kx ? kBsStepExt : 0) | early0 | early2 | no2, ahead, 0));
        }
    }
    // ---- chunks, a warp's one after the other
    long unit = 0;
    for (int k = 0; k < ns; k++) {
        const int f = S.strip_steps[k], steps = S.strip_steps[k + 1] - f;
        const int rb = R.lower ? cut[s0 + k] : R.n - cut[s0 + k + 1];
        for (int w = 0; w < kBsK; w++) {
            const int c0 = (int)B.chunk.size();
            B.strip.push_back(make_int4(rb, steps, (int)unit, 0));
            for (int st = f + w; st < f + steps; st += kBsK) {
                const int ahead = B.step[st].z;
                B.chunk.push_back(make_int4((int)unit, st, 0, rb));
                unit += 1 + step_rows(st) * np + (ahead >= 0 ? (step_rows(ahead) * 2 + 15) / 16 : 0);
            }
            const int nch = (int)B.chunk.size() - c0;
            int sz[8] = {0};
            for (int c = 0; c < nch; c++) {
                const int size = (int)((c + 1 < nch ? B.chunk[c0 + c + 1].x : unit) - B.chunk[c0 + c].x);
                if (c < D) sz[c] = size;
                else B.chunk[c0 + c - D].z = size;
            }
            B.strip.push_back(make_int4(sz[0] | sz[1] << 16, sz[2] | sz[3] << 16, sz[4] | sz[5] << 16, sz[6] | sz[7] << 16));
        }
    }
    B.units = unit;
    for (int w : S.touched) S.window[w] = 0;
}

namespace {

// The phases of one sweep's plan
struct Sweep {
    const Rows R;
    const int n, rev, nonunit, xsize, np, cap, ranges;
    BsPlan &P;
    std::vector<int> mx, wide, cut;
    int bw = 0, d2 = 0, T = 0, nstrips = 0, spb = 1, nblk = 0, cl = 1, runs = 0;
    bool deep = false, planned = false;
    std::vector<BlockOut> out;
    std::vector<std::vector<int2>> watch;
    std::vector<std::vector<Halo>> far;   // entries from earlier clusters
    BsArray<int> done;                    // end of the step of every row (by position), on its strip's clock
    std::vector<std::vector<Lag>> lag;    // of every strip, behind strips of earlier blocks
    std::vector<char> mailed;
    struct Base {
        size_t strip, chunk, step, watch, ext;
        long unit, mail;
    };
    std::vector<Base> base;

    Sweep(int n_, const int *pntr, const int *indx, const int *diag, int lower, int rev_, int nonunit_, int xsize_, BsPlan &P_)
        : R{n_, lower, pntr, indx, diag}, n(n_), rev(rev_), nonunit(nonunit_), xsize(xsize_), np(bs_np(xsize_, nonunit_)),
          cap(std::min(kBsNoSlot, bs_slots_max(xsize_, nonunit_))), ranges(std::max(1, std::min(64, n_ / 8192))), P(P_),
          mx(ranges, 0), wide(ranges, -1) {}

    // the largest distance of an entry (limit < 0), or the largest one up to a limit, over a range of rows
    void scan(int k, int limit) {
        int m = 0;
        for (int row = (int)((long)n * k / ranges); row < (int)((long)n * (k + 1) / ranges); row++) {
            int a, e;
            R.deps(row, a, e);
            if (e - a > 0xFFFF) wide[k] = row;
            if (limit < 0) {
                if (e > a) m = std::max(m, R.lower ? row - R.indx[a] : R.indx[e - 1] - row);
            } else {
                for (int q = a; q < e; q++) {
                    const int d = std::abs(row - R.indx[q]);
                    if (d <= limit) m = std::max(m, d);
                }
            }
        }
        mx[k] = m;
    }
    int widest() const { return *std::max_element(mx.begin(), mx.end()); }

    // Strips per block.  Patterns of 3D grids (deep): as many as the CTA has warps and slots: the
    // next strip but few is the same place one plane on, and hand-overs inside a CTA are the cheapest.
    // Others (2D grids): each strip runs a whole strip's width of steps behind the one before it, so
    // hand-overs are few and a CTA's strips only slow one another; one strip per CTA until they
    // no longer fit a cluster of 16 CTAs.
    int cut_blocks(const std::function<int(int)> &cluster_of) {
        bs_strips(n, bw, d2, cut, T, deep);
        nstrips = (int)cut.size() - 1;
        for (int k = 0; k < nstrips; k++)
            if (cut[k + 1] - cut[k] > kBsMaxStrip)
                return fail(HGB_ERR_UNSUPPORTED, "triangular plan: a strip of %d rows", cut[k + 1] - cut[k]);
        const int by_rows = std::max(1, (xsize == 8 ? 20480 : 32768) / T);
        spb = std::min({kBsW, by_rows, deep ? kBsW : std::max(1, (nstrips + 15) / 16)});
        P.pk.resize(n);
        P.pk_of_row.resize(n);
        P.watched.assign(n, 0);
        done.resize(n);
        group(cluster_of);
        return HGB_OK;
    }
    // spb strips to a block
    void group(const std::function<int(int)> &cluster_of) {
        nblk = (nstrips + spb - 1) / spb;
        cl = cluster_of(nblk);
        runs = (nblk + cl - 1) / cl;
        out.assign(nblk, BlockOut());
        watch.resize(nblk);
        far.resize(nblk);
        lag.resize(nstrips);
        mailed.assign(nblk, 0);
    }
    // after the blocks are planned: whether all of them fit.  Where one does not, the sweep takes blocks of
    // half as many strips (one strip fits: kBsMaxStrip rows are fewer than the slots).
    int settle(const std::function<int(int)> &cluster_of) {
        planned = true;
        for (const BlockOut &B : out) planned = planned && B.nslots <= cap;
        if (planned) return HGB_OK;
        if (spb == 1) return fail(HGB_ERR_UNSUPPORTED, "triangular plan: a strip's rows exceed the slots");
        spb /= 2;
        group(cluster_of);
        return HGB_OK;
    }
    void block(int b, Scratch &scr) {
        bs_plan_block(R, rev, np, xsize, cap, bw, cut.data(), b * spb, std::min(nstrips, (b + 1) * spb), P.pk.data(),
                      P.pk_of_row.data(), done.data(), out[b], scr);
    }
    // where the halos of a cluster's blocks come from: inside the cluster they are pushed
    void halos(int run) {
        const int b0 = run * cl, b1 = std::min(nblk, b0 + cl);
        for (int b = b0; b < b1; b++) {
            lags(b, b0);
            for (const Halo &h : out[b].halo) {
                if (h.row < 0) continue;   // padding
                const int pj = R.pos_of(h.row);
                const int pb = strip_of(pj) / spb;
                int4 &k = P.pk[P.pk_of_row[h.row]];
                if (pb >= b0 && !(k.w & kBsPush)) {
                    k.z |= (int)((unsigned)h.slot << 16);
                    k.w |= kBsPush | (b - pb);
                } else {
                    far[b].push_back({h.row, h.slot, h.key << 8 | std::min(b - pb, 255)});
                }
            }
        }
    }
    int strip_of(int pos) const { return (int)(std::upper_bound(cut.begin(), cut.end(), pos) - cut.begin() - 1); }
    // how far the strips of a block start behind those of earlier ones (b0: the first block of its cluster)
    void lags(int b, int b0) {
        std::vector<int> late(b * spb, INT_MIN), seen;   // behind every strip of an earlier block
        const std::vector<Use> &use = out[b].use;
        for (size_t i = 0; i < use.size(); i++) {
            const int pj = R.pos_of(use[i].row), ps = strip_of(pj);
            if (late[ps] == INT_MIN) seen.push_back(ps);
            late[ps] = std::max(late[ps], done[pj] + bs_hop_cost(xsize, ps / spb >= b0) - use[i].begin);
            if (i + 1 < use.size() && use[i + 1].strip == use[i].strip) continue;
            for (int s : seen) {
                lag[b * spb + use[i].strip].push_back({s, late[s]});
                late[s] = INT_MIN;
            }
            seen.clear();
        }
    }
    // the sweep's length on the strips' clocks, each strip running as a whole from the time at which all that it waits
    // for comes no later than it reads it
    void path() {
        std::vector<long> start(nstrips, 0);
        P.path = P.levels = 0;
        for (const BlockOut &B : out) P.levels = std::max(P.levels, B.levels);
        for (int k = 0; k < nstrips; k++) {
            const BlockOut &B = out[k / spb];
            const int first = k / spb * spb;
            for (int s = first; s < k; s++)
                if (B.late[k - first][s - first] != INT_MIN) start[k] = std::max(start[k], start[s] + B.late[k - first][s - first]);
            for (const Lag &l : lag[k]) start[k] = std::max(start[k], start[l.strip] + l.offset);
            P.path = std::max(P.path, start[k] + B.span[k - first]);
        }
    }
    // the rows that push to no block of their own cluster mail to the first block that needs them (in
    // block order: a row's readers in several clusters are told apart by the order of the blocks)
    void mails() {
        for (int b = 0; b < nblk; b++)
            for (Halo &h : far[b]) {
                int4 &k = P.pk[P.pk_of_row[h.row]];
                const int delta = h.key & 255;
                if (!(k.w & (kBsPush | kBsMail)) && delta < 255) {
                    k.z |= (int)((unsigned)h.slot << 16);
                    k.w |= kBsMail | delta;
                    mailed[b] = 1;
                    h.row = -1;
                }
            }
    }
    // the rest is watched: by the time of the first use in windows of 8 steps, by row inside a window, so
    // that the loads touch a few consecutive rows of each grid line instead of one sector per row
    void watches(int b) {
        std::vector<Halo> &f = far[b];
        f.erase(std::remove_if(f.begin(), f.end(), [](const Halo &h) { return h.row < 0; }), f.end());
        for (Halo &h : f) h.key >>= 11;
        std::sort(f.begin(), f.end(), [](const Halo &x, const Halo &y) { return x.key != y.key ? x.key < y.key : x.row < y.row; });
        for (const Halo &h : f) {
            watch[b].push_back(make_int2(h.row, h.slot));
            __atomic_store_n(&P.watched[h.row], (unsigned char)1, __ATOMIC_RELAXED);
        }
        for (int row : out[b].direct) __atomic_store_n(&P.watched[row], (unsigned char)1, __ATOMIC_RELAXED);
    }
    // one set of arrays
    int sizes() {
        const int qe = 16 / xsize;   // elements of a 16-byte unit
        base.assign(nblk + 1, Base{0, 0, 0, 0, 0, 0, 0});
        int nslots = 1, nflag = 1;
        for (int b = 0; b < nblk; b++) {
            const BlockOut &B = out[b];
            base[b + 1] = Base{base[b].strip + B.strip.size(), base[b].chunk + B.chunk.size(), base[b].step + B.step.size(),
                               base[b].watch + watch[b].size(), base[b].ext + B.ext_codes.size(), base[b].unit + B.units,
                               base[b].mail + (mailed[b] ? (B.nflag + qe - 1) / qe : 0)};
            nslots = std::max(nslots, B.nslots);
            nflag = std::max(nflag, B.nflag);
        }
        if (nslots > cap) return fail(HGB_ERR_UNSUPPORTED, "triangular plan: a block needs %d slots of %d", nslots, cap);
        const Base &tot = base[nblk];
        if (tot.unit > INT_MAX || tot.mail > INT_MAX || tot.ext > INT_MAX)
            return fail(HGB_ERR_UNSUPPORTED, "triangular plan: packed arrays exceed 2^31 entries");
        P.blk.resize(4 * (size_t)nblk);
        P.strip.resize(tot.strip);
        P.chunk.resize(tot.chunk);
        P.step.resize(tot.step);
        P.watch.resize(tot.watch);
        P.ext_codes.resize(tot.ext);
        P.ext_map.resize(tot.ext);
        P.n = n;
        P.nblk = nblk;
        P.cl = cl;
        P.nslots = nslots;
        P.nflag = nflag;
        P.nonunit = nonunit;
        P.deep = deep;
        P.lower = R.lower;
        P.rev = rev;
        P.xsize = xsize;
        P.units = tot.unit;
        P.mail_units = tot.mail;
        return HGB_OK;
    }
    void gather(int b) {
        const BlockOut &B = out[b];
        const Base &o = base[b];
        const int ub = (int)o.unit, sb = (int)o.step, eb = (int)o.ext, qe = 16 / xsize;
        int m[2 * kBsW];   // mail units of the strips
        for (int k = 0; k < kBsW; k++) {
            m[2 * k] = B.seg[k] / qe;
            m[2 * k + 1] = (B.seg[k + 1] + qe - 1) / qe;
        }
        P.blk[4 * b + 2] = make_int4(m[0], m[1], m[2], m[3]);
        P.blk[4 * b + 3] = make_int4(m[4], m[5], m[6], m[7]);
        P.blk[4 * b] = make_int4((int)(o.strip / (2 * kBsK)), (int)(B.strip.size() / (2 * kBsK)), B.nflag, B.nslots);
        P.blk[4 * b + 1] = make_int4((int)o.watch, (int)watch[b].size(), mailed[b] ? (int)o.mail : -1, 0);
        for (size_t i = 0; i < B.strip.size(); i++) {
            int4 v = B.strip[i];
            if (i % 2 == 0) v.z += ub;
            P.strip[o.strip + i] = v;
        }
        for (size_t i = 0; i < B.chunk.size(); i++) {
            int4 v = B.chunk[i];
            v.x += ub;
            v.y += sb;
            P.chunk[o.chunk + i] = v;
        }
        for (size_t i = 0; i < B.step.size(); i++) {
            int4 v = B.step[i];
            if (v.z >= 0) v.z += sb;
            v.w = b;
            P.step[o.step + i] = v;
            if (v.y & kBsStepExt)   // the ext rows' first entries count from the plan's array
                for (int q = 0; q < (v.y & 0xFF); q++) {
                    int4 &k = P.pk[v.x + q];
                    if (k.w & kBsExt) k.x += eb;
                }
        }
        std::copy(watch[b].begin(), watch[b].end(), P.watch.begin() + o.watch);
        std::copy(B.ext_codes.begin(), B.ext_codes.end(), P.ext_codes.begin() + o.ext);
        std::copy(B.ext_map.begin(), B.ext_map.end(), P.ext_map.begin() + o.ext);
    }
};

}  // namespace

int bs_plan_sweeps(int n, const int *pntr, const int *indx, const int *diag, int xsize, const std::function<int(int)> &cluster_of,
                   int sweeps, const BsSweepKind *kind, BsPlan **plan) {
    HostTeam team(n);
    std::vector<Sweep> S;
    S.reserve(sweeps);
    for (int q = 0; q < sweeps; q++)
        S.emplace_back(n, pntr, indx, diag, kind[q].lower, kind[q].rev, kind[q].nonunit, xsize, *plan[q]);
    // phase(count, f): f(sweep, i) for the first count(sweep) items of every sweep
    auto phase = [&](auto count, auto f) {
        std::vector<int> first(sweeps + 1, 0);
        for (int q = 0; q < sweeps; q++) first[q + 1] = first[q] + count(S[q]);
        team.run(first[sweeps], [&](int i) {
            int q = 0;
            while (i >= first[q + 1]) q++;
            f(S[q], i - first[q]);
        });
    };
    auto ranges = [](Sweep &s) { return s.ranges; };
    auto blocks = [](Sweep &s) { return s.nblk; };
    phase(ranges, [](Sweep &s, int k) { s.scan(k, -1); });
    for (Sweep &s : S) {
        s.bw = s.widest();
        for (int w : s.wide)
            if (w >= 0) return fail(HGB_ERR_UNSUPPORTED, "triangular plan: row %d has more than 65535 entries", w);
    }
    phase(ranges, [](Sweep &s, int k) { s.scan(k, s.bw / 2); });
    for (Sweep &s : S) {
        s.d2 = s.widest();
        HGB_TRY(s.cut_blocks(cluster_of));
    }
    {
        std::vector<Scratch> scr(16);
        std::vector<std::atomic<int>> used(16);
        for (auto &u : used) u = 0;
        auto left = [&] { return std::any_of(S.begin(), S.end(), [](const Sweep &s) { return !s.planned; }); };
        while (left()) {
            phase([](Sweep &s) { return s.planned ? 0 : s.nblk; }, [&](Sweep &s, int b) {
                int w = 0;   // at most 16 threads take items
                for (int expect = 0; !used[w].compare_exchange_strong(expect, 1); expect = 0) w = (w + 1) % 16;
                s.block(b, scr[w]);
                used[w] = 0;
            });
            for (Sweep &s : S)
                if (!s.planned) HGB_TRY(s.settle(cluster_of));
        }
    }
    phase([](Sweep &s) { return s.runs; }, [](Sweep &s, int r) { s.halos(r); });
    phase([](Sweep &) { return 1; }, [](Sweep &s, int) {
        s.mails();
        s.path();
    });
    phase(blocks, [](Sweep &s, int b) { s.watches(b); });
    for (Sweep &s : S) HGB_TRY(s.sizes());
    phase(blocks, [](Sweep &s, int b) { s.gather(b); });
    // each sweep of a pair resets the entries of the other one's output that are watched there
    if (sweeps == 2) {
        BsPlan &A = *plan[0], &B = *plan[1];
        phase([](Sweep &s) { return s.ranges; }, [&](Sweep &s, int k) {
            if (&s != &S[0]) return;
            for (int row = (int)((long)n * k / s.ranges); row < (int)((long)n * (k + 1) / s.ranges); row++) {
                if (A.watched[row]) B.pk[B.pk_of_row[row]].w |= kBsReset;
                if (B.watched[row]) A.pk[A.pk_of_row[row]].w |= kBsReset;
            }
        });
    }
    return HGB_OK;
}

}  // namespace hgb
