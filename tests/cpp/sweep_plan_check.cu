// Host check of a triangular-sweep plan (hgb_bsplan.cu), no GPU: every packet has to name its own row, every
// slot has to fit the CTA's shared memory, and a sweep run step by step on the host, with row numbers in the
// place of values, has to find each of a row's entries in the slot that its code names.
#include "../../hala_gb300/csrc/hgb_bsplan.cu"

#include <cstring>

namespace hgb {
int fail(int code, const char *, ...) { return code; }
}  // namespace hgb

using namespace hgb;

namespace {
enum { ROWS = 0, SLOTS, VALUES, STUCK, TARGETS, STRIPS, COUNT };

struct Sim {
    const BsPlan &P;
    const Rows R;
    int nonunit, rev;
    long bad[COUNT] = {};

    // units of a block's mail that strip k brings in
    void seg(int b, int k, int &first, int &end) const {
        const int4 v = P.blk[4 * b + 2 + (k >> 1)];
        first = (k & 1) ? v.z : v.x;
        end = (k & 1) ? v.w : v.y;
    }
    void run() {
        const int cap = bs_slots_max(P.xsize, nonunit), qe = 16 / P.xsize;
        if (P.nslots > cap) bad[SLOTS]++;
        struct Put {
            int slot, row;
        };
        std::vector<std::vector<Put>> in(P.nblk);
        std::vector<std::vector<int2>> watch(P.nblk);
        std::vector<char> done(P.n, 0);
        for (int b = 0; b < P.nblk; b++) {
            const int4 w = P.blk[4 * b + 1];
            for (int i = 0; i < w.y; i++) {
                watch[b].push_back(P.watch[w.x + i]);
                if (!P.watched[P.watch[w.x + i].x]) bad[TARGETS]++;
            }
        }
        size_t chunk = 0;
        for (int b = 0; b < P.nblk; b++) {
            const int4 bi = P.blk[4 * b];
            if (bi.w > cap || bi.z > P.nflag || bi.w > P.nslots) bad[SLOTS]++;
            std::vector<int> slot(std::max(bi.w, bi.z), -1);   // -1: pending; else the row whose value it holds
            auto put = [&](int s, int row, bool flagged) {
                if (s <= 0 || s >= bi.w || (flagged && (s >= bi.z || slot[s] != -1))) bad[TARGETS]++;
                else slot[s] = row;
            };
            for (const Put &p : in[b]) put(p.slot, p.row, true);
            for (const int2 &w : watch[b]) {
                if (!done[w.x]) bad[STUCK]++;
                put(w.y, w.x, true);
            }
            // the steps of every strip, in order
            struct Strip {
                int rb, at = 0;
                std::vector<int> step;
            };
            if (bi.y > kBsW) bad[STRIPS]++;
            std::vector<Strip> strips(bi.y);
            for (int s = 0; s < bi.y; s++)
                for (int k = 0; k < kBsK; k++) {
                    const int4 sd = P.strip[2 * (((size_t)bi.x + s) * kBsK + k)];
                    strips[s].rb = sd.x;
                    strips[s].step.resize(sd.y);
                    for (int st = k; st < sd.y; st += kBsK, chunk++) {
                        strips[s].step[st] = P.chunk[chunk].y;
                        if (P.chunk[chunk].w != sd.x) bad[ROWS]++;
                    }
                }
            auto ready = [&](const Strip &S, int4 st) {   // all codes of the step's rows are in
                const int nr = st.y & 0xFF;
                for (int i = 0; i < nr; i++) {
                    const int4 p = P.pk[st.x + i];
                    if (p.w & kBsExt) {
                        for (int q = 0; q < (p.y & 0xFFFF); q++) {
                            const int cd = P.ext_codes[(size_t)p.x + (size_t)q * nr];
                            if (cd >= (int)slot.size() || (cd > 0 && slot[cd] == -1) || (cd < 0 && !done[-cd - 1])) return false;
                        }
                        continue;
                    }
                    for (const unsigned cd : {(unsigned)p.x & 0xFFFF, (unsigned)p.x >> 16, (unsigned)p.y & 0xFFFF})
                        if (cd >= slot.size() || (cd && slot[cd] == -1)) return false;
                }
                return true;
            };
            auto solve = [&](const Strip &S, int4 st) {
                const int nr = st.y & 0xFF;
                std::vector<Put> out;
                if (st.w != b) bad[ROWS]++;
                for (int i = 0; i < nr; i++) {
                    const int at = st.x + i;
                    const int4 p = P.pk[at];
                    const int row = S.rb + (p.z & 0xFFFF);
                    if (row < 0 || row >= P.n || P.pk_of_row[row] != at || done[row]) {
                        bad[ROWS]++;
                        continue;
                    }
                    int a, e;
                    R.deps(row, a, e);
                    const bool ext = p.w & kBsExt;
                    if (ext ? e - a != (p.y & 0xFFFF) : e - a > 3) {
                        bad[VALUES]++;
                        continue;
                    }
                    const unsigned code[3] = {(unsigned)p.x & 0xFFFF, (unsigned)p.x >> 16, (unsigned)p.y & 0xFFFF};
                    for (int q = 0; q < (ext ? e - a : 3); q++) {
                        const int ix = q < e - a ? (rev ? e - 1 - q : a + q) : -1, want = ix < 0 ? 0 : R.indx[ix];
                        if (ext) {
                            const size_t k = (size_t)p.x + (size_t)q * nr;
                            const int cd = P.ext_codes[k];
                            if (P.ext_map[k] != ix) bad[VALUES]++;
                            else if (cd < 0 ? (-cd - 1 != want || !P.watched[want]) : (cd == 0 || slot[cd] != want)) bad[VALUES]++;
                        } else if (ix < 0 ? code[q] != 0 : (code[q] == 0 || slot[code[q]] != want)) {
                            bad[VALUES]++;
                        }
                    }
                    const int own = (int)((unsigned)p.y >> 16);
                    if (own != kBsNoSlot) out.push_back({own, row});
                    if (p.w & (kBsPush | kBsMail)) {
                        const int tb = b + (p.w & 0xFF), ts = (int)((unsigned)p.z >> 16);
                        if (tb >= P.nblk || ts <= 0 || ts >= P.blk[4 * tb].z || ((p.w & kBsPush) && (tb <= b || tb / P.cl != b / P.cl))) {
                            bad[TARGETS]++;
                            continue;
                        }
                        if (p.w & kBsMail) {   // the mail of exactly one strip
                            int holders = 0;
                            for (int k = 0; k < kBsW; k++) {
                                int f, l;
                                seg(tb, k, f, l);
                                holders += ts / qe >= f && ts / qe < l;
                            }
                            if (holders != 1 || P.blk[4 * tb + 1].z < 0) bad[TARGETS]++;
                        }
                        in[tb].push_back({ts, row});
                    }
                    done[row] = 1;
                }
                for (const Put &o : out) put(o.slot, o.row, o.slot < bi.z);
            };
            for (bool moved = true; moved;) {
                moved = false;
                for (Strip &S : strips)
                    while (S.at < (int)S.step.size() && ready(S, P.step[S.step[S.at]])) {
                        solve(S, P.step[S.step[S.at++]]);
                        moved = true;
                    }
            }
            for (Strip &S : strips) bad[STUCK] += (long)S.step.size() - S.at;
            for (int k = 0, last = 0; k < kBsW; k++) {   // no unit of the mail belongs to two strips
                int f, l;
                seg(b, k, f, l);
                if (f < last || l < f) bad[TARGETS]++;
                last = l;
            }
            std::vector<Put>().swap(in[b]);
        }
        for (char d : done) bad[ROWS] += !d;
    }
};
}  // namespace

extern "C" {
// Plans the lower sweep only; -1 where it threw.
int sweep_plan_throws(int n, const int *pntr, const int *indx, const int *diag) {
    BsPlan P;
    BsPlan *plan[1] = {&P};
    const BsSweepKind kind[1] = {{1, 0, 0}};
    try {
        return bs_plan_sweeps(n, pntr, indx, diag, 8, [](int nblk) { return std::min(2, nblk); }, 1, kind, plan);
    } catch (const std::exception &) {
        return -1;
    }
}
// Plans both sweeps and runs them; bad[2][6]: what was found wrong in each; shape[2][4]: blocks, slots, path, levels of
// the strip with the most.  most: the largest cluster.
// Returns the planner's status.
int sweep_plan_check(int n, const int *pntr, const int *indx, const int *diag, int xsize, int most, int nonunit_a, int nonunit_b,
                     int rev_b, long *bad, int *shape) {
    BsPlanPair *pair = new BsPlanPair();
    const BsSweepKind kind[2] = {{1, 0, nonunit_a}, {0, rev_b, nonunit_b}};
    BsPlan *plan[2] = {&pair->A, &pair->B};
    const int st = bs_plan_sweeps(n, pntr, indx, diag, xsize, [&](int nblk) { return std::max(1, std::min(most, nblk)); }, 2, kind, plan);
    std::memset(bad, 0, sizeof(long) * 2 * COUNT);
    for (int k = 0; k < 2 && st == 0; k++) {
        Sim s{*plan[k], Rows{n, kind[k].lower, pntr, indx, diag}, kind[k].nonunit, kind[k].rev};
        s.run();
        std::memcpy(bad + k * COUNT, s.bad, sizeof(s.bad));
        shape[4 * k] = plan[k]->nblk;
        shape[4 * k + 1] = plan[k]->nslots;
        shape[4 * k + 2] = (int)std::min<long>(plan[k]->path, INT_MAX);
        shape[4 * k + 3] = plan[k]->levels;
    }
    delete pair;
    return st;
}
}
