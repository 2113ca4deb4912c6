// rdst_records.h -- the factor records of the subdomain ILU apply (host code,
// no CUDA: the plan is checked on the CPU by tests/test_ilu_records.py).
//
// A sweep of one subdomain is a list of tasks, each up to six rows of one
// wavefront level (a warp, five lanes a row).  Task t belongs to compute warp
// t mod W; consecutive tasks form groups, and a group is one contiguous byte
// range that one bulk copy brings into a shared-memory stage:
//
//   16 B    group header: tasks of the group, first row, tasks of the sweep,
//           levels of the sweep
//   32 B    per task:
//     w0    columns/16 | values/16 << 16      offsets from the group start
//     w1    n | S << 8 | flags << 16 | dl << 24    rows; slots of the longest
//           row; levels from here to the warp's next task (or to the last)
//     w2    first row
//     w3    level-buffer row of the first row (0xffff: level not kept)
//           | blocks << 16
//     w4    rows that have more than k slots, k = 0..3 (a byte each)
//     w5-6  row of the task at each position (six bytes) | level << 16
//     w7    index of the warp's next task in its group | groups to get there
//           << 8 | first row less the group's << 16
//   then per task
//     columns  max(1, ceil(S/4)) x [n] int4: >= 0 byte offset of the row in
//              the level buffers (a row of zeros past them where the row has
//              no such slot), < 0 row -v - 1 of the global vector; with more
//              than four slots, 16 bytes: rows that have more than k slots
//   then per task
//     values   the blocks' rows of five entries, in vector pieces so that
//              lane (position, component) of a slot reads whole 16-byte (8
//              for BF16) words, neighbouring lanes neighbouring words:
//              FP64  [5 blocks] double2 (entries 0, 1), [5 blocks] double2
//                    (2, 3), [5 blocks] double (4)
//              FP32  [5 blocks] float4 (0..3), [5 blocks] float (4)
//              BF16  [5 blocks] four bf16 (0..3), [5 blocks] bf16 (4)
//
// The rows of a task are held in descending order of their slot counts, so
// the blocks of slot k are those of the first n_k positions: block number
// n_0 + ... + n_{k-1} + position.  Backward the pivot inverses come first
// (n blocks).  Only stored blocks take space.
#pragma once

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <exception>
#include <thread>
#include <vector>

#ifdef __CUDACC__
#define RDST_HD __host__ __device__ __forceinline__
#else
#define RDST_HD inline
#endif

namespace rdst {

constexpr int REC_ROWS = 6;             // rows of a task
constexpr int REC_MAXW = 8;             // compute warps at most
constexpr int REC_MAXS = 16;            // slots of a row at most
// Stages, and the bytes of one at most.  A group's end costs every warp a
// wait and the producer a round trip, so two large stages beat more and
// smaller ones (1.2 M-cell wing FP32: two 196 -> 187 us against three, 256
// against six; 442 k-cell wing FP64 with 16 / 24 / 32 KB: 140 / 111 / 110 us).
// The first two groups of a sweep are smaller: nothing runs before the first.
constexpr int REC_STAGES = 2;
constexpr size_t REC_STAGE_CAP = 65536, REC_RAMP0 = 8192, REC_RAMP1 = 20480;
constexpr int REC_WARP_LAST = 1;        // the warp's last task of the sweep
constexpr int REC_FAR = 2;              // some column lies in the global vector

// The level barriers of a sweep: nlev - 1, taken by every compute warp in the
// same order, waiting on it or not, and also by a warp that has given up, since
// the others may be waiting in one.  A warp goes past at most W - 1 of them
// without waiting (its next task is at most W levels on), so with more than W
// ids in turn none is used again before its last use is complete.  For that to
// hold at the turn too, where a warp that gave up does not wait for the others'
// forward sweep, the backward sweep goes on with the id after the forward one's.
template <bool TIGHT> struct RecBarriers {
    static constexpr int ids = TIGHT ? 4 : 15;
    int id, taken = 0;      // the next barrier's; of this sweep
    RDST_HD RecBarriers(int nlev, bool back) : id(back ? 1 + (nlev - 1) % ids : 1) {}
    RDST_HD void next() { id = id == ids ? 1 : id + 1; ++taken; }
};

// What a warp still has to take once its wait for a group has expired: the rest
// of this sweep's barriers and, from the forward sweep, the backward one's.  The
// others go on into that sweep and give up there (this warp's arrivals are
// missing) or compute on; either way they take all of its barriers.
template <typename Bar, typename Await>
RDST_HD void rec_give_up(Bar& bar, int nlev, bool back, Await&& await) {
    while (bar.taken < nlev - 1) await();
    if (back) return;
    bar.taken = 0;
    while (bar.taken < nlev - 1) await();
}

struct RecGroup { uint32_t off16; uint32_t bytes; int32_t row0; int32_t nrows; };
struct RecTask { uint32_t head16; uint32_t group16; };   // a task's header and its group, from the records' start / 16

// The plan holds what is known of the records before the factors are: each
// group's headers and columns (its first meta bytes), one after the other.
struct RecMeta { uint32_t off16; uint32_t n16; };        // a group's part of RecSide::meta, in 16-byte words

struct RecSide {
    std::vector<unsigned char> meta;
    std::vector<RecMeta> group_meta;
    size_t bytes = 0;                   // of the records
    std::vector<RecGroup> groups;
    std::vector<int> part_g;            // first group of each part
    std::vector<RecTask> tasks;
    std::vector<int> part_t;            // first task of each part
};

struct RecPlan {
    bool ok = false;
    int warps = 0;                      // compute warps W
    bool tight = false;                 // the instance for five or six CTAs an SM
    int stage_bytes = 0;                // largest group, multiple of 128
    int y0_rows = 0;                    // rows of a stage's starting values (even)
    int lb_rows = 0;                    // rows of each of the two level buffers
    RecSide f, b;
};

// bytes of one level-buffer row: five values in the compute type, padded to
// 16-byte words
inline int rec_lb_row_bytes(int elem) { return elem == 8 ? 48 : 32; }

inline size_t rec_smem(const RecPlan& P, int elem) {
    return (size_t)REC_STAGES * (P.stage_bytes + 40 * (size_t)P.y0_rows) +
           (2 * (size_t)P.lb_rows + 1) * rec_lb_row_bytes(elem);
}

// Plan for factors of `elem` bytes.  Rows of part p are the levels
// part_lvl0[p] .. part_lvl0[p+1]-1, level l the rows lvl_off[l] ..
// lvl_off[l+1]-1; factor slot s of row r has id ((r/32) MS + s) 32 + r % 32
// and column lu_col[id]; nl lower slots from s = 0, nu upper ones from ML
// (nu 0: the backward sweep applies the pivot inverses alone).
inline RecPlan rec_plan(int N, int nparts, const std::vector<int>& part_lvl0, const std::vector<int>& lvl_off,
                        const std::vector<int>& lu_col, const std::vector<int>& nl, const std::vector<int>& nu, int ML,
                        int MS, int elem, int sms, size_t smem_sm, size_t smem_block, size_t reserved) {
    RecPlan P;
    const int nlev = (int)lvl_off.size() - 1;
    std::vector<int> lev(N);
    int maxw = 0;
    for (int l = 0; l < nlev; ++l) {
        maxw = std::max(maxw, lvl_off[l + 1] - lvl_off[l]);
        for (int r = lvl_off[l]; r < lvl_off[l + 1]; ++r) lev[r] = l;
    }
    auto fid = [&](int r, int s) { return ((r >> 5) * MS + s) * 32 + (r & 31); };
    auto r16 = [](size_t v) { return (v + 15) / 16 * 16; };
    // CTAs an SM has to hold for all subdomains to run at once, six at most
    // (a larger number runs in turns)
    const int k = std::min(6, std::max(1, (nparts + sms - 1) / std::max(sms, 1)));
    // Compute warps.  A warp spends longer on bringing a task's data into
    // registers than on the part of it that waits for the level before, so
    // even levels of one task want several warps taking turns (four: airfoil
    // 34.4 us, eight 35.9), and wider levels as many as there are (110 k-cell
    // wing FP64, 3.5 tasks a level: four 54.8, six 50.7, eight 48.6 us).  The
    // registers of k CTAs bound the number: 96 a thread up to four CTAs; with
    // five or six three warps of 80, two of 112 with FP64.
    P.tight = k >= 5;
    const int wmax = P.tight ? (elem == 8 ? 2 : 3) : std::min(REC_MAXW, 21 / k - 1);
    const int want = N > REC_ROWS * nlev ? REC_MAXW : 4;
    const size_t budget = std::min(smem_block, smem_sm / k - reserved) - 1024;    // static shared memory, alignment

    struct Task { int r0, n, l, S, tot; };
    auto cnt = [&](int r, bool back) { return back ? nu[r] : nl[r]; };
    auto meta_bytes = [&](const Task& t) {
        return 32 + (size_t)16 * t.n * std::max(1, (t.S + 3) / 4) + (t.S > 4 ? 16 : 0);
    };
    auto value_bytes = [&](const Task& t) { return r16((size_t)t.tot * 25 * elem); };
    // tasks of both sweeps; the backward chunks of a level descend, so that
    // consecutive tasks always cover one contiguous row range
    std::vector<Task> tasks[2];
    std::vector<size_t> task0[2];
    size_t max_one = 0, total[2] = {0, 0};
    for (int back = 0; back < 2; ++back) {
        task0[back].assign(nparts + 1, 0);
        for (int p = 0; p < nparts; ++p) {
            const int a = part_lvl0[p], e = part_lvl0[p + 1];
            for (int i = 0; i < e - a; ++i) {
                const int l = back ? e - 1 - i : a + i;
                const int r0 = lvl_off[l], n = lvl_off[l + 1] - r0, nc = (n + REC_ROWS - 1) / REC_ROWS;
                for (int c = 0; c < nc; ++c) {
                    const int cc = back ? nc - 1 - c : c;
                    Task t{r0 + cc * REC_ROWS, std::min(REC_ROWS, n - cc * REC_ROWS), l, 0, 0};
                    t.tot = back ? t.n : 0;
                    for (int q = 0; q < t.n; ++q) {
                        t.S = std::max(t.S, cnt(t.r0 + q, back));
                        t.tot += cnt(t.r0 + q, back);
                    }
                    max_one = std::max(max_one, meta_bytes(t) + value_bytes(t));
                    total[back] += meta_bytes(t) + value_bytes(t);
                    tasks[back].push_back(t);
                }
            }
            task0[back][p + 1] = tasks[back].size();
        }
    }
    for (int W = std::min(wmax, want); W > 0; W /= 2) {
        P.warps = W;
        const int lbr = rec_lb_row_bytes(elem);
        P.lb_rows = (int)std::min<size_t>(maxw, budget / 2 / (2 * (size_t)lbr));
        P.lb_rows = std::min(P.lb_rows, 16383);
        // a warp may hold a stage until its task is computed while another
        // waits W - 1 tasks further on: that window must fit the stages
        const size_t room = budget - (2 * (size_t)P.lb_rows + 1) * lbr;
        const size_t qmin = std::max(1, W - 1), least = 16 + qmin * max_one;
        size_t cap = room / REC_STAGES;           // a stage: its group and the rows' starting values
        if (cap < least + 40 * qmin * REC_ROWS + 256) continue;      // 256: rounding of both parts
        cap = std::max(least + 40 * qmin * REC_ROWS, std::min(cap - 256, REC_STAGE_CAP));
        // rows of a group of the mean size, never fewer than qmin tasks'
        const size_t mean = std::max(total[0], total[1]) / N + 40;
        const size_t cap_rows = std::max<size_t>(qmin * REC_ROWS, std::min((cap - least) / 40, cap / mean));
        const size_t cap_bytes = cap - 40 * cap_rows;
        size_t max_group = 0;
        int max_rows = 0;
        for (int back = 0; back < 2; ++back) {
            RecSide& S = back ? P.b : P.f;
            const std::vector<Task>& ts = tasks[back];
            // ---- groups, and per task its group and place there
            std::vector<int> grp(ts.size()), place(ts.size());
            std::vector<size_t> gstart;
            S.groups.clear();
            S.part_g.assign(nparts + 1, 0);
            for (int p = 0; p < nparts; ++p) {
                S.part_g[p] = (int)gstart.size();
                size_t bytes = 0, rows = 0;
                for (size_t t = task0[back][p]; t < task0[back][p + 1]; ++t) {
                    const size_t b = meta_bytes(ts[t]) + value_bytes(ts[t]);
                    const size_t nth = gstart.size() - S.part_g[p];      // groups of the part so far
                    const size_t most = nth <= 1 ? REC_RAMP0 : nth == 2 ? REC_RAMP1 : cap_bytes;
                    const size_t in = nth ? t - gstart.back() : 0;
                    if (nth == 0 || (in >= qmin && (bytes + b > std::min(most, cap_bytes) ||
                                                    rows + ts[t].n > cap_rows || in >= 255))) {
                        gstart.push_back(t);
                        bytes = 16;
                        rows = 0;
                    }
                    bytes += b;
                    rows += ts[t].n;
                    grp[t] = (int)gstart.size() - 1;
                    place[t] = (int)(t - gstart.back());
                }
            }
            S.part_g[nparts] = (int)gstart.size();
            gstart.push_back(ts.size());
            const size_t ng = gstart.size() - 1;
            S.group_meta.assign(ng, RecMeta{0, 0});
            S.tasks.assign(ts.size(), RecTask{0, 0});
            S.part_t.assign(task0[back].begin(), task0[back].end());
            size_t rec = 0, meta = 0;
            for (size_t g = 0; g < ng; ++g) {
                int lo = ts[gstart[g]].r0, hi = lo;
                size_t mb = 16, vb = 0;
                for (size_t t = gstart[g]; t < gstart[g + 1]; ++t) {
                    lo = std::min(lo, ts[t].r0);
                    hi = std::max(hi, ts[t].r0 + ts[t].n);
                    mb += meta_bytes(ts[t]);
                    vb += value_bytes(ts[t]);
                    S.tasks[t] = {(uint32_t)(rec / 16 + 1 + 2 * (t - gstart[g])), (uint32_t)(rec / 16)};
                }
                S.groups.push_back({(uint32_t)(rec / 16), (uint32_t)(mb + vb), lo, hi - lo});
                S.group_meta[g] = {(uint32_t)(meta / 16), (uint32_t)(mb / 16)};
                rec += mb + vb;
                meta += mb;
                max_group = std::max(max_group, mb + vb);
                max_rows = std::max(max_rows, hi - lo);
            }
            S.bytes = rec;
            S.meta.assign(meta, 0);
            // ---- headers and columns, the parts shared out over threads
            auto kept = [&](int l) { return lvl_off[l + 1] - lvl_off[l] <= P.lb_rows; };   // levels the buffers hold
            auto fill = [&](int p0, int p1) {
                for (int p = p0; p < p1; ++p) {
                    const size_t tend = task0[back][p + 1];
                    const int nlv = part_lvl0[p + 1] - part_lvl0[p];
                    auto level_of = [&](size_t t) {       // in the order of the sweep
                        return back ? part_lvl0[p + 1] - 1 - ts[t].l : ts[t].l - part_lvl0[p];
                    };
                    for (int gi = S.part_g[p]; gi < S.part_g[p + 1]; ++gi) {
                        const size_t i = gstart[gi], j = gstart[gi + 1];
                        const RecGroup& G = S.groups[gi];
                        unsigned char* g = S.meta.data() + (size_t)S.group_meta[gi].off16 * 16;
                        const int32_t gh[4] = {(int32_t)(j - i), G.row0, (int32_t)(tend - task0[back][p]), nlv};
                        std::memcpy(g, gh, 16);
                        size_t coff = 16 + 32 * (j - i), voff = (size_t)S.group_meta[gi].n16 * 16;
                        for (size_t t = i; t < j; ++t) {
                            const Task& T = ts[t];
                            int ord[REC_ROWS];
                            for (int q = 0; q < T.n; ++q) ord[q] = q;
                            std::stable_sort(ord, ord + T.n, [&](int a, int b) {
                                return cnt(T.r0 + a, back) > cnt(T.r0 + b, back);
                            });
                            const int nq = std::max(1, (T.S + 3) / 4);
                            unsigned char nk[REC_MAXS] = {0};
                            for (int q = 0; q < T.n; ++q)
                                for (int s = 0; s < cnt(T.r0 + q, back); ++s) ++nk[s];
                            if (T.S > 4) std::memcpy(g + coff + (size_t)16 * T.n * nq, nk, REC_MAXS);
                            int32_t* cols = reinterpret_cast<int32_t*>(g + coff);
                            for (int q = 0; q < T.n * 4 * nq; ++q) cols[q] = 2 * P.lb_rows * lbr;
                            const int own = kept(T.l) ? (T.l & 1) * P.lb_rows + T.r0 - lvl_off[T.l] : 0xffff;
                            const int lp = back ? T.l + 1 : T.l - 1;          // the level taken just before
                            bool far = false;
                            for (int s = 0; s < T.S; ++s)
                                for (int q = 0; q < nk[s]; ++q) {
                                    const int c = lu_col[fid(T.r0 + ord[q], back ? ML + s : s)];
                                    const bool near = lev[c] == lp && kept(lp);
                                    cols[((size_t)(s / 4) * T.n + q) * 4 + s % 4] =
                                        near ? ((lp & 1) * P.lb_rows + c - lvl_off[lp]) * lbr : -1 - c;
                                    far |= !near;
                                }
                            // the way to the warp's next task
                            const bool last = t + W >= tend;
                            const int dl = last ? 0 : level_of(t + W) - level_of(t);
                            const uint32_t fl = (last ? REC_WARP_LAST : 0) | (far ? REC_FAR : 0);
                            uint32_t h[8] = {(uint32_t)(coff / 16) | (uint32_t)(voff / 16) << 16,
                                             (uint32_t)T.n | (uint32_t)T.S << 8 | fl << 16 | (uint32_t)dl << 24,
                                             (uint32_t)T.r0, (uint32_t)own | (uint32_t)T.tot << 16, 0u, 0u,
                                             (uint32_t)level_of(t) << 16,
                                             (last ? 0u : (uint32_t)place[t + W] | (uint32_t)(grp[t + W] - grp[t]) << 8) |
                                                 (uint32_t)(T.r0 - G.row0) << 16};
                            for (int q = 0; q < 4; ++q) h[4] |= (uint32_t)nk[q] << (8 * q);
                            for (int q = 0; q < T.n; ++q) h[5 + q / 4] |= (uint32_t)ord[q] << (8 * (q % 4));
                            std::memcpy(g + 16 + 32 * (t - i), h, 32);
                            coff += meta_bytes(T) - 32;
                            voff += value_bytes(T);
                        }
                    }
                }
            };
            const int nt = (int)std::min<size_t>({8, std::max(1u, std::thread::hardware_concurrency()), ts.size() / 2048 + 1,
                                                  (size_t)nparts});
            std::vector<std::thread> th;
            th.reserve(nt);             // nothing may throw past a running thread
            for (int k2 = 1; k2 < nt; ++k2) {
                const int p0 = (int)((long)nparts * k2 / nt), p1 = (int)((long)nparts * (k2 + 1) / nt);
                try {
                    th.emplace_back(fill, p0, p1);
                } catch (const std::exception&) {         // no thread to be had, or no memory for one
                    fill(p0, p1);
                }
            }
            fill(0, (int)((long)nparts / nt));
            for (auto& x : th) x.join();
        }
        P.stage_bytes = (int)((max_group + 127) / 128 * 128);
        P.y0_rows = (max_rows + 1) / 2 * 2;
        if (rec_smem(P, elem) > budget) continue;
        P.ok = true;
        return P;
    }
    return P;
}

}  // namespace rdst
