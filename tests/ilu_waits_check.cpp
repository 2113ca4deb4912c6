// The waits of the record apply's compute warps when some of them expire, on
// the CPU: the warps walk the plan of rdst_records.h as the kernel walks it, a
// thread each, over stand-ins of the named barriers (W arrivals complete one)
// and of the stages ("full" once all warps have returned the group before,
// backward also once all have ended the forward sweep).  Only an mbarrier wait
// has a bound, so it expires once no warp can go on; a warp that waits in a
// named barrier then is one that the kernel would leave there for ever.
#include <condition_variable>
#include <cstdio>
#include <functional>
#include <mutex>
#include <random>

#include "../rhodst_b200/csrc/rdst_records.h"

using namespace rdst;

namespace {

struct Stuck {};

struct Sim {
    int W;
    std::mutex m;
    std::condition_variable cv;
    int running = 0;
    bool stuck = false, mixed = false;
    struct Wait { std::function<bool()> ready; bool bounded = false, waiting = false, expired = false; };
    std::vector<Wait> waits;
    std::mt19937 rng;
    // named barriers: arrivals so far, completions, and which barrier of the
    // walk the arrivals mean
    int arrivals[16] = {0}, done[16] = {0}, which[16] = {0};
    int fdone = 0;
    std::vector<int> empty[2];          // [sweep][group] warps that returned it

    // with m held: let go on who can, else expire one bounded wait
    void settle() {
        while (running == 0) {
            std::vector<int> open;
            bool any = false, waiting = false;
            for (int w = 0; w < W; ++w) {
                Wait& x = waits[w];
                if (!x.waiting) continue;
                waiting = true;
                if (x.ready()) { x.waiting = false; ++running; any = true; }
                else if (x.bounded) open.push_back(w);
            }
            if (any || !waiting) break;
            if (open.empty()) { stuck = true; break; }
            Wait& x = waits[open[rng() % open.size()]];
            x.expired = true;
            x.waiting = false;
            ++running;
        }
        cv.notify_all();
    }
    bool wait(std::unique_lock<std::mutex>& lk, int w, bool bounded, std::function<bool()> ready) {
        Wait& x = waits[w];
        x.ready = ready;
        x.bounded = bounded;
        x.waiting = true;
        x.expired = false;
        --running;
        settle();
        cv.wait(lk, [&] { return !x.waiting || stuck; });
        if (stuck) throw Stuck();
        return !x.expired;
    }
    void arrive(int id, int index) {
        if (arrivals[id] == 0) which[id] = index;
        else if (which[id] != index) mixed = true;
        if (++arrivals[id] == W) { arrivals[id] = 0; ++done[id]; }
    }
};

struct Task { int level, group; };

// one compute warp; its wait for group lose_group of sweep lose_sweep expires
template <bool TIGHT>
void walk(Sim& S, int w, const std::vector<Task> (&tasks)[2], const int (&groups)[2], int nlev, int lose_sweep,
          int lose_group) {
    std::unique_lock<std::mutex> lk(S.m);
    int seq = 0;                                    // barriers taken in the whole walk
    for (int back = 0; back < 2; ++back) {
        const std::vector<Task>& T = tasks[back];
        int grp = 0;
        RecBarriers<TIGHT> bar(nlev, back != 0);
        auto arrive = [&] { S.arrive(bar.id, seq++); bar.next(); };
        auto await = [&] {
            const int id = bar.id, n = S.done[id];
            S.arrive(id, seq++);
            S.wait(lk, w, false, [&S, id, n] { return S.done[id] != n; });
            bar.next();
        };
        auto enter = [&] {
            const bool got = !(back == lose_sweep && grp == lose_group) && S.wait(lk, w, true, [&S, grp, back] {
                return (!back || S.fdone == S.W) && (grp < REC_STAGES || S.empty[back][grp - REC_STAGES] == S.W);
            });
            if (!got) rec_give_up(bar, nlev, back != 0, await);
            return got;
        };
        auto next_group = [&] { ++S.empty[back][grp++]; return enter(); };
        auto go = [&] {
            if (!enter()) return false;
            size_t t = w;
            if (t < T.size()) {
                while (grp < T[t].group)
                    if (!next_group()) return false;
                while (bar.taken < T[t].level - 1) arrive();
                if (bar.taken < T[t].level) await();
                for (; t + S.W < T.size(); t += S.W) {
                    const int dl = T[t + S.W].level - T[t].level;
                    for (int q = 1; q < dl; ++q) arrive();
                    while (grp < T[t + S.W].group)
                        if (!next_group()) return false;
                    if (dl > 0) await();
                }
            }
            while (bar.taken < nlev - 1) arrive();
            if (!back) ++S.fdone;
            while (grp + 1 < groups[back])
                if (!next_group()) return false;
            ++S.empty[back][grp];
            return true;
        };
        if (!go()) return;
    }
}

template <bool TIGHT>
int run(int W, const std::vector<Task> (&tasks)[2], const int (&groups)[2], int nlev, unsigned lost, int lose_sweep,
        int lose_group, int seed) {
    Sim S;
    S.W = S.running = W;
    S.waits.resize(W);
    S.rng.seed(seed);
    for (int b = 0; b < 2; ++b) S.empty[b].assign(groups[b], 0);
    std::vector<std::thread> th;
    for (int w = 0; w < W; ++w)
        th.emplace_back([&, w] {
            try {
                walk<TIGHT>(S, w, tasks, groups, nlev, (lost >> w) & 1 ? lose_sweep : -1, lose_group);
            } catch (const Stuck&) {
            }
            std::lock_guard<std::mutex> lk(S.m);
            --S.running;
            S.settle();
        });
    for (auto& t : th) t.join();
    return S.stuck ? 1 : (S.mixed ? 2 : 0);
}

}  // namespace

// One subdomain of `nlev` levels of random widths up to `wide` rows: every
// group of both sweeps lost by one warp, by all but one, and by random ones.
// 0; 1 a warp is left in a barrier; 2 a barrier completed by arrivals of
// different levels; 3 no plan; -1 no case taken.
extern "C" int check_waits(int nlev, int wide, int elem, int nparts, int seed) {
    std::mt19937 rng(seed);
    std::vector<int> lvl_off(1, 0), part_lvl0(nparts + 1, 0);
    for (int p = 0; p < nparts; ++p) {
        for (int l = 0; l < nlev; ++l) lvl_off.push_back(lvl_off.back() + 1 + (int)(rng() % wide));
        part_lvl0[p + 1] = (p + 1) * nlev;
    }
    const int n = lvl_off.back();
    // each row coupled to three of the level before and of the level after
    std::vector<int> nl(n, 0), nu(n, 0), lu_col((size_t)((n + 31) / 32) * 6 * 32, -1);
    for (int p = 0; p < nparts; ++p)
        for (int l = part_lvl0[p]; l < part_lvl0[p + 1]; ++l)
            for (int r = lvl_off[l]; r < lvl_off[l + 1]; ++r)
                for (int q = 0; q < 3; ++q) {
                    if (l > part_lvl0[p]) lu_col[((r >> 5) * 6 + nl[r]++) * 32 + (r & 31)] = lvl_off[l - 1];
                    if (l + 1 < part_lvl0[p + 1]) lu_col[((r >> 5) * 6 + 3 + nu[r]++) * 32 + (r & 31)] = lvl_off[l + 1];
                }
    const RecPlan P = rec_plan(n, nparts, part_lvl0, lvl_off, lu_col, nl, nu, 3, 6, elem, 1, 233472, 232448, 1024);
    if (!P.ok) return 3;
    std::vector<Task> tasks[2];
    int groups[2], cases = 0;
    for (int back = 0; back < 2; ++back) {
        const RecSide& R = back ? P.b : P.f;
        groups[back] = R.part_g[1];
        for (int g = 0; g < R.part_g[1]; ++g) {
            const unsigned char* gp = R.meta.data() + (size_t)R.group_meta[g].off16 * 16;
            int32_t gh[4];
            std::memcpy(gh, gp, 16);
            for (int t = 0; t < gh[0]; ++t) {
                uint32_t h[8];
                std::memcpy(h, gp + 16 + 32 * t, 32);
                tasks[back].push_back({(int)(h[6] >> 16), g});
            }
        }
    }
    for (int back = 0; back < 2; ++back)
        for (int g = 0; g < groups[back]; ++g)
            for (int k = 0; k < 4; ++k) {
                const unsigned all = (1u << P.warps) - 1, one = 1u << (rng() % P.warps);
                const unsigned lost = k == 0 ? one : k == 1 ? all & ~one : k == 2 ? (unsigned)(rng() & all) : all;
                const int rc = P.tight ? run<true>(P.warps, tasks, groups, nlev, lost, back, g, (int)rng())
                                       : run<false>(P.warps, tasks, groups, nlev, lost, back, g, (int)rng());
                if (rc) {
                    std::printf("sweep %d of %d warps, group %d lost by %x: %d\n", back, P.warps, g, lost, rc);
                    return rc;
                }
                ++cases;
            }
    return cases ? 0 : -1;
}
