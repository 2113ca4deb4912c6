// Walks the record plan of rdst_records.h as the apply kernel does, on the
// CPU: every offset inside its group, the blocks of a task filling its values
// once each, the row ranges of the starting values covering each task, and
// the two sweeps equal to the plain substitution.
#include <cmath>
#include <cstdio>
#include <random>

#include "../rhodst_b200/csrc/rdst_records.h"

using namespace rdst;

namespace {
int fail(const char* what, int a = 0, int b = 0) {
    std::printf("%s (%d, %d)\n", what, a, b);
    return 1;
}
}  // namespace

// n rows, parts of about n / nparts rows, at most `wide` blocks a side, the
// levels of a random lower pattern that reaches back `reach` rows
extern "C" int check_records(int n, int nparts, int wide, int reach, int elem, int sms, int gauss_seidel, int seed) {
    std::mt19937 rng(seed);
    std::vector<int> part(n), lev(n, 0);
    for (int i = 0; i < n; ++i) part[i] = (int)((long)i * nparts / n);
    std::vector<std::vector<int>> low(n);
    std::vector<int> nup(n, 0);
    for (int i = 0; i < n; ++i) {
        for (int t = 0; t < wide; ++t) {
            const int k = i - 1 - (int)(rng() % reach);
            if (k < 0 || part[k] != part[i] || nup[k] >= wide) continue;
            if (std::find(low[i].begin(), low[i].end(), k) != low[i].end()) continue;
            low[i].push_back(k);
            ++nup[k];
            lev[i] = std::max(lev[i], lev[k] + 1);
        }
    }
    std::vector<int> perm(n), inv(n);
    for (int i = 0; i < n; ++i) perm[i] = i;
    std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) {
        return part[a] != part[b] ? part[a] < part[b] : lev[a] < lev[b];
    });
    for (int r = 0; r < n; ++r) inv[perm[r]] = r;
    std::vector<std::vector<int>> L(n), U(n);
    for (int i = 0; i < n; ++i)
        for (int k : low[i]) { L[inv[i]].push_back(inv[k]); U[inv[k]].push_back(inv[i]); }
    std::vector<int> nl(n), nu(n), lvl_off, part_lvl0(nparts + 1, 0);
    int ML = 0, MU = 0;
    for (int r = 0; r < n; ++r) {
        std::sort(L[r].begin(), L[r].end());
        std::sort(U[r].begin(), U[r].end());
        nl[r] = (int)L[r].size();
        nu[r] = (int)U[r].size();
        ML = std::max(ML, nl[r]);
        MU = std::max(MU, nu[r]);
    }
    for (int r = 0; r < n; ++r)
        if (r == 0 || part[perm[r]] != part[perm[r - 1]] || lev[perm[r]] != lev[perm[r - 1]]) lvl_off.push_back(r);
    lvl_off.push_back(n);
    for (int p = 0, li = 0; p < nparts; ++p) {
        part_lvl0[p] = li;
        while (li + 1 < (int)lvl_off.size() && part[perm[lvl_off[li]]] == p) ++li;
        part_lvl0[p + 1] = li;
    }
    const int MS = std::max(ML + MU, 1);
    auto fid = [&](int r, int s) { return ((r >> 5) * MS + s) * 32 + (r & 31); };
    std::vector<int> lu_col((size_t)((n + 31) / 32) * MS * 32, -1);
    for (int r = 0; r < n; ++r) {
        for (int q = 0; q < nl[r]; ++q) lu_col[fid(r, q)] = L[r][q];
        for (int q = 0; q < nu[r]; ++q) lu_col[fid(r, ML + q)] = U[r][q];
    }
    const std::vector<int> used = gauss_seidel ? std::vector<int>(n, 0) : nu;
    RecPlan P = rec_plan(n, nparts, part_lvl0, lvl_off, lu_col, nl, used, ML, MS, elem, sms, 233472, 232448, 1024);
    if (!P.ok) return fail("no plan");
    const int W = P.warps;
    if (W < 1 || W > REC_MAXW) return fail("shape");
    if (rec_smem(P, elem) > 232448 - 1024 || P.stage_bytes % 128 || P.y0_rows % 2) return fail("shared memory");
    // scalar stand-ins of the blocks: entry j of row i of a block is
    // 1/(1 + 5 i + j) of the block's number
    std::vector<double> bl(lu_col.size()), bd(n);
    std::uniform_real_distribution<double> ud(-0.2, 0.2);
    for (auto& v : bl) v = ud(rng);
    for (auto& v : bd) v = 1.0 + ud(rng);
    std::vector<double> b(5 * n), x(5 * n), ref(5 * n);
    for (auto& v : b) v = ud(rng);
    auto coef = [](int i, int j) { return 1.0 / (1 + 5 * i + j); };
    auto prod = [&](double blk, const double* v, int i) {
        double t = 0;
        for (int j = 0; j < 5; ++j) t += blk * coef(i, j) * v[j];
        return t;
    };
    for (int r = 0; r < n; ++r)
        for (int i = 0; i < 5; ++i) {
            double y = b[5 * r + i];
            for (int q = 0; q < nl[r]; ++q) y -= prod(bl[fid(r, q)], &ref[5 * L[r][q]], i);
            ref[5 * r + i] = y;
        }
    for (int r = n - 1; r >= 0; --r) {
        double y[5];
        for (int i = 0; i < 5; ++i) {
            y[i] = ref[5 * r + i];
            for (int q = 0; q < used[r]; ++q) y[i] -= prod(bl[fid(r, ML + q)], &ref[5 * U[r][q]], i);
        }
        for (int i = 0; i < 5; ++i) ref[5 * r + i] = prod(bd[r], y, i);
    }
    for (int back = 0; back < 2; ++back) {
        const RecSide& S = back ? P.b : P.f;
        size_t task_no = 0;
        for (int p = 0; p < nparts; ++p) {
            // the tasks in sweep order, then each warp's walk over them
            struct At { const RecGroup* G; const unsigned char* gp; int g, t, meta; };
            int end_meta = 0;
            std::vector<At> tasks;
            int32_t sweep_tasks = 0, sweep_levels = 0;
            for (int g = S.part_g[p]; g < S.part_g[p + 1]; ++g) {
                const RecGroup& G = S.groups[g];
                if (G.bytes % 16 || (int)G.bytes > P.stage_bytes || G.nrows > P.y0_rows) return fail("group size", p, g);
                if ((size_t)G.off16 * 16 + G.bytes > S.bytes) return fail("group outside the records");
                if (g > 0 && (size_t)G.off16 * 16 != (size_t)S.groups[g - 1].off16 * 16 + S.groups[g - 1].bytes)
                    return fail("groups not one after the other", g);
                const RecMeta& M = S.group_meta[g];
                if (((size_t)M.off16 + M.n16) * 16 > S.meta.size() || (size_t)M.n16 * 16 > G.bytes) return fail("group meta", g);
                const unsigned char* gp = S.meta.data() + (size_t)M.off16 * 16;
                end_meta = 16 * M.n16;
                int32_t gh[4];
                std::memcpy(gh, gp, 16);
                if (gh[1] != G.row0 || gh[0] < 1 || gh[0] > 256) return fail("group header");
                sweep_tasks = gh[2];
                sweep_levels = gh[3];
                for (int t = 0; t < gh[0]; ++t) {
                    tasks.push_back({&G, gp, g, t, end_meta});
                    const RecTask& T = S.tasks.at(task_no++);
                    if (T.group16 != G.off16 || T.head16 != G.off16 + 1 + 2 * (uint32_t)t) return fail("task list", g, t);
                }
            }
            if ((int)tasks.size() != sweep_tasks || sweep_levels != part_lvl0[p + 1] - part_lvl0[p])
                return fail("sweep sizes", p);
            std::vector<int> level(tasks.size());
            for (size_t t = 0; t < tasks.size(); ++t) {
                uint32_t h[8];
                std::memcpy(h, tasks[t].gp + 16 + 32 * tasks[t].t, 32);
                level[t] = (int)(h[6] >> 16);
                if (t && level[t] != level[t - 1] && level[t] != level[t - 1] + 1) return fail("levels", p, (int)t);
            }
            for (size_t t = 0; t < tasks.size(); ++t) {
                uint32_t h[8];
                std::memcpy(h, tasks[t].gp + 16 + 32 * tasks[t].t, 32);
                const bool last = ((h[1] >> 16) & REC_WARP_LAST) != 0;
                if (last != (t + W >= tasks.size())) return fail("warp's last task", p, (int)t);
                if (last) continue;
                if ((int)(h[1] >> 24) != level[t + W] - level[t]) return fail("levels to the next task", p, (int)t);
                if ((int)(h[7] & 255) != tasks[t + W].t || (int)((h[7] >> 8) & 255) != tasks[t + W].g - tasks[t].g)
                    return fail("way to the next task", p, (int)t);
                // a stage held at task t is not waited for by the warps ahead
                for (size_t u = t + 1; u < t + W; ++u)
                    if (tasks[u].g - tasks[t].g >= REC_STAGES) return fail("stages too few", p, (int)t);
            }
            std::vector<double> lb(2 * (size_t)P.lb_rows * 5, NAN), lbn;
            lbn = lb;
            for (size_t ti = 0; ti < tasks.size(); ++ti) {
                const RecGroup& G = *tasks[ti].G;
                const unsigned char* gp = tasks[ti].gp;
                const int g = tasks[ti].g, t = tasks[ti].t;
                uint32_t h[8];
                std::memcpy(h, gp + 16 + 32 * t, 32);
                unsigned char nk[REC_MAXS] = {0};
                std::memcpy(nk, &h[4], 4);
                const int coff = 16 * (h[0] & 0xffff), voff = 16 * (h[0] >> 16), m = h[1] & 255, Sx = (h[1] >> 8) & 255;
                const unsigned fl = (h[1] >> 16) & 255;
                const int r0 = (int)h[2], own = h[3] & 0xffff, tot = h[3] >> 16;
                const int nq = std::max(1, (Sx + 3) / 4), lbr = rec_lb_row_bytes(elem), none = 2 * P.lb_rows * lbr;
                if (Sx > 4) std::memcpy(nk, gp + coff + 16 * m * nq, REC_MAXS);
                if (m < 1 || m > REC_ROWS) return fail("task", g, t);
                std::vector<char> filled(tot, 0);
                for (int q = 0; back && q < m; ++q) ++filled[q];
                if (r0 - G.row0 != (int)(h[7] >> 16) || r0 < G.row0 || r0 + m > G.row0 + G.nrows)
                    return fail("rows outside the group's range", g, t);
                if ((size_t)voff + (size_t)tot * 25 * elem > G.bytes) return fail("values outside the group", g, t);
                if (coff + 16 * m * nq + (Sx > 4 ? 16 : 0) > tasks[ti].meta || voff < tasks[ti].meta)
                    return fail("columns and values", g, t);
                char seen[REC_ROWS] = {0};
                for (int q = 0; q < m; ++q) {
                    const int rid = (h[5 + q / 4] >> (8 * (q % 4))) & 255, r = r0 + rid;
                    if (rid >= m || seen[rid]++) return fail("row ids", g, t);
                    double y[5];
                    for (int i = 0; i < 5; ++i) y[i] = back ? x[5 * r + i] : b[5 * r + i];
                    int cum = back ? m : 0;
                    for (int k = 0; k < 4 * nq; ++k) {
                        int c;
                        std::memcpy(&c, gp + coff + 4 * (4 * ((k / 4) * m + q) + k % 4), 4);
                        const bool has = q < nk[k];
                        if ((c != none) != has) return fail("columns and counts", g, t);
                        if (has) {
                            if (c > none || (c >= 0 && c % lbr) || -1 - c >= n) return fail("column range");
                            if (c < 0 && !(fl & REC_FAR)) return fail("far column unannounced", g, t);
                            const double* v = c >= 0 ? &lb[5 * (size_t)(c / lbr)] : &x[5 * (size_t)(-1 - c)];
                            if (cum + q >= tot || filled[cum + q]++) return fail("block place", g, t);
                            const double w = bl[fid(r, back ? ML + k : k)];
                            for (int i = 0; i < 5; ++i) y[i] -= prod(w, v, i);
                        }
                        cum += nk[k];
                    }
                    if (cum != tot) return fail("block count", g, t);
                    if (back) {
                        double z[5];
                        for (int i = 0; i < 5; ++i) z[i] = prod(bd[r], y, i);
                        for (int i = 0; i < 5; ++i) y[i] = z[i];
                    }
                    if (own != 0xffff && own + rid >= 2 * P.lb_rows) return fail("own level buffer");
                    for (int i = 0; i < 5; ++i) {
                        x[5 * r + i] = y[i];
                        if (own != 0xffff) lbn[5 * (size_t)(own + rid) + i] = y[i];
                    }
                }
                // visible to the next level only
                if (ti + 1 == tasks.size() || level[ti + 1] != level[ti]) lb = lbn;
            }
        }
    }
    for (int i = 0; i < 5 * n; ++i)
        if (!(std::fabs(x[i] - ref[i]) <= 1e-12 * (1.0 + std::fabs(ref[i])))) return fail("sweep result", i / 5, i % 5);
    return 0;
}
