// rec_plan when memory runs out at any one of its allocations: std::bad_alloc
// reaches the caller, or the plan is made all the same; the process goes on.
#include <cstdio>
#include <cstdlib>
#include <new>

#include "../rhodst_b200/csrc/rdst_records.h"

using namespace rdst;

static long left = -1;      // allocations until the one that fails (-1: none does)

static void* take(std::size_t n) {
    if (left >= 0 && left-- == 0) return nullptr;
    return std::malloc(n ? n : 1);
}
void* operator new(std::size_t n) {
    if (void* p = take(n)) return p;
    throw std::bad_alloc();
}
void* operator new(std::size_t n, const std::nothrow_t&) noexcept { return std::malloc(n ? n : 1); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
void operator delete(void* p, const std::nothrow_t&) noexcept { std::free(p); }

int main() {
    // four subdomains of 2,000 levels of three rows: several threads fill the plan
    const int parts = 4, nlev = 2000, n = parts * nlev * 3;
    std::vector<int> lvl_off, part_lvl0, nl(n, 0), nu(n, 0), lu_col((size_t)((n + 31) / 32) * 2 * 32, -1);
    for (int l = 0; l <= parts * nlev; ++l) lvl_off.push_back(3 * l);
    for (int p = 0; p <= parts; ++p) part_lvl0.push_back(p * nlev);
    for (int r = 0; r < n; ++r) {
        const int l = r / 3;
        if (l % nlev) { nl[r] = 1; lu_col[((r >> 5) * 2) * 32 + (r & 31)] = r - 3; }
        if (l % nlev != nlev - 1) { nu[r] = 1; lu_col[((r >> 5) * 2 + 1) * 32 + (r & 31)] = r + 3; }
    }
    auto plan = [&] {
        return rec_plan(n, parts, part_lvl0, lvl_off, lu_col, nl, nu, 1, 2, 8, 148, 233472, 232448, 1024);
    };
    const RecPlan whole = plan();
    if (!whole.ok) return 2;
    int thrown = 0;
    for (long k = 0;; ++k) {
        left = k;
        try {
            const RecPlan P = plan();
            const bool done = left >= 0;        // fewer allocations than that
            left = -1;
            if (P.f.meta != whole.f.meta || P.b.meta != whole.b.meta) return 3;
            if (done) break;
        } catch (const std::bad_alloc&) {
            left = -1;
            ++thrown;
        }
    }
    std::printf("%d allocations whose failure reaches the caller\n", thrown);
    return thrown > 0 ? 0 : 4;
}
