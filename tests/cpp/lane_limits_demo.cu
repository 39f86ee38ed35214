// Test driver (CPU): lane_pair, which the choice between the fills asks of unchecked
// tables, agrees with what prep_pair then makes of them, at its limits. Prints "ok"
// or "bad <what>".
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../locarna_gb300/csrc/engine_prep.hh"

// n x m nt without arcs, every row's band `width` columns wide (moving along the diagonal)
static void check(const char *what, int n, int m, int width, int opening, bool anchors, bool want) {
    std::vector<int> sigma((size_t)(n + 1) * (m + 1), 0), gap_a(n + 1, -10), gap_b(m + 1, -10), lo(n + 1), hi(n + 1);
    for (int i = 0; i <= n; ++i) {
        lo[i] = std::min((int)((long long)i * (m + 1 - width) / n), m + 1 - width);
        hi[i] = lo[i] + width - 1;
    }
    lcg_pair_tables t{};
    t.len_a = n;
    t.len_b = m;
    t.sigma = sigma.data();
    t.gap_a = gap_a.data();
    t.gap_b = gap_b.data();
    t.indel_opening = opening;
    t.min_col = lo.data();
    t.max_col = hi.data();
    std::vector<int> a_lo(n + 1, 0), a_hi(n + 1, m), b_lo(m + 1, 0), b_hi(m + 1, n);
    if (anchors) {
        t.match_lo = t.del_lo = a_lo.data();
        t.match_hi = t.del_hi = a_hi.data();
        t.ins_lo = b_lo.data();
        t.ins_hi = b_hi.data();
    }
    lcg_align_opts o{};
    lcg_host::Prep p;
    if (lcg_host::prep_pair(t, o, p, 32) != LCG_OK) {
        std::printf("bad %s: %s\n", what, p.err.c_str());
        std::exit(0);
    }
    long long band = 0;
    const bool lane = lcg_host::lane_pair(t, &band), flag = p.flags & lcg::PF_LANES;
    if (lane != want || flag != want || (!anchors && opening <= 0 && band != p.bandcells)) {
        std::printf("bad %s: lane_pair %d, prep_pair %d, want %d\n", what, lane, flag, want);
        std::exit(0);
    }
}

int main() {
    check("plain", 60, 57, 58, -750, false, true);
    check("no opening", 60, 57, 58, 0, false, true);
    check("positive opening", 60, 57, 58, 1, false, false);
    check("anchors", 60, 57, 58, -750, true, false);
    check("span at the limit", 20, lcg_host::LANE_MAX_SPAN - 3, lcg_host::LANE_MAX_SPAN - 2, -750, false, true);
    check("span past it", 20, lcg_host::LANE_MAX_SPAN - 2, lcg_host::LANE_MAX_SPAN - 1, -750, false, false);
    // square bands of 500 columns: 1,200 rows are 600,000 cells
    check("cells at the limit", 1199, 499, 500, -750, false, true);
    check("cells past it", 1200, 499, 500, -750, false, false);
    lcg_pair_tables none{};
    if (lcg_host::lane_pair(none)) std::printf("bad empty tables\n");
    std::printf("ok\n");
    return 0;
}
