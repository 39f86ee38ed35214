// Test driver (CPU): the plan of the lane-per-group fill (LaneItem, blkrows,
// the order of the D writes, the corner cells of PairDev::cre) as
// lcg_host::prep_pair makes it, walked the way the kernel walks it
// (sankoff_lane_kernels.cu), with every access checked.
// argv: A.pp B.pp nolp stacking max_diff indel_opening groups. Prints "ok <items> <late entries> <D>"
// when every access was in bounds and to a cell already written, every D entry
// read had been written by an earlier item, an earlier quad or (late entries)
// an earlier row, and every D equals the one of a group-by-group evaluation;
// else "bad <what>".
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <sstream>
#include <string>
#include <vector>

#include "../../locarna_gb300/csrc/engine_prep.hh"

using namespace lcg;

static void bad(const char *what, long long a = 0, long long b = 0) {
    std::printf("bad %s %lld %lld\n", what, a, b);
    std::exit(0);
}
static std::string slurp(const char *p) {
    std::ifstream f(p);
    std::stringstream s;
    s << f.rdbuf();
    return s.str();
}

int main(int, char **argv) {
    lcg_prep_opts po;
    lcg_prep_opts_default(&po);
    const bool nolp = std::atoi(argv[3]);
    const int W = std::atoi(argv[7]);
    po.stacking = std::atoi(argv[4]);
    if (po.stacking) po.exp_prob = 0.01;
    po.max_diff = std::atoi(argv[5]);
    po.indel_opening = std::atoi(argv[6]);
    lcg_prepared h;
    if (lcg_prepare_pair(slurp(argv[1]).c_str(), slurp(argv[2]).c_str(), &po, &h)) bad("prepare");
    lcg_pair_tables t;
    lcg_prepared_tables(h, &t);
    lcg_align_opts ao{};
    ao.no_lonely_pairs = nolp;
    lcg_host::Prep p;
    if (lcg_host::prep_pair(t, ao, p, W) != LCG_OK) bad("prep_pair");
    if (!(p.flags & PF_LANES)) bad("no lanes");
    const int n = p.n, m = p.m, go = t.indel_opening;
    auto sigma = [&](int i, int j) { return t.sigma[(size_t)i * (m + 1) + j]; };
    auto cell = [&](int i, int j) { return p.bandoff[i] + j - p.min_col[i]; };
    auto inb = [&](int i, int j) { return i >= 0 && i <= n && p.min_col[i] <= j && j <= p.max_col[i]; };
    const int4 *cre = (const int4 *)p.cre.data();

    // ---- D group by group (init_state, align_in_arcmatch, fill_D_entries)
    std::vector<int> Dref(p.Dinit);
    for (size_t g = 0; g + 1 < p.groups.size(); ++g) {
        const GroupItem &G = p.groups[g];
        const int w = m + 2;
        std::vector<int> M((size_t)(n + 1) * w, NEG), E(w, NEG);
        auto MM = [&](int i, int j) -> int & { return M[(size_t)i * w + j]; };
        MM(G.al, G.bl) = 0;
        for (int j = G.bl + 1, s = go; j < G.br && j <= p.max_col[G.al]; ++j) MM(G.al, j) = s += t.gap_b[j];
        int col = go;
        int k = G.dw_start;
        std::vector<int4> dws(p.dw.begin() + G.dw_start, p.dw.begin() + G.dw_start + G.dw_count);
        for (int i = G.al + 1; i < G.ar; ++i) {
            col += t.gap_a[i];
            if (p.min_col[i] <= G.bl) MM(i, G.bl) = col;
            int F = NEG;
            for (int j = std::max(G.bl + 1, p.min_col[i]); j <= std::min(G.br - 1, p.max_col[i]); ++j) {
                const int up = inb(i - 1, j) ? MM(i - 1, j) : NEG, dg = inb(i - 1, j - 1) ? MM(i - 1, j - 1) : NEG;
                E[j] = norm(std::max(E[j] + t.gap_a[i], up + t.gap_a[i] + go));
                F = norm(std::max(F + t.gap_b[j], MM(i, j - 1) + t.gap_b[j] + go));
                int v = std::max(std::max(dg + sigma(i, j), E[j]), F);
                for (int e = p.cre_start[cell(i, j)]; e < p.cre_start[p.bandcells + cell(i, j)]; ++e) {
                    const int ca = cre[e].y & 0xffff, cb = cre[e].y >> 16;
                    if (ca < G.al || cb < G.bl || !inb(ca, cb) || Dref[cre[e].x] < MIN_FINITE) continue;
                    if (Dref[cre[e].x] == NOT_READY) bad("reference order", g, e);
                    v = std::max(v, MM(ca, cb) + Dref[cre[e].x]);
                }
                MM(i, j) = norm(v);
            }
            for (size_t q = 0; q < dws.size(); ++q)
                if (dws[q].y == i) {
                    int v = MM(i, dws[q].z) + dws[q].w;
                    if (!p.dwn.empty()) {
                        const int2 x = p.dwn[G.dw_start + q];
                        v = std::max(v, (x.x < 0 ? NEG : Dref[x.x]) + x.y);
                    }
                    Dref[dws[q].x] = norm(v);
                }
        }
        (void)k;
    }

    // ---- the same D by items, as the kernel sweeps them
    std::vector<int> D(p.Dinit);
    long long nlate = 0;
    size_t covered = 0;
    for (const LaneItem &it : p.litems) {
        if (it.g0 != (int)covered) bad("groups not consecutive", it.g0, covered);
        covered += it.ng;
        if (it.ng < 1 || it.ng > W) bad("group count", it.ng);
        const long long lines = p.bandoff[it.a1] - p.bandoff[it.a0];
        if (lines > p.lane_slot) bad("slot", lines, p.lane_slot);
        if (it.line + lines > p.lane_lines) bad("kept lines", it.line, lines);
        const int cell0 = p.bandoff[it.a0], shift = nolp ? 2 : 1;
        std::vector<int> M(lines * W, INT_MAX), Q((size_t)(n + 1) * W, INT_MAX);
        auto rd = [&](long long line, int ln) {
            if (line < 0 || line >= lines) bad("read out of the storage", line, lines);
            if (M[line * W + ln] == INT_MAX) bad("read of an unwritten cell", line, ln);
            return M[line * W + ln];
        };
        const GroupItem &gf = p.groups[it.g0], &gl = p.groups[it.g0 + it.ng - 1];
        const unsigned first = (unsigned)gf.al << 16 | gf.bl, last = (unsigned)gl.al << 16 | gl.bl;
        std::vector<int> dwi(W, 0), dwend(W, 0);
        for (int ln = 0; ln < it.ng; ++ln) {
            const GroupItem &g = p.groups[it.g0 + ln];
            dwi[ln] = g.dw_start;
            dwend[ln] = g.dw_start + g.dw_count;
            if (g.al < it.a0 || g.al > it.amax || g.ar > it.a1 || g.bl < it.b0 || g.br > it.b1) bad("extent", it.g0);
        }
        for (int J = it.b0 >> 3; J <= (it.b1 - 1) >> 3; ++J) {
            const int4 bq = p.blkrows[J];
            const int qa = std::max(bq.x, it.a0 >> 2), qb = std::min(bq.y, (it.a1 - 1) >> 2);
            if (qa > qb) break;
            const int j0 = J * 8;
            std::vector<int> Mup(8 * W, NEG), V(8 * W, NEG), Mul(W, NEG);
            if (4 * qa - 1 >= it.a0 && j0 - 1 >= std::max(it.b0, p.min_col[4 * qa - 1]) && j0 - 1 <= p.max_col[4 * qa - 1])
                for (int ln = 0; ln < W; ++ln) Mul[ln] = rd(cell(4 * qa - 1, j0 - 1) - cell0, ln);
            for (int q = qa; q <= qb; ++q) {
                std::vector<int> A(32 * W, NEG);
                bool any_late = false;
                auto lohi = [&](int i, int &lo, int &hi) {
                    lo = INT_MAX, hi = -1;
                    if (i >= it.a0 && i < it.a1) lo = std::max(it.b0, p.min_col[i]), hi = std::min(it.b1 - 1, p.max_col[i]);
                };
                auto terms = [&](int i, bool late_pass) {
                    int lo, hi;
                    lohi(i, lo, hi);
                    const int x = std::max(lo, j0), y = std::min(hi, j0 + 7);
                    if (x > y || i <= it.a0) return;
                    const int k = bq.z + (i >> 2) - bq.x;
                    if (p.cre_start[cell(i, x)] < p.quad_start[k] || p.cre_start[p.bandcells + cell(i, y)] > p.quad_start[k + 1])
                        bad("entry list of the quad", i, J);
                    for (int e = p.cre_start[cell(i, x)]; e < p.cre_start[p.bandcells + cell(i, y)]; ++e) {
                        const int ca = cre[e].y & 0xffff, cb = cre[e].y >> 16, cc = (int)((unsigned)cre[e].z >> 5);
                        if (cc < cell0 || cb < it.b0) continue;
                        const unsigned key = (unsigned)(ca + shift) << 16 | (unsigned)(cb + shift);
                        const bool late = key <= first && key >= last;
                        if (((cre[e].z >> 3) & 3) != (i & 3)) bad("row of the quad", i, e);
                        if (late) any_late = true;
                        if (late != late_pass) continue;
                        nlate += late;
                        const int d = D[cre[e].x];
                        if (d == NOT_READY) bad("wait that no earlier work ends", i, e);
                        if (d < MIN_FINITE) continue;
                        for (int ln = 0; ln < W; ++ln) {
                            int &a = A[(cre[e].z & 31) * W + ln];
                            a = std::max(a, rd(cc - cell0, ln) + d);
                        }
                    }
                };
                for (int r = 0; r < 4; ++r) terms(4 * q + r, false);
                const bool rows = any_late || !p.dwn.empty();  // (whole quads and row by row give the same otherwise)
                auto dwrites = [&](int row) {
                    for (int ln = W - 1; ln >= 0; --ln)
                        while (dwi[ln] < dwend[ln]) {
                            const int4 e = p.dw[dwi[ln]];
                            if (!((e.z >> 3) == J && (row < 0 ? (e.y >> 2) == q : e.y == row))) break;
                            int v = rd(cell(e.y, e.z) - cell0, ln) + e.w;
                            if (!p.dwn.empty()) {
                                const int2 x = p.dwn[dwi[ln]];
                                if (x.x >= 0 && D[x.x] == NOT_READY) bad("inner D not written", it.g0, ln);
                                v = std::max(v, (x.x < 0 ? NEG : D[x.x]) + x.y);
                            }
                            D[e.x] = norm(v);
                            ++dwi[ln];
                        }
                };
                for (int r = 0; r < 4; ++r) {
                    const int i = 4 * q + r;
                    int lo, hi;
                    lohi(i, lo, hi);
                    if (rows) terms(i, true);
                    const bool in = lo <= j0 - 1 && j0 - 1 <= hi;
                    for (int ln = 0; ln < W; ++ln) {
                        int hs = NEG, Md = Mul[ln];
                        Mul[ln] = NEG;
                        if (in) {
                            hs = Q[(size_t)i * W + ln];
                            if (hs == INT_MAX) bad("gap state not written", i, j0);
                            Mul[ln] = rd(cell(i, j0 - 1) - cell0, ln);
                        }
                        const bool on = ln < it.ng;
                        for (int u = 0; u < 8; ++u) {
                            const int j = j0 + u;
                            int x = NEG, E = NEG, F = NEG;
                            const bool ib = j >= lo && j <= hi;
                            if (ib) {
                                E = V[u * W + ln] + t.gap_a[i];
                                F = hs + t.gap_b[j];
                                x = std::max(std::max(std::max(Md + sigma(i, j), E), std::max(F, NEG)), A[(r * 8 + u) * W + ln]);
                                if (on && i == p.groups[it.g0 + ln].al && j == p.groups[it.g0 + ln].bl) x = 0;
                                if (cell(i, j) - cell0 < 0 || cell(i, j) - cell0 >= lines) bad("store", i, j);
                                M[(size_t)(cell(i, j) - cell0) * W + ln] = x;
                            }
                            V[u * W + ln] = ib ? std::max(x + go, E) : NEG;
                            hs = ib ? std::max(x + go, F) : NEG;
                            Md = Mup[u * W + ln];
                            Mup[u * W + ln] = x;
                        }
                        if (i >= it.a0 && i < it.a1) Q[(size_t)i * W + ln] = hs;
                    }
                    if (rows) dwrites(i);
                }
                if (!rows) dwrites(-1);
            }
        }
        for (int ln = 0; ln < it.ng; ++ln)
            if (dwi[ln] != dwend[ln]) bad("D write never reached", it.g0 + ln, dwi[ln]);
    }
    if (covered + 1 != p.groups.size()) bad("groups left out", covered, p.groups.size());
    for (size_t k = 0; k < D.size(); ++k)
        if (D[k] != Dref[k]) bad("D differs", k, D[k]);
    std::printf("ok %zu %lld %zu\n", p.litems.size(), nlate, D.size());
    return 0;
}
