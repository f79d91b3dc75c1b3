// search_runs.h - how the exhaustive search's GEMM divides its tiles (M tiles of
// image rows by N tiles of panel sections) over the SMs; plain C++ on the host,
// where tests/search_runs_check.cpp runs it.
#pragma once

#ifdef __CUDACC__
#define BSG_RUNS_FN __host__ __device__
#else
#define BSG_RUNS_FN
#endif

namespace bsg {

// Panels of SHORT_PANEL N tiles and more: in group g (M tiles first(g) ..
// first(g + 1) - 1) CTA c takes M tile c % size of it and the N tiles of stretch
// c / size.  Groups of 21, seven and four M tiles have 7, 21 and 37 stretches.
// Shorter panels: the tiles in the order (M, N) in equal runs, one per CTA.  Their
// few tiles do not divide into 21 or 37 stretches, and all of B is in L2 anyway:
// 400 images of 64^2 x 25 origins against 2,000 sections took 0.22 ms of GEMM in
// stretches and take 0.17 in runs, 512 of 128^2 against 768 sections 0.28 and
// 0.21.  From 21 tiles on the stretches fill the SMs, and runs, which hold all M
// tiles in flight at once, lose at 128^2 (512 images, 20 tiles: 1.06 and 1.09 ms;
// 28 tiles: 1.33 and 1.53).
// An M tile's partial results sit in slots, one per CTA that took N tiles of it.
struct Runs {
    static constexpr int SMS = 148, SHORT_PANEL = 21;
    int mtiles, ntiles, ctas;
    int groups;                       // groups; short panels: most M tiles in a run
    int large, sevens;                // large groups of 21, then sevens, then fours; sevens < 0: groups of
                                      // nearly equal sizes

    BSG_RUNS_FN bool short_panel() const { return ntiles < SHORT_PANEL; }

    BSG_RUNS_FN static Runs plan(int mtiles, int ntiles) {
        Runs r{mtiles, ntiles, SMS, 0, 0, -1};
        if (r.short_panel()) {
            const long tiles = (long)mtiles * ntiles;
            if (tiles < SMS) r.ctas = (int)tiles;
            r.groups = (int)(((tiles + r.ctas - 1) / r.ctas + 2L * ntiles - 2) / ntiles);
            return r;
        }
        for (int four = 0; four < 7 && r.sevens < 0; ++four)
            if (mtiles >= 4 * four && (mtiles - 4 * four) % 7 == 0) {
                r.sevens = (mtiles - 4 * four) / 7;
                r.large = r.sevens / 3;
                r.sevens -= 3 * r.large;
                r.groups = r.large + r.sevens + four;
            }
        if (r.sevens < 0) r.groups = (mtiles + 6) / 7;     // below 18, where sevens and fours do not add up
        return r;
    }

    // ---- short panels: tile t = mtile ntiles + n
    BSG_RUNS_FN long run(int c) const { return (long)c * mtiles * ntiles / ctas; }      // CTA c's first tile
    BSG_RUNS_FN int cta_of(long t) const { return (int)(((t + 1) * ctas - 1) / ((long)mtiles * ntiles)); }

    // ---- others
    BSG_RUNS_FN int first(int g) const {
        if (sevens < 0) return (int)((long)g * mtiles / groups);
        if (g <= large) return 21 * g;
        g -= large;
        return 21 * large + (g <= sevens ? 7 * g : 7 * sevens + 4 * (g - sevens));
    }
    BSG_RUNS_FN int size(int g) const { return first(g + 1) - first(g); }
    BSG_RUNS_FN int stretches(int g) const {
        const int n = ctas / size(g);
        return n < ntiles ? n : ntiles;
    }
    // first N tile of stretch r
    BSG_RUNS_FN int bound(int g, int r) const {
        const int n = stretches(g);
        return (int)(((long)r * ntiles + (long)g * n / groups) / n);
    }
    BSG_RUNS_FN int group_of(int mtile) const {
        if (sevens >= 0) {
            if (mtile < 21 * large) return mtile / 21;
            const int m = mtile - 21 * large;
            return large + (m < 7 * sevens ? m / 7 : sevens + (m - 7 * sevens) / 4);
        }
        int g = (int)((long)mtile * groups / mtiles);
        while (first(g) > mtile) --g;
        while (first(g + 1) <= mtile) ++g;
        return g;
    }

    // CTA c's M tile and N tiles in group g (short panels: in the g-th M tile of
    // its run); false: none
    BSG_RUNS_FN bool work(int g, int c, int& m, int& n0, int& n1) const {
        if (short_panel()) {
            const long t0 = run(c), t1 = run(c + 1);
            m = (int)(t0 / ntiles) + g;
            const long base = (long)m * ntiles;
            n0 = t0 > base ? (int)(t0 - base) : 0;
            n1 = t1 < base + ntiles ? (int)(t1 - base) : ntiles;
            return n0 < n1;
        }
        const int sz = size(g), r = c / sz;
        if (r >= stretches(g)) return false;
        m = first(g) + c % sz;
        n0 = bound(g, r);
        n1 = bound(g, r + 1);
        return true;
    }
    // the slot of that work's results among its M tile's
    BSG_RUNS_FN int slot(int g, int c) const {
        return short_panel() ? c - cta_of((run(c) / ntiles + g) * ntiles) : c / size(g);
    }
    // an M tile's slots, all of them filled
    BSG_RUNS_FN int slots(int mtile) const {
        if (!short_panel()) return stretches(group_of(mtile));
        const long base = (long)mtile * ntiles;
        return cta_of(base + ntiles - 1) - cta_of(base) + 1;
    }
};

}  // namespace bsg
