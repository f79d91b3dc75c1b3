// Check of the search's division of tiles (bsoft_b200/csrc/search_runs.h) over
// M tiles by N tiles: every tile taken once, in ascending order within a CTA's
// work, every M tile's slots filled once, and, for short panels, no CTA with more
// tiles than groups of ten M tiles by 15 ranges, dealt out item by item, give the
// busiest.  Prints the divisions tried, the wrong ones and those with more.
#include "../bsoft_b200/csrc/search_runs.h"

#include <algorithm>
#include <cstdio>
#include <vector>

static int dealt_out(int mt, int nt) {
    const int mg = std::min(mt, 10);
    int ranges = std::max(1, std::min(nt, (148 + mg - 1) / mg));
    const int per = (nt + ranges - 1) / ranges;
    ranges = (nt + per - 1) / per;
    const int items = (mt + mg - 1) / mg * ranges * mg, ctas = std::min(items, 148);
    std::vector<int> load(148, 0);
    for (int i = 0; i < items; ++i) {
        const int g = i / (ranges * mg), rem = i % (ranges * mg), r = rem / mg;
        if (g * mg + rem % mg < mt) load[i % ctas] += std::min(nt, (r + 1) * per) - r * per;
    }
    return *std::max_element(load.begin(), load.end());
}

int main() {
    std::vector<int> ms, ns;
    for (int m = 1; m <= 60; ++m) ms.push_back(m);
    for (int m : {61, 79, 100, 147, 148, 149, 150, 200, 400, 1000}) ms.push_back(m);
    for (int n = 1; n <= 80; ++n) ns.push_back(n);
    for (int n : {100, 148, 149, 150, 268, 500, 2150}) ns.push_back(n);
    long tried = 0, wrong = 0, more = 0;
    for (int mt : ms)
        for (int nt : ns) {
            const bsg::Runs r = bsg::Runs::plan(mt, nt);
            std::vector<char> tile((size_t)mt * nt, 0);
            std::vector<std::vector<char>> slot(mt);
            for (int m = 0; m < mt; ++m) slot[m].assign(r.slots(m), 0);
            bool ok = r.ctas >= 1 && r.ctas <= 148;
            int most = 0;
            for (int c = 0; c < r.ctas; ++c) {
                int load = 0;
                for (int g = 0; g < r.groups; ++g) {
                    int m, n0, n1;
                    if (!r.work(g, c, m, n0, n1)) continue;
                    if (m < 0 || m >= mt || n0 < 0 || n1 > nt || n0 >= n1) { ok = false; continue; }
                    for (int n = n0; n < n1; ++n) ok = ok && !tile[(size_t)m * nt + n]++;
                    const int s = r.slot(g, c);
                    if (s < 0 || s >= (int)slot[m].size() || slot[m][s]++) ok = false;
                    load += n1 - n0;
                }
                most = std::max(most, load);
            }
            for (char t : tile) ok = ok && t == 1;
            for (auto& v : slot)
                for (char t : v) ok = ok && t == 1;
            wrong += !ok;
            more += nt < bsg::Runs::SHORT_PANEL && most > dealt_out(mt, nt);
            ++tried;
        }
    printf("tried %ld wrong %ld more %ld\n", tried, wrong, more);
    return wrong || more;
}
