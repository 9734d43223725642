// Cells ordered by place, and equal shares of several such lists.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace mantiis
{
// Order of cells by place: row by row.  A contiguous share of such a list is a band
// of the level, whatever the kind of cell, so the cells of one SM read each
// other's sectors; long rows keep a warp's cells side by side (us per step of the
// cooperative engine at 1024^2, single block / two levels, with the cells in
// 32x32 tiles along a Z curve 13.6 / 39, 128x16 12.5 / 36, in rows 12.5 / 34).
inline uint32_t site_order_key(int32_t xy) { return (uint32_t)xy; } // x | y << 16

// one list of cells sorted by site_order_key: x | y << 16 of cell i at xy[i * stride]
struct ShareList
{
    const int32_t *xy;
    int32_t n;
    int stride;
    double weight; // work of a cell
};
// Per list the parts + 1 cuts that give every part the same work and the same patch:
// cut k takes the cells, in the order of all lists together, until their weight reaches
// k / parts of the total.  A list's cells up to the next cell of another list are taken as
// one run (cell by cell, this took 7 ns a cell, 4 % of a context's creation).
inline std::vector<std::vector<int32_t>> share_cuts(const std::vector<ShareList> &lists, int parts)
{
    double total = 0;
    for (const ShareList &l : lists) total += l.weight * (double)l.n;
    std::vector<std::vector<int32_t>> cuts(lists.size(), std::vector<int32_t>((size_t)parts + 1, 0));
    std::vector<int32_t> at(lists.size(), 0);
    auto key = [&](size_t l, int32_t i) { return site_order_key(lists[l].xy[(size_t)i * lists[l].stride]); };
    double done = 0;
    int k = 1; // the next cut
    auto goal = [&]() { return total * k / parts; };
    auto cut = [&]() {
        for (size_t l = 0; l < lists.size(); l++) cuts[l][(size_t)k] = at[l];
        k++;
    };
    while (k <= parts)
    {
        // (the last cut takes what is left)
        while (k < parts && done >= goal()) cut();
        // the list whose next cell comes first, and the first cell of the others
        size_t best = lists.size(), next = lists.size();
        for (size_t l = 0; l < lists.size(); l++)
        {
            if (at[l] >= lists[l].n) continue;
            if (best == lists.size() || key(l, at[l]) < key(best, at[best]))
            {
                next = best;
                best = l;
            }
            else if (next == lists.size() || key(l, at[l]) < key(next, at[next])) next = l;
        }
        if (best == lists.size())
        {
            while (k <= parts) cut();
            break;
        }
        const ShareList &l = lists[best];
        int32_t end = at[best] + 1;
        if (next == lists.size()) end = l.n;
        else
        {
            const uint32_t limit = key(next, at[next]);
            while (end < l.n && key(best, end) < limit) end++;
        }
        while (at[best] < end)
        {
            int32_t take = end - at[best];
            if (k < parts && done + take * l.weight >= goal())
            {
                // the fewest cells that reach the goal
                take = std::max(1, std::min(take, (int32_t)((goal() - done) / l.weight)));
                while (done + take * l.weight < goal()) take++;
                while (take > 1 && done + (take - 1) * l.weight >= goal()) take--;
            }
            at[best] += take;
            done += take * l.weight;
            while (k < parts && done >= goal()) cut();
        }
    }
    return cuts;
}
} // namespace mantiis
