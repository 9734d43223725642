"""Equal shares of several lists of cells (share_cuts.hpp) against the definition, cell
by cell: random lists, empty ones, fewer cells than shares, weights of the solver's."""
import shutil
import subprocess

import pytest
from conftest import ROOT

SOURCE = r"""
#include <cstdio>
#include <random>
#include "mantiis_gb300/csrc/solver/share_cuts.hpp"
using namespace mantiis;
typedef std::vector<std::vector<int32_t>> Cuts;
// the cells one after the other in the order of all lists
static Cuts plain(const std::vector<ShareList> &lists, int parts)
{
    double total = 0, done = 0;
    for (auto &l : lists) total += l.weight * l.n;
    Cuts cuts(lists.size(), std::vector<int32_t>(parts + 1, 0));
    std::vector<int32_t> at(lists.size(), 0);
    for (int k = 1; k <= parts; k++)
    {
        while (k == parts || done < total * k / parts)
        {
            int best = -1;
            for (size_t l = 0; l < lists.size(); l++)
                if (at[l] < lists[l].n && (best < 0 || site_order_key(lists[l].xy[(size_t)at[l] * lists[l].stride]) <
                                                           site_order_key(lists[best].xy[(size_t)at[best] * lists[best].stride])))
                    best = (int)l;
            if (best < 0) break;
            at[best]++;
            done += lists[best].weight;
        }
        for (size_t l = 0; l < lists.size(); l++) cuts[l][k] = at[l];
    }
    return cuts;
}
int main()
{
    std::mt19937 rng(3);
    const double weights[4] = {3.0, 1.5, 1.0, 1.0};
    int wrong = 0, cases = 0;
    for (int t = 0; t < 400; t++)
    {
        const int side = 1 + (int)(rng() % (t < 100 ? 4 : 90)), parts = 1 + (int)(rng() % 160), strides[4] = {8, 8, 1, 1};
        std::vector<int32_t> xy[4];
        for (int y = 0; y < side; y++)
            for (int x = 0, run = 0, l = 0; x < side; x++, run--)
            {
                if (run <= 0)
                {
                    l = (int)(rng() % 5); // 4: no cell
                    run = 1 + (int)(rng() % (t % 2 ? 3 : 40));
                }
                if (l == 4 || (t % 7 == 0 && l < 2)) continue;
                xy[l].push_back(x | y << 16);
                for (int s = 1; s < strides[l]; s++) xy[l].push_back(-1); // a record's other words
            }
        std::vector<ShareList> lists;
        for (int l = 0; l < 4; l++) lists.push_back({xy[l].data(), (int32_t)(xy[l].size() / strides[l]), strides[l], weights[l]});
        wrong += share_cuts(lists, parts) != plain(lists, parts);
        cases++;
    }
    std::printf("%d of %d wrong\n", wrong, cases);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_cuts(tmp_path):
    (tmp_path / "cuts.cpp").write_text(SOURCE)
    exe = tmp_path / "cuts"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-D_GLIBCXX_ASSERTIONS", "-I", ROOT,
                    tmp_path / "cuts.cpp", "-o", exe], check=True)
    assert subprocess.run([exe], check=True, capture_output=True, text=True).stdout == "0 of 400 wrong\n"
