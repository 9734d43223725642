"""Groups of a batch's images for the cooperative launches (coop_groups.hpp), with a
plan that only notes which images it is of: sizes, images that fit no plan, and a
plan that cannot be made, after which the batch holds no group at all."""
import shutil
import subprocess

import pytest
from conftest import ROOT

SOURCE = r"""
#include <cstdio>
#include <stdexcept>
#include "mantiis_gb300/csrc/solver/coop_groups.hpp"
struct Plan { size_t first, count; bool ok; };
typedef std::vector<std::unique_ptr<Plan>> Groups;
// plans of up to four images, none of an image of 1000 bytes; the k-th build throws
static Groups make(const std::vector<int64_t> &bytes, int64_t most, int throws_at)
{
    int builds = 0;
    return mantiis::coop_groups<Plan>(bytes, most, [&](size_t first, size_t count) {
        if (++builds == throws_at) throw std::runtime_error("build");
        bool ok = count <= 4;
        for (size_t i = first; i < first + count; i++) ok = ok && bytes[i] != 1000;
        return std::unique_ptr<Plan>(new Plan{first, count, ok});
    });
}
static void show(const Groups &g)
{
    for (auto &p : g) std::printf("%zu+%zu%s ", p->first, p->count, p->ok ? "" : "!");
    std::printf("\n");
}
int main()
{
    show(make({1, 2, 3}, 10, 0));
    show(make({4, 4, 4, 20, 1, 1}, 8, 0));
    show(make({1, 1, 1, 1, 1, 1, 1, 1, 1}, 100, 0));
    show(make({1000, 1, 1000, 2}, 5000, 0));
    show(make({}, 1, 0));
    show(make({5, 5, 5, 5, 5, 5}, 24, 0)); // 4 + 2 -> 3 + 3
    show(make({9, 1, 1, 1, 1, 1, 1}, 12, 0));
    show(make({2, 3, 4, 5, 6, 7}, 14, 0));
    Groups held; // as the batch holds them: none until a build of every one succeeds
    int thrown = 0;
    for (int k = 1; held.empty() && k < 1000; k++)
        try { held = make({4, 4, 4, 4, 4}, 8, k); } catch (const std::runtime_error &) { thrown++; }
    std::printf("%s %zu", thrown >= 5 ? "thrown" : "", held.size());
    std::printf("\n");
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_groups(tmp_path):
    (tmp_path / "groups.cpp").write_text(SOURCE)
    exe = tmp_path / "groups"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Werror", "-I", ROOT, tmp_path / "groups.cpp", "-o", exe], check=True)
    lines = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.splitlines()
    assert [l.strip() for l in lines] == [
        "0+3",
        "0+2 2+1 3+1 4+2",
        "0+3 3+3 6+3",
        "0+1! 1+1 2+1! 3+1",
        "",
        "0+3 3+3",
        "0+3 3+4",
        "0+4 4+2",
        "thrown 3",
    ]
