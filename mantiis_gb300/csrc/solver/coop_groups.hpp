// Consecutive images of a batch in groups, one cooperative launch each.
#pragma once
#include <algorithm>
#include <cstdint>
#include <memory>
#include <utility>
#include <vector>

namespace mantiis
{
// As many images together as their bytes stay within `most` and build(first, count)
// gives a plan that is ok (it fits the kernel's tables); an image that no plan fits
// is a group of its own, not ok.
template <typename Plan, typename Build>
std::vector<std::unique_ptr<Plan>> greedy_groups(const std::vector<int64_t> &bytes, int64_t most, Build build)
{
    std::vector<std::unique_ptr<Plan>> groups;
    std::unique_ptr<Plan> plan; // of the images first .. i - 1
    size_t first = 0;
    int64_t sum = 0;
    for (size_t i = 0; i < bytes.size(); i++)
    {
        sum += bytes[i];
        std::unique_ptr<Plan> more;
        if (!plan || sum <= most) more = build(first, i + 1 - first);
        if (plan && (!more || !more->ok))
        {
            // the group ends before this image
            groups.push_back(std::move(plan));
            first = i;
            sum = bytes[i];
            more = build(first, 1);
        }
        plan = std::move(more);
    }
    if (plan) groups.push_back(std::move(plan));
    return groups;
}

// As few groups as that, of sizes as equal as a lower limit makes them: a group's
// stages wait for the slowest SM and for two barriers whatever its size, so one image
// left over costs as much as four (eight 512^2 images of two levels in groups of
// 7 + 1 / 4 + 4: 122 / 91 us per coarse step).  The groups come as one value: where
// build throws, the caller has none of them, not the first few.
template <typename Plan, typename Build>
std::vector<std::unique_ptr<Plan>> coop_groups(const std::vector<int64_t> &bytes, int64_t most, Build build)
{
    std::vector<std::unique_ptr<Plan>> groups = greedy_groups<Plan>(bytes, most, build);
    const size_t count = groups.size();
    if (count < 2 || count == bytes.size()) return groups;
    for (const auto &g : groups)
        if (!g->ok) return groups;
    int64_t total = 0;
    for (int64_t v : bytes) total += v;
    int64_t low = (total - 1) / (int64_t)count, high = most; // low: too little for `count` groups
    for (int tries = 0; tries < 5 && low < high - high / 16; tries++)
    {
        // first the limit that equal groups have
        const int64_t limit = tries == 0 ? low + 1 : low + (high - low) / 2;
        std::vector<std::unique_ptr<Plan>> even = greedy_groups<Plan>(bytes, limit, build);
        if (even.size() <= count)
        {
            groups = std::move(even);
            high = limit;
        }
        else low = limit;
    }
    return groups;
}
} // namespace mantiis
