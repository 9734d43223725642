// Consecutive images of a batch in groups, one cooperative launch each.
#pragma once
#include <cstdint>
#include <memory>
#include <utility>
#include <vector>

namespace mantiis
{
// As many images together as their bytes stay within `most` and build(first, count)
// gives a plan that is ok (it fits the kernel's tables); an image that no plan fits
// is a group of its own, not ok.  The groups come as one value: where build throws,
// the caller has none of them, not the first few.
template <typename Plan, typename Build>
std::vector<std::unique_ptr<Plan>> coop_groups(const std::vector<int64_t> &bytes, int64_t most, Build build)
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
} // namespace mantiis
