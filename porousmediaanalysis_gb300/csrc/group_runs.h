// Runs of tile groups whose lists fit a memory budget (containing_balls).
#pragma once

#include <algorithm>
#include <cstddef>

namespace pma {

// End of the run that starts at group g0: at most `end`, and its lists hold at most `budget` entries
// unless one group's alone hold more. Groups come in layers of per_layer; layers[z] is the offset of
// layer z's first entry (and one more, the total). Whole layers are taken where one fits; else a part
// of the layer, cut by the offsets of its groups: group_offsets(z) gives those of layer z's groups and
// the next layer's first, and is only asked for where a layer is cut.
template <class GroupOffsets>
size_t group_run_end(const unsigned long long* layers, size_t per_layer, size_t g0, size_t end, unsigned long long budget,
                     GroupOffsets group_offsets) {
    const size_t z = g0 / per_layer, first = z * per_layer;
    if (g0 == first) {
        size_t to = z;
        while ((to + 1) * per_layer <= end && layers[to + 1] - layers[z] <= budget) ++to;
        if (to > z) return to * per_layer;
    }
    const unsigned long long* groups = group_offsets(z);
    const unsigned long long* beyond = std::upper_bound(groups + (g0 - first) + 1, groups + std::min(per_layer, end - first) + 1,
                                                        groups[g0 - first] + budget);
    return std::max(first + static_cast<size_t>(beyond - groups) - 1, g0 + 1);
}

}  // namespace pma
