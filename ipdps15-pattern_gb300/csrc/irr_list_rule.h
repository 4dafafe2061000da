// irr_list_rule.h -- how many slots per node a neighbour list's one-pass search
// takes (plain C++: the rule is tested without a GPU).
#pragma once
#include <cstdint>

namespace irr {

// sphere: the nodes of the mean list sphere.  A third more than these and some
// (a multiple of 8), 0 where the search counts first: above `most` slots, or
// where all of them do not fit 32 bits, in which the list's offsets are summed.
inline uint32_t list_slots(double sphere, int64_t n, int most)
{
    if (!(sphere < most)) return 0;
    const uint32_t cap = ((uint32_t)(1.35 * sphere) + 31u) / 8u * 8u;
    return cap <= (uint32_t)most && (double)cap * (double)n < 4294967296.0 ? cap : 0u;
}

}  // namespace irr
