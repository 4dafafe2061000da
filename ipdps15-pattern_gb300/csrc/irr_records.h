// irr_records.h -- whether a kernel may read the caller's node records in place
// (plain C++: the rule is tested without a GPU).
#pragma once
#include <cstdint>

namespace irr {

// What the driver says of an address.
struct PointerFacts {
    bool device = false;       // device or managed memory
    bool managed = false;
    int ordinal = -1;          // its device
    uint64_t address = 0;      // as the device addresses it
    uint64_t range_start = 0;  // the allocation it lies in
    uint64_t range_size = 0;
};

// Records of elm (12, 16 or 24) bytes, `bytes` in all, at p, for kernels on
// device `ordinal`: its own memory (or managed memory) at the same address, the
// alignment that their loads want, and all of it in one allocation.  Anything
// else (another GPU's memory, host memory, a range that ends too soon) goes
// through the staging copy, where the runtime copies or refuses it.
inline bool records_in_place(uint64_t p, int elm, uint64_t bytes, int ordinal, const PointerFacts& f)
{
    const uint64_t align = elm == 12 ? 4 : (elm == 16 ? 16 : 8);
    if (p % align || !f.device || f.address != p) return false;
    if (!f.managed && f.ordinal != ordinal) return false;
    return f.range_start <= p && p - f.range_start <= f.range_size && f.range_size - (p - f.range_start) >= bytes;
}

}  // namespace irr
