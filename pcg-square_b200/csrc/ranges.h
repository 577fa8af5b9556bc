// Byte ranges of buffers, and whether they meet.
#ifndef PCGB_RANGES_H_
#define PCGB_RANGES_H_

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace pcgb {

struct Range {
    uintptr_t lo = 0, hi = 0;   // [lo, hi)
};
inline Range range_of(const void* p, size_t bytes) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(p);
    return Range{at, at + bytes};
}
inline bool overlap(const Range& a, const Range& b) {
    return a.lo < b.hi && b.lo < a.hi && a.lo < a.hi && b.lo < b.hi;
}
// Whether any of a meets any of b, in n log n.
inline bool any_overlap(const std::vector<Range>& a, std::vector<Range> b) {
    b.erase(std::remove_if(b.begin(), b.end(), [](const Range& r) { return r.lo == r.hi; }), b.end());
    std::sort(b.begin(), b.end(), [](const Range& x, const Range& y) { return x.lo < y.lo; });
    // Furthest end of the ranges that start at or before each one.
    std::vector<uintptr_t> end(b.size());
    for (size_t i = 0; i < b.size(); ++i) end[i] = i ? std::max(end[i - 1], b[i].hi) : b[i].hi;
    for (const Range& r : a) {
        if (r.lo == r.hi) continue;
        const auto it = std::lower_bound(b.begin(), b.end(), r.hi,
                                         [](const Range& x, uintptr_t v) { return x.lo < v; });
        if (it != b.begin() && end[it - b.begin() - 1] > r.lo) return true;
    }
    return false;
}

}  // namespace pcgb

#endif
