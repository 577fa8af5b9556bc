// any_overlap against all pairs, on small random sets with empty, nested,
// touching and equal ranges.
#include <cstdio>
#include <random>

#include "ranges.h"

int main() {
    std::mt19937 rng(7);
    int met = 0;
    for (int k = 0; k < 200000; ++k) {
        std::vector<pcgb::Range> a(rng() % 4), b(rng() % 6);
        for (auto* v : {&a, &b})
            for (auto& r : *v) {
                const char* p = reinterpret_cast<const char*>(static_cast<uintptr_t>(rng() % 60));
                r = pcgb::range_of(p, rng() % 9);
            }
        bool want = false;
        for (const auto& x : a)
            for (const auto& y : b) {
                bool both = false;
                for (uintptr_t i = x.lo; i < x.hi; ++i) both = both || (i >= y.lo && i < y.hi);
                if (pcgb::overlap(x, y) != both) return std::puts("overlap"), 1;
                want = want || both;
            }
        if (pcgb::any_overlap(a, b) != want) return std::puts("any_overlap"), 1;
        met += want;
    }
    return met > 1000 ? 0 : 1;
}
