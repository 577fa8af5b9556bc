// The transforms' signed arithmetic (ntt_arith.cuh) at and around the ends of
// its stated ranges: residues against 128-bit arithmetic, results inside the
// stated ranges.  Compiled with the signed-overflow sanitizer.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "ntt_arith.cuh"

using namespace pcgb;

namespace {

using I = __int128;
constexpr double kE = 0.05;

std::mt19937_64 rng(20240607);

void expect(bool ok, const char* what) {
    if (ok) return;
    std::fprintf(stderr, "FAILED: %s\n", what);
    std::exit(1);
}
int64_t at(double f) { return static_cast<int64_t>(static_cast<long double>(f) * kPs); }
// A value in [lo p, hi p]: either end, next to it, or anywhere.
int64_t pick(double lo, double hi) {
    const int64_t a = at(lo), b = at(hi);
    const uint64_t span = static_cast<uint64_t>(b) - static_cast<uint64_t>(a);
    switch (rng() % 4) {
        case 0: return a + static_cast<int64_t>(rng() % 3);
        case 1: return b - static_cast<int64_t>(rng() % 3);
        default:
            return static_cast<int64_t>(static_cast<uint64_t>(a) + rng() % (span + 1));
    }
}
uint64_t factor() {
    constexpr uint64_t h = kPm / 2;
    switch (rng() % 4) {
        case 0: return (h - 1 + rng() % 4) % kPm;
        case 1: return rng() % 2 ? rng() % 4 : kPm - 1 - rng() % 4;
        default: return rng() % kPm;
    }
}
uint64_t mod(I v) {
    I r = v % static_cast<I>(kPm);
    return static_cast<uint64_t>(r < 0 ? r + kPm : r);
}
bool in(int64_t v, double lo, double hi) { return v >= at(lo) - 8 && v <= at(hi) + 8; }

void forward(CtKind kind, double lo, double hi, double olo, double ohi) {
    int64_t X = pick(lo, hi), Y = pick(-1.7, 1.7);
    const int64_t x = X, y = Y;
    const uint64_t w = factor();
    ct_bfly(X, Y, ntt_tw_host(w), kind);
    expect(mod(X) == mod(x + static_cast<I>(mod(y)) * w), "forward sum");
    expect(mod(Y) == mod(x - static_cast<I>(mod(y)) * w), "forward difference");
    expect(in(X, olo, ohi) && in(Y, kind == kCtFold ? -ohi : olo, kind == kCtFold ? -olo : ohi),
           "forward range");
}

}  // namespace

int main() {
    for (int k = 0; k < 400000; ++k) {
        forward(kCtFirst, -kE, 1 + kE, -1 - 2 * kE, 1 + 2 * kE);
        forward(kCtFold, -1.75, 1.75, -0.5 - kE, 1.5 + kE);
        forward(kCtXRole, -0.5 - kE, 1.5 + kE, -1.5 - 2 * kE, 1.5 + 2 * kE);
        forward(kCtYRole, -1.5 - kE, 0.5 + kE, -1.5 - 2 * kE, 1.5 + 2 * kE);

        int64_t X = pick(-0.25, 1.25), Y = pick(-0.25, 1.25);
        const int64_t x = X, y = Y;
        const uint64_t w = factor();
        gs_bfly(X, Y, ntt_tw_host(w));
        expect(mod(X) == mod(static_cast<I>(x) + y), "inverse sum");
        expect(mod(Y) == mod(static_cast<I>(mod(static_cast<I>(x) - y)) * w), "inverse difference");
        expect(in(X, -1e-6, 1 + 1e-6) && in(Y, -kE, 1 + kE), "inverse range");

        int64_t U = pick(-kE, 1 + kE), V = pick(-kE, 1 + kE);
        const int64_t u = U, v = V;
        add_sub_bfly(U, V);
        expect(mod(U) == mod(static_cast<I>(u) + v) && mod(V) == mod(static_cast<I>(u) - v),
               "root-free butterfly");
        expect(in(U, -1 - 2 * kE, 1 + 2 * kE) && in(V, -1 - 2 * kE, 1 + 2 * kE),
               "root-free range");

        // Two raw words; two products of the multiply-accumulate.
        const uint64_t r0 = rng() % 2 ? ~uint64_t{0} - rng() % 3 : rng(), r1 = ~(rng() >> (rng() % 64));
        const int64_t s = fold(add_shift(fold_raw(r0), fold_raw(r1)));
        expect(mod(s) == mod(static_cast<I>(r0) + r1) && in(s, -1e-6, 1 + 1e-6), "raw sum");
        const int64_t a = pick(-0.17, 1.17), b = pick(-0.17, 1.17), f = fold(add_shift(a, b));
        expect(mod(f) == mod(static_cast<I>(a) + b) && in(f, -1e-6, 1 + 1e-6), "product sum");
        const int64_t g = pick(-1.7, 1.7), h = pick(-1.7, 1.7), m = mul_var(g, h);
        expect(mod(m) == mod(static_cast<I>(mod(g)) * mod(h)) && in(m, -0.17, 1.17), "product");
        expect(canon(m) == mod(m), "residue");
    }
    return 0;
}
