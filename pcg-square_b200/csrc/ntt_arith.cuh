// Signed lazy arithmetic of the NTT passes, mod p = 2^62 - d, d = 3*2^25 - 1.
//
// B200 issues a 32x32+64 -> 64-bit multiply-add (IMAD.WIDE) at 32 lanes a
// cycle and SM, half the rate of a 32-bit IMAD, and the NTT is bound by that
// pipe, so a product by a fixed w is built from five of them instead of the
// six IMAD.WIDE and four IMAD of a Shoup product (two 64-bit low products
// and a high one):
//
//   a*w = ah*w1 + al*w0,  a = ah*2^32 + al,  w0 = w, w1 = w*2^32 mod p
//
// with al and the low words of w0 and w1 taken as signed 32-bit values and
// w0, w1 in [-p/2, p/2).  The sum is below 2^94, so its part above bit 62 is
// a signed 32-bit word and folds back with one multiply by d (2^62 = d mod
// p).  Result: below 2^62 + 2^58, above -2^58, for any |a| < 2^63 - 2^32.
//
// Bounds.  |al|, |low words| <= 2^31, |ah| <= |a|/2^32 + 1 =: 2^31 A with
// A < 1, |high words| <= 2^29 (p/2 < 2^61).  L = al*w0l + ah*w1l is below
// 2^62 (1 + A) < 2^63; M = al*w0h + ah*w1h + (L >> 32) below 2^60 (1 + A) +
// 2^31 < 2^61, so M >> 30 fits 32 bits; times d < 2^26.6 it adds at most
// 2^57.6 to the 62-bit remainder.
//
// Values between butterflies are signed 64-bit with |v| <= 1.7p, inside the
// range of mul_tw and mul_var.  fold() brings one back to [0, p] up to 2d with one
// IMAD.WIDE.
#ifndef PCGB_NTT_ARITH_CUH_
#define PCGB_NTT_ARITH_CUH_

#include <cstdint>

#include "field.cuh"

namespace pcgb {

constexpr int kDelta = 3 * (1 << 25) - 1;
static_assert((uint64_t{1} << 62) - kPm == static_cast<uint64_t>(kDelta), "2^62 = d mod p");
constexpr int64_t kPs = static_cast<int64_t>(kPm);

// A fixed factor w: (low, high) words of w0 and of w1.
struct alignas(16) NttTw {
    int32_t w0l, w0h, w1l, w1h;
};

// c centred to [-p/2, p/2), then split with a signed low word.
PCGB_HD void split_centred(uint64_t c, int32_t* lo, int32_t* hi) {
    const int64_t s = c > kPm / 2 ? static_cast<int64_t>(c) - kPs : static_cast<int64_t>(c);
    *lo = static_cast<int32_t>(static_cast<uint32_t>(s));
    *hi = static_cast<int32_t>((s - *lo) >> 32);
}
// From w and w * 2^32 mod p, both in [0, p).
PCGB_HD NttTw ntt_tw(uint64_t w, uint64_t w32) {
    NttTw t;
    split_centred(w, &t.w0l, &t.w0h);
    split_centred(w32, &t.w1l, &t.w1h);
    return t;
}
inline NttTw ntt_tw_host(uint64_t w) { return ntt_tw(w, mul_p_host(w, uint64_t{1} << 32)); }

// One IMAD.WIDE with its 64-bit addend.  The product is written out because a
// 64-bit C product of words taken out of 64-bit values compiles to a full
// 64x64 multiply; the add stays a C add, which fuses into the same
// instruction (mad.wide.s32 spelled out kept extra moves: 23 instructions a
// butterfly against 19).
PCGB_HD int64_t wide_mad(int32_t a, int32_t b, int64_t c) {
#if defined(__CUDA_ARCH__)
    int64_t r;
    asm("mul.wide.s32 %0, %1, %2;" : "=l"(r) : "r"(a), "r"(b));
    return r + c;
#else
    return static_cast<int64_t>(a) * b + c;
#endif
}
// 62-bit remainder hi30:lo32 of a split sum as a 64-bit word.
PCGB_HD int64_t rem62(uint32_t hi, uint32_t lo) {
    return static_cast<int64_t>((static_cast<uint64_t>(hi & 0x3FFFFFFFu) << 32) | lo);
}
// The high word of the split with a signed low word.
PCGB_HD int32_t balanced_hi(int64_t a) {
    return static_cast<int32_t>((a >> 32) + (static_cast<uint32_t>(a) >> 31));
}

// a*w mod p, in (-2^58, 2^62 + 2^58).
PCGB_HD int64_t mul_tw(int64_t a, const NttTw& w) {
    const int32_t al = static_cast<int32_t>(static_cast<uint32_t>(a)), ah = balanced_hi(a);
    const int64_t L = wide_mad(ah, w.w1l, wide_mad(al, w.w0l, 0));
    const int64_t M = wide_mad(ah, w.w1h, wide_mad(al, w.w0h, L >> 32));
    return wide_mad(static_cast<int32_t>(M >> 30), kDelta,
                    rem62(static_cast<uint32_t>(M), static_cast<uint32_t>(L)));
}

// v mod p for |v| < 2p, in [-2d, 2^62 + d].
PCGB_HD int64_t fold(int64_t v) {
    const int32_t hi = static_cast<int32_t>(v >> 32);
    return wide_mad(hi >> 30, kDelta, rem62(static_cast<uint32_t>(hi), static_cast<uint32_t>(v)));
}

// v mod p for |v| < 1.75p, centred: in [-p/2, p/2] up to 2d.
PCGB_HD int64_t fold_centred(int64_t v) {
    const uint32_t hi = static_cast<uint32_t>(static_cast<uint64_t>(v) >> 32);
    const int32_t h = ((static_cast<int32_t>(hi) >> 29) + 1) >> 1;
    const uint64_t rem = (static_cast<uint64_t>(hi - (static_cast<uint32_t>(h) << 30)) << 32) |
                         static_cast<uint32_t>(v);
    return wide_mad(h, kDelta, static_cast<int64_t>(rem));
}

// v mod p for any unsigned 64-bit v, in [0, 2^62 + 3d].
PCGB_HD int64_t fold_raw(uint64_t v) {
    const uint32_t hi = static_cast<uint32_t>(v >> 32);
    return wide_mad(static_cast<int32_t>(hi >> 30), kDelta, rem62(hi, static_cast<uint32_t>(v)));
}

// a*b mod p for |a|, |b| <= 1.7p, in (-0.17p, 1.17p): the full product in
// balanced 32-bit words, its part above bit 64 folded with 2^64 = 4d, then the
// part above bit 62 in two pieces (it has up to 34 bits).  With |ah|, |bh| <=
// 0.85*2^31: |M| <= 2*0.85*2^62 + 2^58 + 2^31 < 2^63, and its high word times 4d
// is below 0.17p.
PCGB_HD int64_t mul_var(int64_t a, int64_t b) {
    const int32_t al = static_cast<int32_t>(static_cast<uint32_t>(a)), ah = balanced_hi(a);
    const int32_t bl = static_cast<int32_t>(static_cast<uint32_t>(b)), bh = balanced_hi(b);
    const int64_t C2 = wide_mad(ah, bh, 0);
    const int32_t c2l = static_cast<int32_t>(static_cast<uint32_t>(C2)), c2h = balanced_hi(C2);
    const int64_t L = wide_mad(c2l, 4 * kDelta, wide_mad(al, bl, 0));
    const int64_t M = wide_mad(c2h, 4 * kDelta, wide_mad(al, bh, wide_mad(ah, bl, L >> 32)));
    const uint32_t ml = static_cast<uint32_t>(M);
    const int64_t r = rem62(ml, static_cast<uint32_t>(L)) +
                      static_cast<int64_t>((ml >> 30) * static_cast<uint32_t>(kDelta));
    return wide_mad(static_cast<int32_t>(M >> 32), 4 * kDelta, r);
}

// The residue in [0, p) of v in (-p, 2p).
PCGB_HD uint64_t canon(int64_t v) {
    uint64_t u = static_cast<uint64_t>(v + ((v >> 63) & kPs));
    return u >= kPm ? u - kPm : u;
}

// ---- butterflies -------------------------------------------------------------
// Values are signed and lazily reduced: a product t lies in [-e p, (1 + e)p],
// e < 0.05, for a factor of at most 1.7p in magnitude.

// a + b - p for values whose plain sum may pass 2^63: 2p is only 2d below it.
// (Here and in the butterflies p goes in before the second operand, so that no
// intermediate leaves the signed range.)
PCGB_HD int64_t add_shift(int64_t a, int64_t b) { return a - kPs + b; }

// Forward butterfly X + wY, X - wY.  A stage with FOLD brings X back first;
// the next one adds another product to that, shifted by p so that the range
// stays centred, which needs the role the element had in the last stage:
//   FIRST  X in [-e, 1 + e]p           -> both within (1 + 2e)p
//   FOLD   |X| < 1.75p, folded to +-p/2 -> X' in [-1/2 - e, 3/2 + e]p, Y' in
//                                         its negative
//   XROLE  X an X' of a FOLD stage     -> both within (1.5 + 2e)p
//   YROLE  X a Y' of a FOLD stage      -> both within (1.5 + 2e)p
enum CtKind { kCtFirst, kCtFold, kCtXRole, kCtYRole };
PCGB_HD void ct_bfly(int64_t& X, int64_t& Y, const NttTw& w, CtKind kind) {
    const int64_t x = kind == kCtFold ? fold_centred(X) : X;
    const int64_t t = mul_tw(Y, w);
    X = (kind == kCtFirst || kind == kCtXRole) ? add_shift(x, t) : x + t;
    Y = kind == kCtYRole ? x + kPs - t : x - t;
}
// Stage q of a phase starting at stage s0: phase 0 begins on reduced values
// and folds at q = 1, 3; later phases fold at q = 0, 2.  xrole: the X operand
// was an X' of the previous stage.
#if defined(__CUDACC__)
__host__ __device__
#endif
constexpr CtKind ct_kind(int s0, int q, bool xrole) {
    if (s0 + q == 0) return kCtFirst;
    if ((q & 1) == (s0 == 0 ? 1 : 0)) return kCtFold;
    return xrole ? kCtXRole : kCtYRole;
}

// Inverse butterfly: X, Y in [-0.25p, 1.25p] -> X + Y in [0, p] up to 2d,
// (X - Y) w in [-e p, (1 + e)p].
PCGB_HD void gs_bfly(int64_t& X, int64_t& Y, const NttTw& w) {
    const int64_t s = fold(add_shift(X, Y));
    Y = mul_tw(X - Y, w);
    X = s;
}

// Butterfly of a stage whose root has been folded into the per-element
// twiddles (the row pass's first forward stage and last inverse stage):
// X, Y in [-e p, (1 + e)p] -> X + Y, X - Y within (1 + 2e)p.
PCGB_HD void add_sub_bfly(int64_t& X, int64_t& Y) {
    const int64_t s = add_shift(X, Y);
    Y = X - Y;
    X = s;
}

}  // namespace pcgb

#endif
