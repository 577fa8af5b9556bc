// Negacyclic NTT over F_p for N = 2^logN (1 <= logN <= 24): one row up to
// 2^9 (N = n2, n1 = 1, a single CTA per transform), four-step above.
//
// N = n1 * n2 with n1 = 2^floor(logN/2), n2 = 2^ceil(logN/2); coefficient j
// sits at row j / n2, column j % n2.  With psi a primitive 2N-th root:
//   column pass: negacyclic NTT of length n1 on every column (root
//                psi1 = psi^n2);
//   row pass:    multiply element (k, j2) by the twiddle
//                psi^(j2 * (2*i1 + 1 - n1)), i1 = brev(k), then a
//                negacyclic NTT of length n2 on every row (root psi2 =
//                psi^n1).  The row transform's first stage has a single
//                root w0; it is folded into the twiddles of the row's upper
//                half, so that stage only adds and subtracts.
// Element (k, k2) then holds A(psi^(2*(i1 + n1*i2) + 1)) with i1 = brev(k),
// i2 = brev(k2): the evaluations of a(x) mod x^N + 1.  The row pass stores
// its outputs in a fixed permuted order (below) that every operand of a
// pointwise product shares; the inverse runs the passes backwards with
// inverse roots and folds N^-1 into its twiddle.
//
// Each sub-transform is the merged-twist Cooley-Tukey (forward) /
// Gentleman-Sande (inverse) negacyclic NTT of Longa and Naehrig (CANS 2016,
// Algorithms 1-2).  Values are signed and lazily reduced: |v| <= 1.7p < 2^63,
// with products by table entries in (-0.05p, 1.05p) (ntt_arith.cuh).  What
// bounds the passes is the multiplier pipe together with the register ports
// it shares with the integer ALU: a butterfly is about 19 instructions (5
// IMAD.WIDE for the product, one for the fold of the other operand) and 37
// cycles a warp and sub-partition, against 26 instructions and 47 cycles for
// Shoup products with Harvey's [0, 4p) ranges (a loop of radix-16 phases in
// registers).  Sixteen products of 2^20 together with the launches shared by
// both operands: 835 -> 753 us.
//
// Register blocking.  A thread owns E = 16 elements of one sub-transform of
// length n = 2^L (all n when n < 16), so T = n / 16 threads share it.  The L
// stages run in phases of four (radix 16) entirely in registers; between
// phases the elements are exchanged through shared memory.  In phase P
// (first stage s0 = 4P, r = min(4, L - s0) stages) a unit is the 2^r
// elements g*2^(L-s0) + j + k*tl (tl = 2^(L-s0-r), k < 2^r) that the phase
// combines; thread t owns units t*U .. t*U+U-1 (U = 16 / 2^r), unit u = (g,
// j) with g = u / tl, j = u % tl.  Phase 0 owns elements t + T*k, the last
// phase the 16 consecutive elements 16t .. 16t+15, so global loads and stores
// coalesce in both the column pass (lanes run over adjacent columns) and the
// row pass (lanes run over t).  Row-pass outputs of element i are stored at
// (i % 16) * T + i / 16 -- the permuted evaluation order.  Shared memory holds
// element i at (i + i/16) * stride, which keeps every exchange free of bank
// conflicts for the strides used here.
//
// The twiddle of stage s and butterfly group i = g*2^q + sub (q = s - s0) is
// stored at 2^s + sub*2^s0 + g, so the lanes of a warp read the same or
// adjacent table entries in every phase.
//
// The passes are two HBM sweeps per transform; the pointwise product with a
// resident operand and the multiply-accumulate over several transforms are
// fused into the row pass, where the forward phases end in the same register
// layout the inverse phases start from.  Replaces the reference's radix-2
// per-stage v1 kernels (GPU_baseline/common/poly_mul_cuda.cu:137-200) and its
// 20-kernel four-step (poly_mul_gpuntt_square.cu:171-613).
#include "pcgb_internal.h"

#include <algorithm>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <type_traits>
#include <vector>

#include "chain.cuh"
#include "field.cuh"
#include "ntt_arith.cuh"
#include "ranges.h"

namespace pcgb {

struct NttPlan {
    int logN = 0, l1 = 0, l2 = 0;
    size_t N = 0;
    int n1 = 0, n2 = 0;
    NttTw* tw1 = nullptr;    // column roots, phase-permuted (none when l1 = 0)
    NttTw* tw1i = nullptr;
    NttTw* tw2 = nullptr;    // row roots
    NttTw* tw2i = nullptr;
    // [n1][n2] four-step twiddles, the row transform's first (forward) / last
    // (inverse) root folded into the upper half of each row
    NttTw* Wf = nullptr;     // forward twiddle
    NttTw* Wif = nullptr;    // inverse twiddle * N^-1
    // The same three tables of the one-row form (tw2, tw2i, Wif themselves when
    // l1 = 0), up to kOneRowLogN: whole products in one launch
    NttTw* one_tw = nullptr;
    NttTw* one_twi = nullptr;
    NttTw* one_Wi = nullptr;
    bool direct() const { return l1 == 0; }   // one row: no column passes
};

namespace {

__device__ __forceinline__ NttTw ldtw(const NttTw* __restrict__ w) {
    const int4 v = __ldg(reinterpret_cast<const int4*>(w));
    return NttTw{v.x, v.y, v.z, v.w};
}

// ---- phase geometry ----------------------------------------------------------

template <int L>
struct Geo {
    static constexpr int n = 1 << L;
    static constexpr int E = L >= 4 ? 16 : n;         // elements per thread
    static constexpr int T = n / E;                    // threads per transform
    static constexpr int NPH = (L + 3) / 4;            // phases (0 when n = 1)
    static constexpr int PAD = n + n / 16;             // padded smem length
    __host__ __device__ static constexpr int r(int p) { return L - 4 * p < 4 ? L - 4 * p : 4; }
};

__host__ __device__ constexpr int last_phase(int L) { return L == 0 ? 0 : (L + 3) / 4 - 1; }

// Element index (within the transform) of register e of thread t in phase P.
template <int L, int P>
__device__ __forceinline__ int eidx(int t, int e) {
    constexpr int s0 = 4 * P, r = Geo<L>::r(P), U = Geo<L>::E >> r, ltl = L - s0 - r;
    const int v = e >> r, k = e & ((1 << r) - 1);
    const int u = t * U + v;
    return ((u >> ltl) << (L - s0)) + (u & ((1 << ltl) - 1)) + (k << ltl);
}

// Position of element i in the permuted row-output order.
template <int L>
__device__ __forceinline__ int perm_pos(int i) {
    if constexpr (L >= 4) return (i & 15) * Geo<L>::T + (i >> 4);
    else return i;
}

// FOLD: stage 0 (a single root) has that root folded into the per-element
// twiddles the caller applies (before the forward phases, after the inverse
// ones), so it is a plain add/sub; its inputs are in [0, 2p).
template <int L, int P, bool INV, bool FOLD>
__device__ __forceinline__ void run_phase(int64_t (&x)[Geo<L>::E], int t,
                                          const NttTw* __restrict__ tw) {
    constexpr int s0 = 4 * P, r = Geo<L>::r(P), U = Geo<L>::E >> r, ltl = L - s0 - r;
#pragma unroll
    for (int v = 0; v < U; ++v) {
        const int g = (t * U + v) >> ltl;
        const int o = v << r;
        if constexpr (!INV) {
#pragma unroll
            for (int q = 0; q < r; ++q) {
#pragma unroll
                for (int sub = 0; sub < (1 << q); ++sub) {
                    if (FOLD && s0 + q == 0) {
#pragma unroll
                        for (int kk = 0; kk < (1 << (r - 1)); ++kk)
                            add_sub_bfly(x[o + kk], x[o + kk + (1 << (r - 1))]);
                        continue;
                    }
                    const NttTw w = ldtw(tw + (1 << (s0 + q)) + (sub << s0) + g);
#pragma unroll
                    for (int kk = 0; kk < (1 << (r - 1 - q)); ++kk) {
                        const int k = o + (sub << (r - q)) + kk;
                        // k's bit of stage q - 1 tells its role there
                        const bool xrole = q == 0 || ((k >> (r - q)) & 1) == 0;
                        ct_bfly(x[k], x[k + (1 << (r - 1 - q))], w, ct_kind(s0, q, xrole));
                    }
                }
            }
        } else {
            // Gentleman-Sande: the same stages, last to first (an ascending
            // counter keeps the loop fully unrolled and x in registers).
#pragma unroll
            for (int qq = 0; qq < r; ++qq) {
                const int q = r - 1 - qq;
#pragma unroll
                for (int sub = 0; sub < (1 << q); ++sub) {
                    if (FOLD && s0 + q == 0) {
#pragma unroll
                        for (int kk = 0; kk < (1 << (r - 1)); ++kk)
                            add_sub_bfly(x[o + kk], x[o + kk + (1 << (r - 1))]);
                        continue;
                    }
                    const NttTw w = ldtw(tw + (1 << (s0 + q)) + (sub << s0) + g);
#pragma unroll
                    for (int kk = 0; kk < (1 << (r - 1 - q)); ++kk) {
                        const int k = o + (sub << (r - q)) + kk;
                        gs_bfly(x[k], x[k + (1 << (r - 1 - q))], w);
                    }
                }
            }
        }
    }
}

// Element i of one transform in shared memory: base[(i + i/16) * S].
template <int S>
struct SmemLay {
    int64_t* base;
    __device__ __forceinline__ int64_t& at(int i) const { return base[(i + (i >> 4)) * S]; }
};

// Registers in phase A layout -> shared memory -> registers in phase B
// layout.  CLEAN: no thread can still be reading the buffer (the first
// exchange of a kernel), so the leading barrier is left out.
template <int L, int A, int B, bool CLEAN, class Lay>
__device__ __forceinline__ void exchange(int64_t (&x)[Geo<L>::E], int t, const Lay& lay) {
    if constexpr (!CLEAN) __syncthreads();
#pragma unroll
    for (int e = 0; e < Geo<L>::E; ++e) lay.at(eidx<L, A>(t, e)) = x[e];
    __syncthreads();
#pragma unroll
    for (int e = 0; e < Geo<L>::E; ++e) x[e] = lay.at(eidx<L, B>(t, e));
}

// All forward phases: registers start in phase 0 layout, end in the last.
// CLEAN: as for exchange, of the first one.
template <int L, bool FOLD, bool CLEAN, int P = 0, class Lay>
__device__ __forceinline__ void forward_all(int64_t (&x)[Geo<L>::E], int t,
                                            const NttTw* __restrict__ tw, const Lay& lay) {
    if constexpr (P < Geo<L>::NPH) {
        if constexpr (P > 0) exchange<L, P - 1, P, CLEAN && P == 1>(x, t, lay);
        run_phase<L, P, false, FOLD>(x, t, tw);
        forward_all<L, FOLD, CLEAN, P + 1>(x, t, tw, lay);
    }
}

// All inverse phases: registers start in the last phase layout, end in phase 0.
template <int L, bool FOLD, bool CLEAN, int P = Geo<L>::NPH - 1, class Lay>
__device__ __forceinline__ void inverse_all(int64_t (&x)[Geo<L>::E], int t,
                                            const NttTw* __restrict__ twi, const Lay& lay) {
    if constexpr (P >= 0) {
        if constexpr (P < Geo<L>::NPH - 1)
            exchange<L, P + 1, P, CLEAN && P == Geo<L>::NPH - 2>(x, t, lay);
        run_phase<L, P, true, FOLD>(x, t, twi);
        inverse_all<L, FOLD, CLEAN, P - 1>(x, t, twi, lay);
    }
}

// ---- kernels -----------------------------------------------------------------

// Columns per CTA of the column passes.  Adjacent columns ride on adjacent
// lanes: 128-byte row segments up to n1 = 512, then 64, 32 and 16 bytes so
// that the CTA stays at 512 threads.  The column kernels are register-capped
// for 1024 threads per SM (64 registers), so one CTA's loads overlap another's
// butterflies.  A launch with too few tiles for the chip takes the narrower
// tiles of col_C_min (col_width).  (n2 >= n1 = 2^L, so C never exceeds the row
// length.)
__host__ __device__ constexpr int col_C(int L) {
    return L <= 3 ? (1 << L) : (L <= 9 ? 16 : (L == 10 ? 8 : (L == 11 ? 4 : 2)));
}
__host__ __device__ constexpr int col_C_min(int L) {
    return L >= 5 && L <= 10 ? 4 : col_C(L);
}
template <int L, int C>
__host__ __device__ constexpr int col_threads() { return Geo<L>::T * C; }
template <int L, int C>
__host__ __device__ constexpr int col_min_ctas() {
    return col_threads<L, C>() >= 64 ? 1024 / col_threads<L, C>() : 16;
}
// Transforms per CTA of the row passes (n1 >= 2^(L-1) rows exist).
template <int L>
__host__ __device__ constexpr int row_V() {
    constexpr int half = L >= 1 ? (1 << L) / 2 : 1;
    return Geo<L>::T >= 64 ? 1 : (64 / Geo<L>::T < half ? 64 / Geo<L>::T : half);
}
template <int L>
__host__ __device__ constexpr int row_threads() { return Geo<L>::T * row_V<L>(); }
// CTAs per SM the row kernels are compiled for: 768 threads (85 registers).
// 1024 threads (64 registers) are 2 % faster at 16 x 2^20 and 10 % slower
// where a pass is one short wave (2^13 .. 2^18).
template <int L>
__host__ __device__ constexpr int row_min_ctas() {
    return row_threads<L>() >= 64 ? 768 / row_threads<L>() + (row_threads<L>() > 768) : 12;
}

// Up to three transforms of one length and batch in one launch: transform z
// takes src[z] (plus add[z] when set) to dst[z].
struct FwdIn {
    const uint64_t* src[3] = {nullptr, nullptr, nullptr};
    const uint64_t* add[3] = {nullptr, nullptr, nullptr};
    uint64_t* dst[3] = {nullptr, nullptr, nullptr};
};
template <class T>
__device__ __forceinline__ T pick(T const (&v)[3], int z) {
    return z == 0 ? v[0] : (z == 1 ? v[1] : v[2]);
}

// ---- pass bodies ---------------------------------------------------------------
// Shared by the per-length kernels (one length, batch in gridDim.y) and the
// mixed-length kernels (a job table names each CTA's polynomial and tile).
// Pointers arrive already offset to the polynomial's first word.  Buffers
// between the passes of one transform hold signed lazy values.

// Any 64-bit word (plus another) as a residue in [0, p] up to 3d.
__device__ __forceinline__ int64_t load_raw(const uint64_t* src, const uint64_t* add, size_t i) {
    int64_t v = fold_raw(src[i]);
    if (add) v = fold(add_shift(v, fold_raw(add[i])));
    return v;
}

// Column pass, forward, for columns [tile*C, tile*C + C).  src may equal
// dst (every CTA loads its columns before its first store).  Inputs are any
// 64-bit words.  Outputs within 1.6p, without the four-step twiddle: the row pass
// applies it together with its own first root.  L2 fixes log2(n2) at compile time
// (element offsets become immediates).
template <int L, int C, int L2>
__device__ __forceinline__ void col_fwd_body(const uint64_t* src, const uint64_t* add,
                                             uint64_t* dst, size_t tile,
                                             const NttTw* __restrict__ tw, int64_t* sm) {
    constexpr int E = Geo<L>::E, LP = last_phase(L);
    const int t = threadIdx.x / C, c = threadIdx.x % C;
    constexpr size_t n2 = size_t{1} << L2;
    const size_t col = tile * C + c;
    int64_t x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = load_raw(src, add, col + eidx<L, 0>(t, e) * n2);
    forward_all<L, false, true>(x, t, tw, SmemLay<C>{sm + c});
#pragma unroll
    for (int e = 0; e < E; ++e)
        dst[col + eidx<L, LP>(t, e) * n2] = static_cast<uint64_t>(x[e]);
}

// Column pass, inverse, in place: inputs in [-e p, (1 + e)p], output in
// natural coefficient order, in [0, p).  L2 as in col_fwd_body.
template <int L, int C, int L2>
__device__ __forceinline__ void col_inv_body(uint64_t* d, size_t tile,
                                             const NttTw* __restrict__ twi, int64_t* sm) {
    constexpr int E = Geo<L>::E, LP = last_phase(L);
    const int t = threadIdx.x / C, c = threadIdx.x % C;
    constexpr size_t n2 = size_t{1} << L2;
    const size_t col = tile * C + c;
    int64_t x[E];
#pragma unroll
    for (int e = 0; e < E; ++e)
        x[e] = static_cast<int64_t>(d[col + eidx<L, LP>(t, e) * n2]);
    inverse_all<L, false, true>(x, t, twi, SmemLay<C>{sm + c});
#pragma unroll
    for (int e = 0; e < E; ++e) d[col + eidx<L, 0>(t, e) * n2] = canon(x[e]);
}

// Row pass, forward, of one row (thread t of its T): the four-step twiddle
// with the row transform's first root folded in (Wf, the row's first entry),
// then the row transform; outputs in the permuted order: in [0, p) (kRowCanon),
// within 1.6p (kRowLazy), or times img (kRowTimes: any residues within 1.7p, at
// the same positions), in [-0.17p, 1.17p].  src may equal dst (a row's threads load it
// before the first barrier or read and write the same positions).  DIRECT:
// the row is a whole polynomial of any 64-bit words (n1 = 1), untwisted.
enum RowOut { kRowLazy, kRowCanon, kRowTimes };
template <int L, bool DIRECT, RowOut OUT>
__device__ __forceinline__ void row_fwd_body(const uint64_t* src, const uint64_t* add,
                                             const uint64_t* __restrict__ img, uint64_t* dst,
                                             int t, bool valid,
                                             const NttTw* __restrict__ tw,
                                             const NttTw* __restrict__ Wf, int64_t* sm) {
    constexpr int E = Geo<L>::E, LP = last_phase(L);
    int64_t x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = eidx<L, 0>(t, e);
        if constexpr (DIRECT) x[e] = valid ? load_raw(src, add, i) : 0;
        else x[e] = mul_tw(static_cast<int64_t>(src[i]), ldtw(Wf + i));
    }
    forward_all<L, !DIRECT, true>(x, t, tw, SmemLay<1>{sm});
    if (!valid) return;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = perm_pos<L>(eidx<L, LP>(t, e));
        if constexpr (OUT == kRowCanon) dst[i] = canon(fold(x[e]));
        else if constexpr (OUT == kRowTimes)
            dst[i] = static_cast<uint64_t>(mul_var(x[e], static_cast<int64_t>(__ldg(img + i))));
        else dst[i] = static_cast<uint64_t>(x[e]);
    }
}

// Inverse row pass of one row, out row = Wi (.) INTT(y row), with
//   y = g (.) img         (SUM false: two transforms within 1.7p), or
//   y = sum_{q < Q} g_q   (SUM: g_q = g + q*N, products of kRowTimes),
// in the permuted evaluation order; Wif is the inverse twiddle with the
// inverse row transform's last root folded in.  Each thread loads the
// permuted positions of its last-phase registers, so the inverse starts where
// the forward ended.  out is in [-e p, (1 + e)p], or in [0, p) (CANON), and may
// alias g (a row's threads read all of it before the first store).
template <int L, bool SUM, bool CANON>
__device__ __forceinline__ void row_inv_body(const uint64_t* g, const uint64_t* img, int Q,
                                             size_t N, int t, bool valid,
                                             const NttTw* __restrict__ twi,
                                             const NttTw* __restrict__ Wif, uint64_t* out,
                                             int64_t* sm) {
    constexpr int E = Geo<L>::E, LP = last_phase(L);
    int64_t x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = perm_pos<L>(eidx<L, LP>(t, e));
        x[e] = valid ? static_cast<int64_t>(g[i]) : 0;
        if constexpr (!SUM)
            x[e] = mul_var(x[e], valid ? static_cast<int64_t>(img[i]) : 0);
    }
    if constexpr (SUM) {
        for (int q = 1; q < Q; ++q) {
            g += N;
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const int64_t y = valid ? static_cast<int64_t>(g[perm_pos<L>(eidx<L, LP>(t, e))]) : 0;
                x[e] = fold(add_shift(x[e], y));
            }
        }
    }
    inverse_all<L, true, true>(x, t, twi, SmemLay<1>{sm});
    if (!valid) return;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = eidx<L, 0>(t, e);
        const int64_t v = mul_tw(x[e], ldtw(Wif + i));
        out[i] = CANON ? canon(v) : static_cast<uint64_t>(v);
    }
}

// ---- per-length kernels: grid = (tiles, batch, transforms) ------------------------

// The column kernels fix the row length: l2 = L + DL (l2 - l1 is 0 or 1).
template <int L, int C, int DL>
__global__ void __launch_bounds__(col_threads<L, C>(), col_min_ctas<L, C>())
    col_fwd_kernel(const FwdIn in, const NttTw* __restrict__ tw) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const size_t off = static_cast<size_t>(blockIdx.y) << (2 * L + DL);
    const int z = blockIdx.z;
    const uint64_t* add = pick(in.add, z);
    col_fwd_body<L, C, L + DL>(pick(in.src, z) + off, add ? add + off : nullptr,
                               pick(in.dst, z) + off, blockIdx.x, tw, sm);
}

template <int L, int C, int DL>
__global__ void __launch_bounds__(col_threads<L, C>(), col_min_ctas<L, C>())
    col_inv_kernel(uint64_t* d, const NttTw* __restrict__ twi) {
    extern __shared__ int64_t sm[];
    chain_begin();
    col_inv_body<L, C, L + DL>(d + (static_cast<size_t>(blockIdx.y) << (2 * L + DL)), blockIdx.x,
                               twi, sm);
}

// The row of thread group v of this CTA.  DIRECT: rows are the batch's
// polynomials, V per CTA, the last CTA ragged.
struct RowAt {
    size_t inst, base;   // polynomial of the batch; offset of the row in it
    bool valid;
};
template <int L, bool DIRECT>
__device__ __forceinline__ RowAt row_at(int batch) {
    const int v = threadIdx.x / Geo<L>::T;
    const size_t r = static_cast<size_t>(blockIdx.x) * row_V<L>() + v;
    if constexpr (DIRECT) return RowAt{r, 0, r < static_cast<size_t>(batch)};
    else return RowAt{blockIdx.y, r << L, true};
}

// img (kRowTimes): instance b's image at img + b*N.
template <int L, bool DIRECT, RowOut OUT>
__global__ void __launch_bounds__(row_threads<L>(), row_min_ctas<L>()) row_fwd_kernel(
    const FwdIn in, const uint64_t* __restrict__ img, int batch, int l1,
    const NttTw* __restrict__ tw, const NttTw* __restrict__ Wf) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const int t = threadIdx.x % Geo<L>::T, v = threadIdx.x / Geo<L>::T, z = blockIdx.z;
    const RowAt r = row_at<L, DIRECT>(batch);
    const size_t off = (r.inst << (L + l1)) + r.base;
    const uint64_t* add = DIRECT ? pick(in.add, z) : nullptr;
    row_fwd_body<L, DIRECT, OUT>(pick(in.src, z) + off, add ? add + off : nullptr,
                                 OUT == kRowTimes ? img + off : nullptr, pick(in.dst, z) + off, t,
                                 r.valid, tw, Wf + r.base, sm + v * Geo<L>::PAD);
}

// Instance b reads g (and img) at b*Q*N and writes out at b*N; Q = 1 unless SUM.
template <int L, bool DIRECT, bool SUM>
__global__ void __launch_bounds__(row_threads<L>(), row_min_ctas<L>()) row_inv_kernel(
    const uint64_t* g, const uint64_t* img, int Q, int batch, int l1,
    const NttTw* __restrict__ twi, const NttTw* __restrict__ Wif, uint64_t* out) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const int t = threadIdx.x % Geo<L>::T, v = threadIdx.x / Geo<L>::T;
    const RowAt r = row_at<L, DIRECT>(batch);
    const size_t N = size_t{1} << (L + l1);
    const size_t gi = r.inst * Q * N + r.base;
    row_inv_body<L, SUM, DIRECT>(g + gi, SUM ? nullptr : img + gi, Q, N, t, r.valid, twi,
                                 Wif + r.base, out + r.inst * N + r.base, sm + v * Geo<L>::PAD);
}

// A whole product of one-row polynomials (n1 = 1) in one launch: both forward
// transforms, the pointwise product and the inverse in registers, V products
// per CTA.  At N = 2^12 it takes 18.5 us, where the passes took 39 (six
// launches on a handful of CTAs, 12 for a batch); it is bound by the
// multiplier pipe of one SM (73.7 K butterflies at about 37 cycles a warp).  A
// second half of the CTA for b's transform gained nothing (24.8 us).  c may
// alias a or b.
template <int L>
__global__ void __launch_bounds__(row_threads<L>()) row_product_kernel(
    uint64_t* c, const uint64_t* a, const uint64_t* b, int batch,
    const NttTw* __restrict__ tw, const NttTw* __restrict__ twi,
    const NttTw* __restrict__ Wif) {
    extern __shared__ int64_t sm[];
    constexpr int E = Geo<L>::E;
    const int t = threadIdx.x % Geo<L>::T, v = threadIdx.x / Geo<L>::T;
    const RowAt r = row_at<L, true>(batch);
    const size_t off = r.inst << L;
    const SmemLay<1> lay{sm + v * Geo<L>::PAD};
    int64_t x[E], y[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const size_t i = off + eidx<L, 0>(t, e);
        x[e] = r.valid ? fold_raw(a[i]) : 0;
        y[e] = r.valid ? fold_raw(b[i]) : 0;
    }
    forward_all<L, false, true>(x, t, tw, lay);
    forward_all<L, false, false>(y, t, tw, lay);
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = mul_var(x[e], y[e]);
    inverse_all<L, true, false>(x, t, twi, lay);
    if (!r.valid) return;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = eidx<L, 0>(t, e);
        c[off + i] = canon(mul_tw(x[e], ldtw(Wif + i)));
    }
}

// Row passes of the three transforms X0, X1, Z of an OLE relation, side by side
// in one CTA, then the number of slots with X0*X1 != Z added to *bad: the
// transformed rows are compared where they are made instead of being written,
// read back and compared by a launch of their own (an extraction and two checks
// at N = 2^19: 140.4 -> 134.6 us).  Bound by the same multiplies as the row pass.
template <int L, bool DIRECT>
__global__ void __launch_bounds__(3 * row_threads<L>()) row_check_kernel(
    const FwdIn in, int l1, const NttTw* __restrict__ tw, const NttTw* __restrict__ Wf,
    unsigned long long* bad) {
    constexpr int E = Geo<L>::E, T = Geo<L>::T, V = row_V<L>();
    extern __shared__ int64_t sm[];
    if (!DIRECT) chain_begin();
    const int t = threadIdx.x % T, v = threadIdx.x / T % V, z = threadIdx.x / (T * V);
    const size_t row = static_cast<size_t>(blockIdx.x) * V + v, off = row << L;
    const bool valid = !DIRECT || row == 0;
    const uint64_t* src = pick(in.src, z);
    const uint64_t* add = pick(in.add, z);
    int64_t* mine = sm + (z * V + v) * Geo<L>::PAD;
    int64_t x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int i = eidx<L, 0>(t, e);
        if constexpr (DIRECT) x[e] = valid ? load_raw(src, add, i) : 0;
        else x[e] = mul_tw(static_cast<int64_t>(ld_chained(src + off + i)), ldtw(Wf + off + i));
    }
    forward_all<L, !DIRECT, true>(x, t, tw, SmemLay<1>{mine});
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; ++e) mine[e * T + t] = x[e];
    __syncthreads();
    // Every thread compares its share of the CTA's slots (a direct plan has one row).
    constexpr int n = 1 << L, kThreads = 3 * T * V, kPad = Geo<L>::PAD;
    unsigned wrong = 0;
    for (int k = threadIdx.x; k < (DIRECT ? n : n * V); k += kThreads) {
        const int64_t* s = sm + (k >> L) * kPad + (k & (n - 1));
        wrong += canon(mul_var(s[0], s[V * kPad])) != canon(fold(s[2 * V * kPad]));
    }
    if (wrong) atomicAdd(bad, static_cast<unsigned long long>(wrong));
}

// ---- mixed-length kernels --------------------------------------------------------
// One launch per pass over a batch of products whose lengths range over
// 2^16 .. 2^20 (sub-lengths 2^8 .. 2^10 in both passes).  At these lengths
// every column CTA holds 512 threads x 16 elements (C = 32, 16, 8 columns)
// and every row CTA 64 threads (V = 4, 2, 1 rows), with the same shared
// memory, so one launch shape serves every length; each CTA reads its
// polynomial and tile from a job table and runs that length's body.

struct MixedPoly {
    const uint64_t* a;
    const uint64_t* b;
    uint64_t* c;
    uint64_t* A;                 // NTT(a), scratch
    const NttTw* tw1;
    const NttTw* tw1i;
    const NttTw* tw2;
    const NttTw* tw2i;
    const NttTw* Wf;
    const NttTw* Wif;
    int l1, l2;
};
struct MixedCta {
    uint32_t poly, tile;
};
constexpr int kMixedColThreads = 512, kMixedRowThreads = 64;
constexpr int kMixedLmin = 8, kMixedLmax = 10;
template <int L>
__host__ __device__ constexpr int mixed_C() { return kMixedColThreads / Geo<L>::T; }
template <int L>
__host__ __device__ constexpr int mixed_V() { return kMixedRowThreads / Geo<L>::T; }
constexpr size_t kMixedColSmem = sizeof(uint64_t) * Geo<10>::PAD * mixed_C<10>();
constexpr size_t kMixedRowSmem = sizeof(uint64_t) * Geo<10>::PAD * mixed_V<10>();
static_assert(sizeof(uint64_t) * Geo<8>::PAD * mixed_C<8>() == kMixedColSmem &&
              sizeof(uint64_t) * Geo<9>::PAD * mixed_C<9>() == kMixedColSmem, "col smem");

// Row `tile * V + thread group` of a row CTA of the mixed shapes.
template <int L>
struct MixedRow {
    int t = threadIdx.x % Geo<L>::T, v = threadIdx.x / Geo<L>::T;
    size_t base;
    __device__ __forceinline__ explicit MixedRow(uint32_t tile)
        : base((static_cast<size_t>(tile) * mixed_V<L>() + threadIdx.x / Geo<L>::T) << L) {}
    template <RowOut OUT>
    __device__ __forceinline__ void fwd(uint64_t* d, const uint64_t* img, const NttTw* tw,
                                        const NttTw* Wf, int64_t* sm) const {
        row_fwd_body<L, false, OUT>(d + base, nullptr, img + base, d + base, t, true, tw, Wf + base,
                                    sm + v * Geo<L>::PAD);
    }
    template <bool SUM>
    __device__ __forceinline__ void inv(const uint64_t* g, const uint64_t* img, int Q, size_t N,
                                        const NttTw* twi, const NttTw* Wif, uint64_t* out,
                                        int64_t* sm) const {
        row_inv_body<L, SUM, false>(g + base, SUM ? nullptr : img + base, Q, N, t, true, twi,
                                    Wif + base, out + base, sm + v * Geo<L>::PAD);
    }
};

#define PCGB_MIXED_SWITCH(LEN, CALL) \
    switch (LEN) {                    \
        case 8: CALL(8); break;       \
        case 9: CALL(9); break;       \
        case 10: CALL(10); break;     \
        default: break;               \
    }
// Column passes: (l1, l2) pairs, l2 = l1 or l1 + 1, both compile-time.
#define PCGB_MIXED_COL_SWITCH(P1, P2, CALL)           \
    switch (2 * (P1) + ((P2) - (P1))) {                \
        case 16: CALL(8, 8); break;                    \
        case 17: CALL(8, 9); break;                    \
        case 18: CALL(9, 9); break;                    \
        case 19: CALL(9, 10); break;                   \
        case 20: CALL(10, 10); break;                  \
        default: break;                                \
    }

// Column pass of a into A (which = 0) and of b into c (which = 1), which =
// first + blockIdx.y.
__global__ void __launch_bounds__(kMixedColThreads, 2) mixed_col_fwd_kernel(
    const MixedPoly* __restrict__ polys, const MixedCta* __restrict__ ctas, int first) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const MixedCta j = ctas[blockIdx.x];
    const MixedPoly& p = polys[j.poly];
    const bool which = first + blockIdx.y != 0;
    const uint64_t* src = which ? p.b : p.a;
    uint64_t* dst = which ? p.c : p.A;
#define PCGB_CALL(LL, L2) \
    col_fwd_body<LL, mixed_C<LL>(), L2>(src, nullptr, dst, j.tile, p.tw1, sm)
    PCGB_MIXED_COL_SWITCH(p.l1, p.l2, PCGB_CALL)
#undef PCGB_CALL
}

// Row pass of A (blockIdx.y = 0) and c (1).
__global__ void __launch_bounds__(kMixedRowThreads) mixed_row_fwd_kernel(
    const MixedPoly* __restrict__ polys, const MixedCta* __restrict__ ctas) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const MixedCta j = ctas[blockIdx.x];
    const MixedPoly& p = polys[j.poly];
    uint64_t* d = blockIdx.y ? p.c : p.A;
#define PCGB_CALL(LL) MixedRow<LL>(j.tile).template fwd<kRowLazy>(d, nullptr, p.tw2, p.Wf, sm)
    PCGB_MIXED_SWITCH(p.l2, PCGB_CALL)
#undef PCGB_CALL
}

// c = Wi (.) INTT( c (.) A ), in place on c.
__global__ void __launch_bounds__(kMixedRowThreads) mixed_row_mul_kernel(
    const MixedPoly* __restrict__ polys, const MixedCta* __restrict__ ctas) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const MixedCta j = ctas[blockIdx.x];
    const MixedPoly& p = polys[j.poly];
#define PCGB_CALL(LL) \
    MixedRow<LL>(j.tile).template inv<false>(p.c, p.A, 1, 0, p.tw2i, p.Wif, p.c, sm)
    PCGB_MIXED_SWITCH(p.l2, PCGB_CALL)
#undef PCGB_CALL
}

__global__ void __launch_bounds__(kMixedColThreads, 2) mixed_col_inv_kernel(
    const MixedPoly* __restrict__ polys, const MixedCta* __restrict__ ctas) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const MixedCta j = ctas[blockIdx.x];
    const MixedPoly& p = polys[j.poly];
#define PCGB_CALL(LL, L2) col_inv_body<LL, mixed_C<LL>(), L2>(p.c, j.tile, p.tw1i, sm)
    PCGB_MIXED_COL_SWITCH(p.l1, p.l2, PCGB_CALL)
#undef PCGB_CALL
}
#undef PCGB_MIXED_SWITCH
#undef PCGB_MIXED_COL_SWITCH

// ---- multi-request multiply-accumulate ------------------------------------
// The step-4 transforms of several expansions of different lengths
// 2^14 .. 2^20 (sub-lengths 2^7 .. 2^10) in four launches: the column pass and
// the row pass (times the image) of every request's Q g' buffers, the Q-way
// sum with the inverse row pass, and the inverse column pass into each
// request's z.  The CTA shapes are the mixed kernels' (512 column threads, 64 row
// threads, the same shared memory at every sub-length down to 2^7).
struct MacReq {
    uint64_t* g;                 // Q*N words, transformed in place
    const uint64_t* img;         // Q*N, evaluation images
    uint64_t* z;                 // N
    const NttTw* tw1;
    const NttTw* tw1i;
    const NttTw* tw2;
    const NttTw* tw2i;
    const NttTw* Wf;
    const NttTw* Wif;
    int Q, l1, l2;
};
struct MacCta {
    uint32_t req, q, tile;
};
constexpr int kMacLmin = 7;
static_assert(sizeof(uint64_t) * Geo<7>::PAD * mixed_C<7>() == kMixedColSmem &&
              sizeof(uint64_t) * Geo<7>::PAD * mixed_V<7>() == kMixedRowSmem,
              "sub-length 2^7 fits the mixed CTA shapes");

#define PCGB_MAC_SWITCH(LEN, CALL) \
    switch (LEN) {                  \
        case 7: CALL(7); break;     \
        case 8: CALL(8); break;     \
        case 9: CALL(9); break;     \
        case 10: CALL(10); break;   \
        default: break;             \
    }
#define PCGB_MAC_COL_SWITCH(P1, P2, CALL)             \
    switch (2 * (P1) + ((P2) - (P1))) {                \
        case 14: CALL(7, 7); break;                    \
        case 15: CALL(7, 8); break;                    \
        case 16: CALL(8, 8); break;                    \
        case 17: CALL(8, 9); break;                    \
        case 18: CALL(9, 9); break;                    \
        case 19: CALL(9, 10); break;                   \
        case 20: CALL(10, 10); break;                  \
        default: break;                                \
    }

__global__ void __launch_bounds__(kMixedColThreads, 2) mac_col_fwd_kernel(
    const MacReq* __restrict__ reqs, const MacCta* __restrict__ ctas) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const MacCta j = ctas[blockIdx.x];
    const MacReq& r = reqs[j.req];
    uint64_t* d = r.g + (static_cast<size_t>(j.q) << (r.l1 + r.l2));
#define PCGB_CALL(LL, L2) col_fwd_body<LL, mixed_C<LL>(), L2>(d, nullptr, d, j.tile, r.tw1, sm)
    PCGB_MAC_COL_SWITCH(r.l1, r.l2, PCGB_CALL)
#undef PCGB_CALL
}

__global__ void __launch_bounds__(kMixedRowThreads) mac_row_fwd_kernel(
    const MacReq* __restrict__ reqs, const MacCta* __restrict__ ctas) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const MacCta j = ctas[blockIdx.x];
    const MacReq& r = reqs[j.req];
    const size_t off = static_cast<size_t>(j.q) << (r.l1 + r.l2);
#define PCGB_CALL(LL) \
    MixedRow<LL>(j.tile).template fwd<kRowTimes>(r.g + off, r.img + off, r.tw2, r.Wf, sm)
    PCGB_MAC_SWITCH(r.l2, PCGB_CALL)
#undef PCGB_CALL
}

__global__ void __launch_bounds__(kMixedRowThreads) mac_row_inv_kernel(
    const MacReq* __restrict__ reqs, const MacCta* __restrict__ ctas) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const MacCta j = ctas[blockIdx.x];
    const MacReq& r = reqs[j.req];
    const size_t N = size_t{1} << (r.l1 + r.l2);
#define PCGB_CALL(LL) \
    MixedRow<LL>(j.tile).template inv<true>(r.g, nullptr, r.Q, N, r.tw2i, r.Wif, r.z, sm)
    PCGB_MAC_SWITCH(r.l2, PCGB_CALL)
#undef PCGB_CALL
}

__global__ void __launch_bounds__(kMixedColThreads, 2) mac_col_inv_kernel(
    const MacReq* __restrict__ reqs, const MacCta* __restrict__ ctas) {
    extern __shared__ int64_t sm[];
    chain_begin();
    const MacCta j = ctas[blockIdx.x];
    const MacReq& r = reqs[j.req];
#define PCGB_CALL(LL, L2) col_inv_body<LL, mixed_C<LL>(), L2>(r.z, j.tile, r.tw1i, sm)
    PCGB_MAC_COL_SWITCH(r.l1, r.l2, PCGB_CALL)
#undef PCGB_CALL
}
#undef PCGB_MAC_SWITCH
#undef PCGB_MAC_COL_SWITCH

// The table entry of v given in Montgomery form (v * 2^64); c32 = 2^32 mod p.
__device__ __forceinline__ NttTw tw_from_mont(uint64_t vR) {
    return ntt_tw(mont_mul(vR, 1), mont_mul(vR, uint64_t{1} << 32));
}

// Twiddle tables, element k*n2 + j2 with e = j2*(2*brev(k)+1-n1) mod 2N:
//   Wf  = psi^e,          times w0 = psi2^(n2/2) for j2 >= n2/2,
//   Wif = psi^-e * N^-1,  times w0i = psi2^-(n2/2) for j2 >= n2/2,
// w0 / w0i being the single root of the row transform's first forward /
// last inverse stage (that stage then only adds and subtracts).
// powR[b] = psi^(2^b) * R mod p; w0R, w0iR are w0, w0i times R.
__global__ void twiddle_kernel(NttTw* Wf, NttTw* Wif, int l1, int l2,
                               const uint64_t* __restrict__ powR, uint64_t oneR, uint64_t ninvR,
                               uint64_t w0R, uint64_t w0iR) {
    const size_t N = static_cast<size_t>(1) << (l1 + l2);
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= N) return;
    const int n1 = 1 << l1;
    const uint32_t k = static_cast<uint32_t>(idx >> l2);
    const uint32_t j2 = static_cast<uint32_t>(idx & ((1u << l2) - 1));
    const uint32_t i1 = l1 ? (__brev(k) >> (32 - l1)) : 0;
    const int64_t twoN = static_cast<int64_t>(2 * N);
    int64_t e = (static_cast<int64_t>(j2) * (2 * static_cast<int64_t>(i1) + 1 - n1)) % twoN;
    if (e < 0) e += twoN;
    const int64_t ei = (twoN - e) % twoN;
    uint64_t a = oneR, b = oneR;
    for (int bit = 0; bit <= l1 + l2; ++bit) {
        if ((e >> bit) & 1) a = mont_mul(a, powR[bit]);
        if ((ei >> bit) & 1) b = mont_mul(b, powR[bit]);
    }
    b = mont_mul(b, ninvR);        // psi^-e * N^-1 * R
    if (j2 >= (1u << (l2 - 1))) {
        a = mont_mul(a, w0R);
        b = mont_mul(b, w0iR);
    }
    Wf[idx] = tw_from_mont(a);
    Wif[idx] = tw_from_mont(b);
}

__global__ void reduce_kernel(uint64_t* d, const uint64_t* s, size_t n) {
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) d[i] = reduce_p(s[i]);
}

// ---- host side ---------------------------------------------------------------

uint32_t brev_host(uint32_t x, int bits) {
    uint32_t r = 0;
    for (int i = 0; i < bits; ++i) r |= ((x >> i) & 1u) << (bits - 1 - i);
    return r;
}

// Smallest primitive root of F_p, as the reference's NTT picks it
// (CPU_baseline/ntt.h:200-222): p - 1 = 2^25 * 47189 * 2912521, and g is
// primitive iff g^((p-1)/q) != 1 for each prime q | p - 1.  (It is 3.)  The
// slot values of a transform, which triples expose, depend on this choice.
uint64_t primitive_root_host() {
    constexpr uint64_t kQ[3] = {2, 47189, 2912521};
    static_assert((kPm - 1) == (uint64_t{1} << 25) * 47189ULL * 2912521ULL, "p - 1 factors");
    for (uint64_t g = 2;; ++g) {
        bool ok = true;
        for (uint64_t q : kQ) ok = ok && pow_p_host(g, (kPm - 1) / q) != 1;
        if (ok) return g;
    }
}

// Roots of a length-2^logn negacyclic transform with psi_n a primitive
// 2n-th root: stage s, group i uses psi_n^brev_logn(2^s + i) (Longa-Naehrig
// table), stored at the phase-permuted slot 2^s + (i % 2^q) * 2^s0 + i / 2^q.
NttTw* upload_root_table(uint64_t psi_n, int logn) {
    const int n = 1 << logn;
    std::vector<uint64_t> pw(n);
    uint64_t a = 1;
    for (int k = 0; k < n; ++k) { pw[k] = a; a = mul_p_host(a, psi_n); }
    std::vector<NttTw> tab(n > 1 ? n : 2, NttTw{0, 0, 0, 0});
    for (int s = 0; s < logn; ++s) {
        const int s0 = 4 * (s / 4), q = s - s0;
        for (int i = 0; i < (1 << s); ++i) {
            const uint64_t v = pw[brev_host(static_cast<uint32_t>((1 << s) + i), logn)];
            const int slot = (1 << s) + ((i & ((1 << q) - 1)) << s0) + (i >> q);
            tab[slot] = ntt_tw_host(v);
        }
    }
    NttTw* d = nullptr;
    PCGB_CK(cudaMalloc(&d, sizeof(NttTw) * tab.size()));
    upload_blocking(d, tab.data(), sizeof(NttTw) * tab.size());
    return d;
}

// Transforms up to 2^9 are one row (l1 = 0): a row CTA holds the whole
// polynomial, so there are no column passes.  Longer ones would keep a single
// SM busy where the four-step passes spread over several (2^12, three
// transforms: 18 us against 10).  A product is one launch instead of four
// passes, so it stays one row up to 2^12.  In us, one launch / four chained
// passes: 10.3 / 14.4 at 2^10; at 2^12 18.5 / 16.5 for one to three products,
// equal from four on, 18.6 / 28.3 for 74 and 121 / 138.7 for 1000; 55 / 24.7 at 2^13.
// The 2 us of one to three products at 2^12 would cost three more launches and a
// scratch allocation on the host, so there is no rule for them.
constexpr int kDirectLogN = 9, kOneRowLogN = 12;

NttPlan* build_plan(int logN) {
    auto* pl = new NttPlan();
    pl->logN = logN;
    pl->N = static_cast<size_t>(1) << logN;
    pl->l1 = logN <= kDirectLogN ? 0 : logN / 2;
    pl->l2 = logN - pl->l1;
    pl->n1 = 1 << pl->l1;
    pl->n2 = 1 << pl->l2;
    const uint64_t g = primitive_root_host();
    const uint64_t psi = pow_p_host(g, (kPm - 1) / (2 * pl->N));
    const uint64_t psi_inv = pow_p_host(psi, kPm - 2);
    if (!pl->direct()) {
        pl->tw1 = upload_root_table(pow_p_host(psi, pl->n2), pl->l1);
        pl->tw1i = upload_root_table(pow_p_host(psi_inv, pl->n2), pl->l1);
    }
    pl->tw2 = upload_root_table(pow_p_host(psi, pl->n1), pl->l2);
    pl->tw2i = upload_root_table(pow_p_host(psi_inv, pl->n1), pl->l2);
    PCGB_CK(cudaMalloc(&pl->Wf, sizeof(NttTw) * pl->N));
    PCGB_CK(cudaMalloc(&pl->Wif, sizeof(NttTw) * pl->N));
    const uint64_t R = r_mod_p();
    std::vector<uint64_t> powR(logN + 2);
    uint64_t pb = psi;
    for (int b = 0; b < logN + 2; ++b) { powR[b] = mul_p_host(pb, R); pb = mul_p_host(pb, pb); }
    uint64_t* d_pow = nullptr;
    PCGB_CK(cudaMalloc(&d_pow, sizeof(uint64_t) * powR.size()));
    upload_blocking(d_pow, powR.data(), sizeof(uint64_t) * powR.size());
    const uint64_t ninvR = mul_p_host(pow_p_host(pl->N % kPm, kPm - 2), R);
    // The row transform's stage-0 root: psi2^brev(1) = psi2^(n2/2) = psi^(N/2).
    const uint64_t w0R = mul_p_host(pow_p_host(psi, pl->N / 2), R);
    const uint64_t w0iR = mul_p_host(pow_p_host(psi_inv, pl->N / 2), R);
    twiddle_kernel<<<static_cast<unsigned>((pl->N + 255) / 256), 256>>>(
        pl->Wf, pl->Wif, pl->l1, pl->l2, d_pow, R, ninvR, w0R, w0iR);
    PCGB_POST_LAUNCH();
    if (pl->direct()) {
        pl->one_tw = pl->tw2;
        pl->one_twi = pl->tw2i;
        pl->one_Wi = pl->Wif;
    } else if (logN <= kOneRowLogN) {
        pl->one_tw = upload_root_table(psi, logN);
        pl->one_twi = upload_root_table(psi_inv, logN);
        // (a forward twiddle table comes with it: N entries of ones and w0)
        PCGB_CK(cudaMalloc(&pl->one_Wi, 2 * sizeof(NttTw) * pl->N));
        twiddle_kernel<<<static_cast<unsigned>((pl->N + 255) / 256), 256>>>(
            pl->one_Wi + pl->N, pl->one_Wi, 0, logN, d_pow, R, ninvR, w0R, w0iR);
        PCGB_POST_LAUNCH();
    }
    PCGB_CK(cudaDeviceSynchronize());
    cudaFree(d_pow);
    return pl;
}

template <int L, int C>
constexpr size_t col_smem() { return Geo<L>::NPH > 1 ? sizeof(uint64_t) * Geo<L>::PAD * C : 0; }
template <int L>
constexpr size_t row_smem() { return Geo<L>::NPH > 1 ? sizeof(uint64_t) * Geo<L>::PAD * row_V<L>() : 0; }

// Once per kernel and device: opt into dynamic shared memory above 48 KB and
// ask for the largest shared-memory carveout, so the CTAs that the register
// budget admits are not limited by a smaller L1/shared split.
struct OptinOnce {
    std::mutex mu;
    std::map<std::pair<const void*, int>, bool> done;
    template <class K>
    void operator()(K* kernel, size_t bytes) {
        if (bytes == 0) return;
        int dev = 0;
        PCGB_CK(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> lk(mu);
        auto key = std::make_pair(reinterpret_cast<const void*>(kernel), dev);
        if (done[key]) return;
        const void* f = reinterpret_cast<const void*>(kernel);
        if (bytes > 48 * 1024)
            PCGB_CK(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(bytes)));
        PCGB_CK(cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared));
        done[key] = true;
    }
};
OptinOnce g_optin;

// Column tile width for a launch over `work` = columns x batch: the widest one
// if that still gives every SM its 1024 threads, else 8 columns (64-byte row
// segments) if that gives ctas8 CTAs, else 4.  ctas8 is one per SM for the
// forward pass and three quarters of that for the inverse.  Products in us, with 4
// columns below the first line / with this: 64 x 2^13 37.5 / 29.6 (4 columns are
// half a warp there), 1 x 2^19 49.6 / 47.7, 2 x 2^19 63.4 / 60, 1 x 2^20 79.9 / 76,
// three transforms of 2^19 and the checks 122.7 / 119.5.  With 8 columns below
// that 1 x 2^14 goes from 18.5 to 20.5 and 1 x 2^18 (128 forward CTAs) from 32.8 to
// 34.3; with 4 in the inverse pass of 2^19 (128 CTAs) it stays at 50.5.
template <int L, int C = col_C(L), class F>
void col_width(size_t work, size_t ctas8, F&& f) {
    if constexpr (C > col_C_min(L)) {
        const size_t full = static_cast<size_t>(sm_count()) * (1024 / col_threads<L, C>());
        if (work / C < (C > 8 ? full : ctas8)) {
            col_width<L, C / 2>(work, ctas8, f);
            return;
        }
    }
    f(std::integral_constant<int, C>{});
}

template <int L>
void col_fwd_l(const NttPlan& pl, const FwdIn& in, int count, int batch, bool chained,
               cudaStream_t st) {
    col_width<L>(static_cast<size_t>(pl.n2) * batch * count, sm_count(), [&](auto CC) {
        constexpr int C = decltype(CC)::value;
        constexpr size_t sm = col_smem<L, C>();
        auto go = [&](auto kernel) {
            g_optin(kernel, sm);
            launch({dim3(pl.n2 / C, batch, count), col_threads<L, C>(), sm, chained}, st, kernel, in,
                   pl.tw1);
        };
        pl.l2 != L ? go(col_fwd_kernel<L, C, 1>) : go(col_fwd_kernel<L, C, 0>);
    });
}

template <int L>
void col_inv_l(const NttPlan& pl, uint64_t* d, int batch, cudaStream_t st) {
    col_width<L>(static_cast<size_t>(pl.n2) * batch, sm_count() * 3 / 4, [&](auto CC) {
        constexpr int C = decltype(CC)::value;
        constexpr size_t sm = col_smem<L, C>();
        auto go = [&](auto kernel) {
            g_optin(kernel, sm);
            launch({dim3(pl.n2 / C, batch), col_threads<L, C>(), sm, true}, st, kernel, d, pl.tw1i);
        };
        pl.l2 != L ? go(col_inv_kernel<L, C, 1>) : go(col_inv_kernel<L, C, 0>);
    });
}

// Grid of a row pass: V rows of one polynomial per CTA, or (direct plans) V
// polynomials of the batch.
template <int L>
dim3 row_grid(const NttPlan& pl, int batch, int count) {
    if (pl.direct()) return dim3((batch + row_V<L>() - 1) / row_V<L>(), 1, count);
    return dim3(pl.n1 / row_V<L>(), batch, count);
}

template <int L>
void row_fwd_l(const NttPlan& pl, const FwdIn& in, const uint64_t* img, int count, int batch,
               RowOut out, bool chained, cudaStream_t st) {
    constexpr size_t sm = row_smem<L>();
    auto go = [&](auto kernel) {
        g_optin(kernel, sm);
        launch({row_grid<L>(pl, batch, count), row_threads<L>(), sm, chained}, st, kernel, in, img,
               batch, pl.l1, pl.tw2, pl.Wf);
    };
    auto by_out = [&](auto D) {
        constexpr bool d = decltype(D)::value;
        if (out == kRowCanon) go(row_fwd_kernel<L, d, kRowCanon>);
        else if (out == kRowTimes) go(row_fwd_kernel<L, d, kRowTimes>);
        else if constexpr (!d) go(row_fwd_kernel<L, d, kRowLazy>);   // a product's operands
    };
    if constexpr (L <= kDirectLogN) {
        if (pl.direct()) by_out(std::true_type{});
    }
    if constexpr (L > kDirectLogN / 2) {
        if (!pl.direct()) by_out(std::false_type{});
    }
}

template <int L>
void row_inv_l(const NttPlan& pl, const uint64_t* g, const uint64_t* img, int Q, int batch,
               uint64_t* out, cudaStream_t st) {
    constexpr size_t sm = row_smem<L>();
    auto go = [&](auto kernel) {
        g_optin(kernel, sm);
        launch({row_grid<L>(pl, batch, 1), row_threads<L>(), sm, true}, st, kernel, g, img, Q, batch,
               pl.l1, pl.tw2i, pl.Wif, out);
    };
    if constexpr (L <= kDirectLogN) {
        if (pl.direct()) go(row_inv_kernel<L, true, true>);   // products run as one launch
    }
    if constexpr (L > kDirectLogN / 2) {
        if (!pl.direct()) img ? go(row_inv_kernel<L, false, false>) : go(row_inv_kernel<L, false, true>);
    }
}

template <int L>
void row_product_l(const NttPlan& pl, uint64_t* c, const uint64_t* a, const uint64_t* b, int batch,
                   cudaStream_t st) {
    constexpr size_t sm = row_smem<L>();
    g_optin(row_product_kernel<L>, sm);
    row_product_kernel<L><<<(batch + row_V<L>() - 1) / row_V<L>(), row_threads<L>(), sm, st>>>(
        c, a, b, batch, pl.one_tw, pl.one_twi, pl.one_Wi);
    PCGB_POST_LAUNCH();
}

// Runtime row length -> template instance (2^1 .. 2^12).
template <class F>
void by_len(int L, F&& f) {
    switch (L) {
        case 1: f(std::integral_constant<int, 1>{}); break;
        case 2: f(std::integral_constant<int, 2>{}); break;
        case 3: f(std::integral_constant<int, 3>{}); break;
        case 4: f(std::integral_constant<int, 4>{}); break;
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 6: f(std::integral_constant<int, 6>{}); break;
        case 7: f(std::integral_constant<int, 7>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 9: f(std::integral_constant<int, 9>{}); break;
        case 10: f(std::integral_constant<int, 10>{}); break;
        case 11: f(std::integral_constant<int, 11>{}); break;
        case 12: f(std::integral_constant<int, 12>{}); break;
        default: fail(PCGB_EINVAL, "NTT sub-length out of range");
    }
}
// Column sub-lengths: 2^5 .. 2^12 (logN 10 .. 24).
template <class F>
void by_col_len(int L, F&& f) {
    switch (L) {
        case 5: f(std::integral_constant<int, 5>{}); break;
        case 6: f(std::integral_constant<int, 6>{}); break;
        case 7: f(std::integral_constant<int, 7>{}); break;
        case 8: f(std::integral_constant<int, 8>{}); break;
        case 9: f(std::integral_constant<int, 9>{}); break;
        case 10: f(std::integral_constant<int, 10>{}); break;
        case 11: f(std::integral_constant<int, 11>{}); break;
        case 12: f(std::integral_constant<int, 12>{}); break;
        default: fail(PCGB_EINVAL, "NTT sub-length out of range");
    }
}

// chained: a kernel of the same call precedes this one on the stream
// (chain.cuh).  The inverse passes always have one.
void col_fwd(const NttPlan& pl, const FwdIn& in, int count, int batch, bool chained,
             cudaStream_t st) {
    by_col_len(pl.l1,
               [&](auto L) { col_fwd_l<decltype(L)::value>(pl, in, count, batch, chained, st); });
}
void col_inv(const NttPlan& pl, uint64_t* d, int batch, cudaStream_t st) {
    by_col_len(pl.l1, [&](auto L) { col_inv_l<decltype(L)::value>(pl, d, batch, st); });
}
void row_fwd(const NttPlan& pl, const FwdIn& in, const uint64_t* img, int count, int batch,
             RowOut out, bool chained, cudaStream_t st) {
    by_len(pl.l2, [&](auto L) {
        row_fwd_l<decltype(L)::value>(pl, in, img, count, batch, out, chained, st);
    });
}
template <int L>
void row_check_l(const NttPlan& pl, const FwdIn& in, unsigned long long* bad, cudaStream_t st) {
    constexpr size_t sm = sizeof(uint64_t) * Geo<L>::PAD * row_V<L>() * 3;
    auto go = [&](auto kernel, unsigned grid, bool chained) {
        g_optin(kernel, sm);
        launch({grid, 3 * row_threads<L>(), sm, chained}, st, kernel, in, pl.l1, pl.tw2, pl.Wf, bad);
    };
    if constexpr (L <= kDirectLogN) {
        if (pl.direct()) go(row_check_kernel<L, true>, 1, false);
    }
    if constexpr (L > kDirectLogN / 2) {
        if (!pl.direct())
            go(row_check_kernel<L, false>, static_cast<unsigned>(pl.n1 / row_V<L>()), true);
    }
}
// Sum of Q products (img null), or the product g (.) img.
void row_inv(const NttPlan& pl, const uint64_t* g, const uint64_t* img, int Q, int batch,
             uint64_t* out, cudaStream_t st) {
    by_len(pl.l2, [&](auto L) { row_inv_l<decltype(L)::value>(pl, g, img, Q, batch, out, st); });
}

// Forward transforms of `count` batches, any 64-bit inputs: the column pass
// from src (plus add) to dst and the row pass in place, or the single row
// pass of a direct plan.  out and img as for row_fwd_body.
void forward(const NttPlan& pl, const FwdIn& in, const uint64_t* img, int count, int batch,
             RowOut out, bool chained, cudaStream_t st) {
    if (pl.direct()) {
        row_fwd(pl, in, img, count, batch, out, chained, st);
        return;
    }
    col_fwd(pl, in, count, batch, chained, st);
    FwdIn rows;
    for (int z = 0; z < count; ++z) rows.src[z] = rows.dst[z] = in.dst[z];
    row_fwd(pl, rows, img, count, batch, out, true, st);
}

FwdIn fwd_one(const uint64_t* src, uint64_t* dst) {
    FwdIn in;
    in.src[0] = src;
    in.dst[0] = dst;
    return in;
}
FwdIn fwd_two(const uint64_t* s0, uint64_t* d0, const uint64_t* s1, uint64_t* d1) {
    FwdIn in;
    in.src[0] = s0; in.dst[0] = d0;
    in.src[1] = s1; in.dst[1] = d1;
    return in;
}

}  // namespace

const NttPlan& ntt_plan(int logN) {
    if (logN < 1 || logN > kMaxLogN) fail(PCGB_EINVAL, "NTT length must be 2^1 .. 2^24");
    static std::mutex mu;
    static std::map<std::pair<int, int>, std::unique_ptr<NttPlan>> cache;
    int dev = 0;
    PCGB_CK(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    auto& slot = cache[{dev, logN}];
    if (!slot) slot.reset(build_plan(logN));
    return *slot;
}

void ntt_forward3(const NttPlan& pl, const uint64_t* const (&src)[3],
                  const uint64_t* const (&add)[3], uint64_t* const (&dst)[3], cudaStream_t st) {
    FwdIn in;
    for (int z = 0; z < 3; ++z) {
        in.src[z] = src[z];
        in.add[z] = add[z];
        in.dst[z] = dst[z];
    }
    forward(pl, in, nullptr, 3, 1, kRowCanon, false, st);
}

bool ntt_check_needs_scratch(const NttPlan& pl) { return !pl.direct(); }

void ntt_check_ole(const NttPlan& pl, const uint64_t* x0, const uint64_t* x1, const uint64_t* z0,
                   const uint64_t* z1, uint64_t* scratch, unsigned long long* bad,
                   cudaStream_t st) {
    FwdIn in;
    in.src[0] = x0; in.src[1] = x1; in.src[2] = z0;
    in.add[2] = z1;
    if (!pl.direct()) {
        for (int z = 0; z < 3; ++z) in.dst[z] = scratch + z * pl.N;
        col_fwd(pl, in, 3, 1, false, st);
        in.add[2] = nullptr;
        for (int z = 0; z < 3; ++z) in.src[z] = in.dst[z];
    }
    by_len(pl.l2, [&](auto L) { row_check_l<decltype(L)::value>(pl, in, bad, st); });
}

void ntt_log_sizes(const NttPlan& pl, int* l1, int* l2) {
    *l1 = pl.l1;
    *l2 = pl.l2;
}

void ntt_forward(const NttPlan& pl, uint64_t* d, int batch, cudaStream_t st) {
    forward(pl, fwd_one(d, d), nullptr, 1, batch, kRowCanon, false, st);
}

// Per device: a second stream and two events for the two-half schedule of
// poly_mul_device; the mutex keeps one call's fork, launches and join
// together when several host threads multiply on the same device.
struct HalfFork {
    std::mutex mu;
    cudaStream_t side = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
};
HalfFork& half_fork() {
    static HalfFork f[64];
    int dev = 0;
    PCGB_CK(cudaGetDevice(&dev));
    return f[dev];
}

bool poly_mul_needs_scratch(const NttPlan& pl) { return pl.one_tw == nullptr; }

void poly_mul_device(const NttPlan& pl, uint64_t* c, const uint64_t* a, const uint64_t* b,
                     int batch, uint64_t* scratch, cudaStream_t st) {
    if (pl.one_tw) {
        by_len(pl.logN,
               [&](auto L) { row_product_l<decltype(L)::value>(pl, c, a, b, batch, st); });
        return;
    }
    // A = NTT(a) in scratch and c = NTT(b) as one launch per pass, then
    // c = INTT(c (.) A).  When c overlaps a, the column pass of a runs first.
    auto product = [&](size_t first, int count, cudaStream_t s) {
        uint64_t *A = scratch + first, *C = c + first;
        const uint64_t *x = a + first, *y = b + first;
        const size_t n = static_cast<size_t>(count) * pl.N * sizeof(uint64_t);
        if (overlap(range_of(C, n), range_of(x, n))) {
            col_fwd(pl, fwd_one(x, A), 1, count, false, s);
            col_fwd(pl, fwd_one(y, C), 1, count, true, s);
        } else {
            col_fwd(pl, fwd_two(x, A, y, C), 2, count, false, s);
        }
        row_fwd(pl, fwd_two(A, A, C, C), nullptr, 2, count, kRowLazy, true, s);
        row_inv(pl, C, A, 1, count, C, s);
        col_inv(pl, C, count, s);
    };
    // A batch of 2^18 words or more runs as two halves on two streams: each
    // pass alone leaves the multiplier pipe a third idle (barriers, loads,
    // its tail), and the other half's CTAs fill those slots (16 x 2^20: 829
    // -> 801 us, 2 x 2^18: 49.7 -> 42.9; at 4 x 2^16 no difference, below it
    // the fork costs 1 us).  Each half reads and writes only its own
    // products, so aliasing holds per half.
    if (batch < 2 || static_cast<size_t>(batch) * pl.N < (size_t{1} << 18)) {
        product(0, batch, st);
        return;
    }
    HalfFork& f = half_fork();
    std::lock_guard<std::mutex> lk(f.mu);
    if (!f.side) {
        PCGB_CK(cudaEventCreateWithFlags(&f.fork, cudaEventDisableTiming));
        PCGB_CK(cudaEventCreateWithFlags(&f.join, cudaEventDisableTiming));
        PCGB_CK(cudaStreamCreateWithFlags(&f.side, cudaStreamNonBlocking));
    }
    const int h0 = batch / 2;
    PCGB_CK(cudaEventRecord(f.fork, st));
    PCGB_CK(cudaStreamWaitEvent(f.side, f.fork, 0));
    product(static_cast<size_t>(h0) * pl.N, batch - h0, f.side);
    product(0, h0, st);
    PCGB_CK(cudaEventRecord(f.join, f.side));
    PCGB_CK(cudaStreamWaitEvent(st, f.join, 0));
}

bool poly_mul_mixed_ok(int logN) { return logN >= 2 * kMixedLmin && logN <= 2 * kMixedLmax; }

void poly_mul_device_mixed(int count, uint64_t* const* c, const uint64_t* const* a,
                           const uint64_t* const* b, const int* logN, cudaStream_t st) {
    if (count <= 0) return;
    std::vector<int> order(count);
    size_t scratch_words = 0;
    for (int i = 0; i < count; ++i) {
        if (!poly_mul_mixed_ok(logN[i])) fail(PCGB_EINVAL, "mixed poly-mul: N must be 2^16 .. 2^20");
        order[i] = i;
        scratch_words += size_t{1} << logN[i];
    }
    // Both operands' column passes share a launch unless some output
    // overlaps a first operand (which must then be read before).
    std::vector<Range> outs(count), firsts(count);
    for (int i = 0; i < count; ++i) {
        outs[i] = range_of(c[i], sizeof(uint64_t) << logN[i]);
        firsts[i] = range_of(a[i], sizeof(uint64_t) << logN[i]);
    }
    const bool alias = any_overlap(outs, firsts);
    // Longest products first, so the last CTAs of each pass are short ones.
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return logN[x] > logN[y]; });
    std::vector<MixedPoly> polys(count);
    std::vector<MixedCta> col, row;
    uint64_t* scratch = static_cast<uint64_t*>(pool_alloc(8 * scratch_words, st));
    size_t off = 0;
    for (int k = 0; k < count; ++k) {
        const int i = order[k];
        const NttPlan& pl = ntt_plan(logN[i]);
        MixedPoly& m = polys[k];
        m.a = a[i]; m.b = b[i]; m.c = c[i]; m.A = scratch + off;
        m.tw1 = pl.tw1; m.tw1i = pl.tw1i; m.tw2 = pl.tw2; m.tw2i = pl.tw2i;
        m.Wf = pl.Wf; m.Wif = pl.Wif;
        m.l1 = pl.l1; m.l2 = pl.l2;
        off += pl.N;
        int C = 0, V = 0;
        by_len(pl.l1, [&](auto L) {
            if constexpr (decltype(L)::value >= kMixedLmin && decltype(L)::value <= kMixedLmax)
                C = mixed_C<decltype(L)::value>();
        });
        by_len(pl.l2, [&](auto L) {
            if constexpr (decltype(L)::value >= kMixedLmin && decltype(L)::value <= kMixedLmax)
                V = mixed_V<decltype(L)::value>();
        });
        for (uint32_t tl = 0; tl < static_cast<uint32_t>(pl.n2 / C); ++tl) col.push_back({uint32_t(k), tl});
        for (uint32_t tl = 0; tl < static_cast<uint32_t>(pl.n1 / V); ++tl) row.push_back({uint32_t(k), tl});
    }
    const size_t b_polys = sizeof(MixedPoly) * polys.size();
    const size_t b_col = sizeof(MixedCta) * col.size(), b_row = sizeof(MixedCta) * row.size();
    const size_t o_col = (b_polys + 255) & ~size_t{255};
    const size_t o_row = (o_col + b_col + 255) & ~size_t{255};
    char* tab = static_cast<char*>(pool_alloc(o_row + b_row, st));
    upload_table(tab, polys.data(), b_polys, st);
    upload_table(tab + o_col, col.data(), b_col, st);
    upload_table(tab + o_row, row.data(), b_row, st);
    const MixedPoly* d_polys = reinterpret_cast<const MixedPoly*>(tab);
    const MixedCta* d_col = reinterpret_cast<const MixedCta*>(tab + o_col);
    const MixedCta* d_row = reinterpret_cast<const MixedCta*>(tab + o_row);
    const unsigned n_col = static_cast<unsigned>(col.size()), n_row = static_cast<unsigned>(row.size());
    g_optin(mixed_col_fwd_kernel, kMixedColSmem);
    g_optin(mixed_col_inv_kernel, kMixedColSmem);
    g_optin(mixed_row_fwd_kernel, kMixedRowSmem);
    g_optin(mixed_row_mul_kernel, kMixedRowSmem);
    for (int first = 0; first < (alias ? 2 : 1); ++first) {
        launch({dim3(n_col, alias ? 1 : 2), kMixedColThreads, kMixedColSmem, first > 0}, st,
               mixed_col_fwd_kernel, d_polys, d_col, first);
    }
    launch({dim3(n_row, 2), kMixedRowThreads, kMixedRowSmem, true}, st, mixed_row_fwd_kernel, d_polys,
           d_row);
    launch({n_row, kMixedRowThreads, kMixedRowSmem, true}, st, mixed_row_mul_kernel, d_polys, d_row);
    launch({n_col, kMixedColThreads, kMixedColSmem, true}, st, mixed_col_inv_kernel, d_polys, d_col);
    PCGB_CK(cudaFreeAsync(tab, st));
    PCGB_CK(cudaFreeAsync(scratch, st));
}

void ntt_mac_inverse(const NttPlan& pl, uint64_t* g, const uint64_t* img, int Q, uint64_t* acc,
                     cudaStream_t st) {
    forward(pl, fwd_one(g, g), img, 1, Q, kRowTimes, true, st);
    row_inv(pl, g, nullptr, Q, 1, acc, st);
    if (!pl.direct()) col_inv(pl, acc, 1, st);
}

bool ntt_mac_multi_ok(int logN) { return logN >= 2 * kMacLmin && logN <= 2 * kMixedLmax; }

void ntt_mac_inverse_multi(int count, uint64_t* const* g, const uint64_t* const* img, const int* Q,
                           uint64_t* const* z, const int* logN, cudaStream_t st) {
    if (count <= 0) return;
    std::vector<int> order(count);
    for (int i = 0; i < count; ++i) {
        if (!ntt_mac_multi_ok(logN[i])) fail(PCGB_EINVAL, "multi MAC: N must be 2^14 .. 2^20");
        if (Q[i] < 1 || !g[i] || !img[i] || !z[i]) fail(PCGB_EINVAL, "multi MAC: bad request");
        order[i] = i;
    }
    // Most work first, so the last CTAs of each pass are short ones.
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
        return (static_cast<uint64_t>(Q[x]) << logN[x]) > (static_cast<uint64_t>(Q[y]) << logN[y]);
    });
    std::vector<MacReq> reqs(count);
    std::vector<MacCta> colf, rowf, row, coli;
    for (int k = 0; k < count; ++k) {
        const int i = order[k];
        const NttPlan& pl = ntt_plan(logN[i]);
        MacReq& m = reqs[k];
        m.g = g[i]; m.img = img[i]; m.z = z[i];
        m.tw1 = pl.tw1; m.tw1i = pl.tw1i; m.tw2 = pl.tw2; m.tw2i = pl.tw2i;
        m.Wf = pl.Wf; m.Wif = pl.Wif;
        m.Q = Q[i]; m.l1 = pl.l1; m.l2 = pl.l2;
        int C = 0, V = 0;
        by_len(pl.l1, [&](auto L) {
            if constexpr (decltype(L)::value >= kMacLmin && decltype(L)::value <= kMixedLmax)
                C = mixed_C<decltype(L)::value>();
        });
        by_len(pl.l2, [&](auto L) {
            if constexpr (decltype(L)::value >= kMacLmin && decltype(L)::value <= kMixedLmax)
                V = mixed_V<decltype(L)::value>();
        });
        const uint32_t kk = static_cast<uint32_t>(k);
        const uint32_t nc = static_cast<uint32_t>(pl.n2 / C), nr = static_cast<uint32_t>(pl.n1 / V);
        for (uint32_t q = 0; q < static_cast<uint32_t>(m.Q); ++q) {
            for (uint32_t tl = 0; tl < nc; ++tl) colf.push_back({kk, q, tl});
            for (uint32_t tl = 0; tl < nr; ++tl) rowf.push_back({kk, q, tl});
        }
        for (uint32_t tl = 0; tl < nr; ++tl) row.push_back({kk, 0, tl});
        for (uint32_t tl = 0; tl < nc; ++tl) coli.push_back({kk, 0, tl});
    }
    // All tables in one copy: the requests, then the four CTA lists.
    const std::vector<MacCta>* lists[4] = {&colf, &rowf, &row, &coli};
    size_t o[4], total = sizeof(MacReq) * reqs.size();
    for (int i = 0; i < 4; ++i) {
        o[i] = (total + 255) & ~size_t{255};
        total = o[i] + sizeof(MacCta) * lists[i]->size();
    }
    std::vector<char> host(total);
    std::memcpy(host.data(), reqs.data(), sizeof(MacReq) * reqs.size());
    for (int i = 0; i < 4; ++i)
        std::memcpy(host.data() + o[i], lists[i]->data(), sizeof(MacCta) * lists[i]->size());
    char* tab = static_cast<char*>(pool_alloc(total, st));
    upload_table(tab, host.data(), total, st);
    const MacReq* d_req = reinterpret_cast<const MacReq*>(tab);
    auto ctas = [&](int i) { return reinterpret_cast<const MacCta*>(tab + o[i]); };
    auto grid = [&](int i) { return static_cast<unsigned>(lists[i]->size()); };
    g_optin(mac_col_fwd_kernel, kMixedColSmem);
    g_optin(mac_row_fwd_kernel, kMixedRowSmem);
    g_optin(mac_row_inv_kernel, kMixedRowSmem);
    g_optin(mac_col_inv_kernel, kMixedColSmem);
    launch({grid(0), kMixedColThreads, kMixedColSmem}, st, mac_col_fwd_kernel, d_req, ctas(0));
    launch({grid(1), kMixedRowThreads, kMixedRowSmem, true}, st, mac_row_fwd_kernel, d_req, ctas(1));
    launch({grid(2), kMixedRowThreads, kMixedRowSmem, true}, st, mac_row_inv_kernel, d_req, ctas(2));
    launch({grid(3), kMixedColThreads, kMixedColSmem, true}, st, mac_col_inv_kernel, d_req, ctas(3));
    PCGB_CK(cudaFreeAsync(tab, st));
}

void reduce_mod_p(uint64_t* d, const uint64_t* s, size_t count, cudaStream_t st) {
    reduce_kernel<<<static_cast<unsigned>((count + 255) / 256), 256, 0, st>>>(d, s, count);
    PCGB_POST_LAUNCH();
}

}  // namespace pcgb
