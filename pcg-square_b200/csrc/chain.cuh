// Dependent launches without the gap between them.
//
// The kernels of one call run one after another on a stream, and between two
// of them the chip idles for the launch and for the next grid's start: 2 to 3 us
// where a pass itself takes 4 to 8.  A kernel launched with chained = true may
// start while its predecessor's last CTAs still run (programmatic dependent
// launch); it calls chain_begin() before it touches anything the predecessor
// reads or writes.  Measured: expansion of 2^12 launched directly 52 -> 43 us,
// triples and two checks at 2^19 136 -> 131, nine mixed products 232 -> 222,
// nothing at 16 x 2^20.  In a graph the plain edges are as fast or faster (2^18:
// 554 against 566 us), so a captured launch keeps them; so do the persistent
// AES walks, whose one CTA per SM must not wait for room (373 against 402 us).
// Rules:
//   * the first kernel of a call is launched normally, so everything queued
//     before the call (the caller's own kernels, copies) is complete;
//   * every thread of a chained kernel reaches chain_wait(), so a grid is
//     complete only after all before it;
//   * buffers written earlier in the same call are read with ordinary or
//     L2 loads (ld_chained), never through the read-only path: their writer may
//     still run when this kernel starts.  Inputs of the call and resident tables
//     may use __ldg.
#ifndef PCGB_CHAIN_CUH_
#define PCGB_CHAIN_CUH_

#include <cuda_runtime.h>

#include "pcgb_internal.h"

namespace pcgb {

// Lets the next chained kernel start placing its CTAs.
__device__ __forceinline__ void chain_release() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// Waits until the grids before this one are complete and their writes visible.
__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void chain_begin() {
    chain_release();
    chain_wait();
}

__device__ __forceinline__ Blk ld_chained(const Blk* p) {
    const ulonglong2 v = __ldcg(reinterpret_cast<const ulonglong2*>(p));
    return Blk{v.x, v.y};
}
__device__ __forceinline__ uint64_t ld_chained(const uint64_t* p) {
    return __ldcg(reinterpret_cast<const unsigned long long*>(p));
}
__device__ __forceinline__ ulonglong2 ld_chained(const ulonglong2* p) { return __ldcg(p); }

inline bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
    PCGB_CK(cudaStreamIsCapturing(st, &c));
    return c != cudaStreamCaptureStatusNone;
}

// Two adjacent nodes (p even) with one 32-byte store where their array is
// 32-byte aligned: a lane's own subtree is a line of its own, so a warp's 16-byte
// stores cost a line lookup per lane each, in the same pipe as the AES table
// loads (AES, 777 keys x 2^14: 372 -> 353 us; the ChaCha8 walks, bound by the
// integer ALU, are 0.2 % slower with it and keep the plain stores).
__device__ __forceinline__ bool pair_aligned(const Blk* base) {
    return (reinterpret_cast<uintptr_t>(base) & 31) == 0;
}
__device__ __forceinline__ void st_pair(Blk* p, const Blk& a, const Blk& b, bool aligned) {
    if (aligned) {
        asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(a.lo), "l"(a.hi),
                     "l"(b.lo), "l"(b.hi)
                     : "memory");
    } else {
        *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(a.lo, a.hi);
        *reinterpret_cast<ulonglong2*>(p + 1) = make_ulonglong2(b.lo, b.hi);
    }
}

struct LaunchShape {
    dim3 grid, block;
    size_t smem = 0;
    bool chained = false;
    unsigned cluster = 1;   // CTAs along x
};

template <class... P, class... A>
void launch(const LaunchShape& s, cudaStream_t st, void (*kern)(P...), const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = s.grid;
    cfg.blockDim = s.block;
    cfg.dynamicSmemBytes = s.smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    unsigned n = 0;
    if (s.chained && !capturing(st)) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (s.cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = s.cluster;
        at[n].val.clusterDim.y = 1;
        at[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    PCGB_CK(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...));
    PCGB_POST_LAUNCH();
}

}  // namespace pcgb

#endif
