// Arrays beyond one CTA, many at a time: the reflection network in passes over
// global memory instead of a cluster's distributed shared memory.
//
// One CTA sorts each slice of 2^LOCAL elements (stages below LOCAL, as a
// single-CTA tile).  Each later stage ST is two passes over the batch, in
// place in the output:
//   far   layers ST .. ST-LK+1: a thread holds the 2^LK elements whose index
//         differs in just those bits, so every layer is in its registers and
//         no shared memory is used.  The elements with bit ST set are taken
//         at the mirrored position (all lower thread bits complemented), which
//         makes the reflection the register pair q, q ^ (2^LK - 1), as in the
//         windows of win_layout.h; both directions read whole cache lines.
//   near  layers ST-LK .. 0: tiles of 2^(ST-LK+1) consecutive elements, loaded
//         straight into the first merge window (coalesced: its registers are
//         the tile's top bits) and stored coalesced.
// A thread of the far pass and a CTA of the near pass write only what they
// read, so the passes run in place; the comparators, their order and the
// keep-own rule are the reference network's, and elements at or beyond n are
// padding that never moves and is never written.
//
// Why: a cross-CTA layer of a cluster reads a whole slice at 2.5 TB/s over all
// SMs with one CTA per SM and nothing to overlap it, about 15 us per 4 M
// records and layer, and 4-CTA clusters leave 16 of 148 SMs idle; a pass moves
// its 8 bytes in and out at HBM rate, about 10 us per 4 M records.  With few
// arrays the passes win too: slices of 4096 spread one array over many SMs
// (one array of 30000 records: 8 slices and 6 short passes take 28 us where
// a cluster of four CTAs takes 43).  Measured against the clusters (us): 256
// arrays of 65536 records 688 -> 502, 128 of 65536 uint64-key records
// 1064 -> 585, 128 of 131072 int32 keys 486 -> 256.  The clusters stay for
// ragged lists, whose counts only the device knows, and for stable records:
// their words need room between passes that a call in place does not have (out
// of place a (key, position) word would fit the record's slot in the output).
//
// Programmatic dependent launch: each kernel waits for the one before it.  It
// lets the next be scheduled at its start (`early`) when no grid can crowd
// another out, i.e. with few CTAs or with a full wave of them; between those,
// CTAs that arrive early pile up on the SMs that the running grid leaves free
// (128 slices of 4096: 50 us instead of 43), and it lets go before its stores.
#pragma once
#include "cta_xpose.cuh"

namespace b200s {

__device__ __forceinline__ void launch_dependents(const bool now) {
    if (now) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Stages 0 .. S::LOGW-1: slice j of array a, a = blockIdx.x >> log_slices.
template <class E, class S, int MINB>
__global__ void __launch_bounds__(S::TPA, MINB)
    k_sort_slices(const typename E::Mem* in, typename E::Mem* out, int n, int log_slices, int early) {
    using R = typename E::Reg;
    using W = Win<E, S::LK, S::LOGW>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* sm = reinterpret_cast<R*>(smem_raw);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    launch_dependents(early);
    const long long a = (long long)blockIdx.x >> log_slices;
    const int first = int(blockIdx.x & ((1u << log_slices) - 1u)) << S::LOGW;
    if (first >= n) return;
    const long long off = a * n + first;
    const int rest = n - first < S::W ? n - first : S::W, t = int(threadIdx.x);
    R v[S::K];
    W::load(v, in + off, t, 0, rest, sm);
    W::network(v, t, rest, sm, CtaBarrier{});
    launch_dependents(!early);
    W::template store<true>(v, out + off, t, 0, rest, sm);
}

constexpr int kFarThreads = 256;

// Layers st .. st-LK+1 of stage st over arrays of 2^logw slots.
template <class E, int LK>
__global__ void __launch_bounds__(kFarThreads, 2) k_merge_far(typename E::Mem* data, int n, int logw, int st,
                                                              int early) {
    using R = typename E::Reg;
    constexpr int K = 1 << LK, H = K >> 1;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    launch_dependents(early);
    const int log_blocks = logw - LK - log2_const(kFarThreads);  // CTAs per array
    const long long a = (long long)blockIdx.x >> log_blocks;
    const int g = int(blockIdx.x & ((1u << log_blocks) - 1u)) * kFarThreads + int(threadIdx.x);
    const int step = st + 1 - LK;  // the registers' lowest index bit
    const int low = g & ((1 << step) - 1), base = (g >> step) << (st + 1);
    if (base + (1 << st) >= n) return;  // nothing above the middle: the stage moves nothing
    typename E::Mem* src = data + a * n;
    const int mirrored = base | ((1 << step) - 1 - low), plain = base | low;
    R v[K];
    sfor<0, K>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        const int i = ((q & H) ? mirrored : plain) + (q << step);
        v[q] = E::pad();
        if (i < n) v[q] = E::from_mem(xp_ld(src + i), i);
    });
    sfor<0, LK>([&](auto rc) {
        constexpr int r = LK - 1 - decltype(rc)::value;
        sfor<0, K>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr int p = r == LK - 1 ? (q ^ (K - 1)) : (q | (1 << r));
            if constexpr (!(q & (1 << r))) xcex<E, q>(v[q], v[p]);
        });
    });
    launch_dependents(!early);
    sfor<0, K>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        const int i = ((q & H) ? mirrored : plain) + (q << step);
        if (i < n) xp_st(src + i, E::to_mem(v[q]));
    });
}

// Layers LOGT-1 .. 0 of stage st = LOGT + LK - 1, one tile of 2^LOGT
// consecutive elements per CTA.
template <class E, int LK, int LOGT, int MINB>
__global__ void __launch_bounds__(1 << (LOGT - LK), MINB)
    k_merge_near(typename E::Mem* data, int n, int logw, int early) {
    using R = typename E::Reg;
    using W = Win<E, LK, LOGT>;
    constexpr int K = 1 << LK, ST = LOGT + LK - 1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* sm = reinterpret_cast<R*>(smem_raw);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    launch_dependents(early);
    const long long a = (long long)blockIdx.x >> (logw - LOGT);
    const int first = int(blockIdx.x & ((1u << (logw - LOGT)) - 1u)) << LOGT;
    if (first >= n || ((first >> (ST + 1)) << (ST + 1)) + (1 << ST) >= n) return;  // padding, or an untouched block
    typename E::Mem* src = data + a * n + first;
    const int rest = n - first, t = int(threadIdx.x);
    R v[K];
    const int i0 = W::merge_index(t);
    sfor<0, K>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        const int i = i0 + (q << W::LT);
        v[q] = E::pad();
        if (i < rest) v[q] = E::from_mem(xp_ld(src + i), i);
    });
    W::merge(v, t, rest, sm, CtaBarrier{});
    launch_dependents(!early);
    W::template store<true>(v, src, t, 0, rest, sm);
}

}  // namespace b200s
