// The reflection network of one tile with every layer in registers: the layers
// are cut into windows across stage boundaries (win_layout.h), one trip through
// shared memory each.  Used by the kernels of cta_xpose.cuh.
//
// The comparators are those of cusort_v6.hpp:90-142 in the same order, with
// the keep-own rule of cusort.hpp:460-472, so the output, tie order of records
// included, is the reference's.  Keys alone (kKeysOnly) sort each thread's
// registers with Batcher's odd-even merge sort instead of stages 0 .. LK-1.
//
// What bounds it: at 16 elements per thread the shared-memory pipe (80 % of its
// wavefronts at W = 4096 records) with the issue slots close behind (72 %);
// the ALU and FMA pipes share the compare-exchanges (ALU 61 %, and 61 % of the
// half of the FMA pipe that multiplies integers, elem.cuh).
// 32 records per thread take a quarter fewer trips but their unrolled code
// (100 KB and more) overflows the instruction cache: W = 2048 / 4096 / 8192 in
// 53.6 / 65.7 / 77.5 us per 4 M records against 47.6 / 53.9 / 66.9 with 16.
#pragma once
#include "win_layout.h"
#include "xpose.cuh"

namespace b200s {

// Lanes of one bank sweep: 2^m elements of this register type fill the banks.
template <class R>
constexpr int win_m() {
    return sizeof(R) == 16 ? 3 : sizeof(R) == 8 ? 4 : 5;
}

template <class E, int LK, int LOGW>
struct Win {
    using R = typename E::Reg;
    using P = WinPlan<LK, LOGW, win_m<R>()>;
    static constexpr int K = 1 << LK, LT = P::LT, LW = P::LW;
    static constexpr int kElems = P::kT.elems;  // shared-memory elements of the tile
    static constexpr int kWindows = P::kT.windows, kMerges = P::kT.merges;

    // Layouts by number: 0 .. kWindows the windows (0 natural), kIo the
    // coalesced global one, kMerge + i the windows of a whole-tile merge.
    static constexpr int kIo = -1, kMerge = 100;
    static constexpr WinLayout layout(int l) {
        return l == kIo ? P::kT.io : l >= kMerge ? P::kT.merge[l - kMerge] : P::kT.win[l];
    }

    // Address part of thread t in a layout (MIR: the thread bits below the
    // reflection's stage complemented).
    template <int L, bool MIR>
    static __device__ __forceinline__ int base(const int t) {
        constexpr WinLayout w = layout(L);
        int a = 0;
        sfor<0, LT>([&](auto jc) {
            constexpr int j = decltype(jc)::value;
            constexpr int wt = P::kT.weight[w.thr[j]];
            constexpr bool flip = MIR && w.thr[j] < w.st;
            const int bit = (t >> j) & 1;
            a += (flip ? 1 - bit : bit) * wt;
        });
        return a;
    }
    // Natural layout: thread t holds elements [rank(t) * K, rank(t) * K + K)
    // (its bits are in the order of the bank classes), and the inverse.
    static __device__ __forceinline__ int rank(const int t) {
        int r = 0;
        sfor<0, LT>([&](auto jc) {
            constexpr int j = decltype(jc)::value;
            constexpr int at = P::kT.win[0].thr[j] - LK;
            r |= ((t >> j) & 1) << at;
        });
        return r;
    }
    static __device__ __forceinline__ int thread_of(const int r) {
        int t = 0;
        sfor<0, LT>([&](auto jc) {
            constexpr int j = decltype(jc)::value;
            constexpr int at = P::kT.win[0].thr[j] - LK;
            t |= ((r >> at) & 1) << j;
        });
        return t;
    }

    // First element of thread t in layout kMerge (register q: q << LT further).
    static __device__ __forceinline__ int merge_index(const int t) {
        constexpr WinLayout w = layout(kMerge);
        int i = 0;
        sfor<0, LT>([&](auto jc) {
            constexpr int j = decltype(jc)::value;
            constexpr int at = w.thr[j];
            i |= ((t >> j) & 1) << at;
        });
        return i;
    }

    template <int L>
    static __device__ __forceinline__ void put(const R (&v)[K], const int t, R* sm) {
        constexpr WinLayout w = layout(L);
        const int bp = base<L, false>(t);
        int bm = bp;
        if constexpr (w.refl >= 0) bm = base<L, true>(t);
        sfor<0, K>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr int off = P::reg_off(w, q);
            sh_st(&sm[(P::mirrored(w, q) ? bm : bp) + off], v[q]);
        });
    }
    template <int L>
    static __device__ __forceinline__ void get(R (&v)[K], const int t, const R* sm) {
        constexpr WinLayout w = layout(L);
        const int bp = base<L, false>(t);
        int bm = bp;
        if constexpr (w.refl >= 0) bm = base<L, true>(t);
        sfor<0, K>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr int off = P::reg_off(w, q);
            v[q] = sh_ld(&sm[(P::mirrored(w, q) ? bm : bp) + off]);
        });
    }
    // Warps of padding.  In a layout where every warp holds its natural part
    // of the tile (32 * K consecutive elements), a warp whose part starts at or
    // beyond n holds only padding, which never moves (keep-own rule): it skips
    // the layout's layers, and its trips, since the places at and beyond n hold
    // padding from the load on.  `dead` is uniform over the warp.
    static constexpr bool own_part(int l) { return LW > 0 && P::same_warps(layout(l), layout(0)); }
    static __device__ __forceinline__ bool dead(const int t, const int n) {
        return LW > 0 && ((t >> 5) << (LK + 5)) >= n;
    }

    // One trip.  A thread puts its elements exactly where it got them, so no
    // thread's put can touch a place that another has still to read, and one
    // barrier between the puts and the next gets is enough: a warp's while
    // every warp keeps its part of the tile, else the team's.
    template <int A, int B, class Bar>
    static __device__ __forceinline__ void move(R (&v)[K], const int t, R* sm, const bool skip, const Bar& bar) {
        constexpr bool local = P::same_warps(layout(A), layout(B));
        if (!own_part(A) || !skip) put<A>(v, t, sm);
        if constexpr (local) __syncwarp();
        else bar();
        if (!own_part(B) || !skip) get<B>(v, t, sm);
    }
    template <int L>
    static __device__ __forceinline__ void layers(R (&v)[K]) {
        constexpr WinLayout w = layout(L);
        sfor<0, w.layers>([&](auto ic) {
            constexpr int r = w.layers - 1 - decltype(ic)::value;
            sfor<0, K>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                constexpr int p = r == w.refl ? (q ^ (K - 1)) : (q | (1 << r));
                if constexpr (!(q & (1 << r))) xcex<E, q>(v[q], v[p]);
            });
        });
    }
    // One window: the trip from layout A and layout B's layers.
    template <int A, int B, class Bar>
    static __device__ __forceinline__ void window(R (&v)[K], const int t, R* sm, const bool skip, const Bar& bar) {
        if constexpr (own_part(A) && own_part(B)) {
            if (!skip) {
                put<A>(v, t, sm);
                __syncwarp();
                get<B>(v, t, sm);
                layers<B>(v);
            }
        } else {
            move<A, B>(v, t, sm, skip, bar);
            if (!own_part(B) || !skip) layers<B>(v);
        }
    }
    // The network, from and to the natural layout; n: elements that are not
    // padding.
    template <class Bar>
    static __device__ __forceinline__ void network(R (&v)[K], const int t, const int n, R* sm, const Bar& bar) {
        const bool skip = dead(t, n);
        if (!skip) {
            if constexpr (keys_only<E>::value) xp_reg_sort_oem<E, LK>(v);
            else sfor<0, LK>([&](auto sc) { xp_reg_stage<E, LK, decltype(sc)::value>(v); });
        }
        sfor<1, kWindows + 1>([&](auto wc) {
            constexpr int L = decltype(wc)::value;
            window<L - 1, L>(v, t, sm, skip, bar);
        });
    }
    // The merges on bits LOGW-1 .. 0, from layout kMerge to the natural one.
    template <class Bar>
    static __device__ __forceinline__ void merge(R (&v)[K], const int t, const int n, R* sm, const Bar& bar) {
        const bool skip = dead(t, n);
        layers<kMerge>(v);
        sfor<1, kMerges>([&](auto mc) {
            constexpr int L = kMerge + decltype(mc)::value;
            window<L - 1, L>(v, t, sm, skip, bar);
        });
        if constexpr (P::kT.merge[kMerges - 1].reg[0] != 0) move<kMerge + kMerges - 1, 0>(v, t, sm, skip, bar);
    }

    // ---- global memory ------------------------------------------------------
    // Each warp moves its natural part of the tile (32 * K consecutive
    // elements) with coalesced accesses through the region, in the layout kIo,
    // so that only the warp has to synchronise.  `first`: index of the tile's
    // element 0 in the array of n; elements at or beyond n are padding.
    // A record buffer that is not aligned to the record moves element by
    // element, 16-byte records word by word in a loop, which keeps that path's
    // code short.
    static __device__ __forceinline__ int io_index(const int t) { return (t & 31) | ((t >> 5) << (LK + 5)); }
    static constexpr bool kWords = sizeof(typename E::Mem) == 16;
    static __device__ __forceinline__ int io_offset(const int q) {
        int a = 0;
        sfor<0, LK>([&](auto rc) {
            constexpr int r = decltype(rc)::value;
            constexpr int wt = P::kT.weight[P::kT.io.reg[r]];
            a += ((q >> r) & 1) * wt;
        });
        return a;
    }

    // Load into the natural layout.  pay: the payloads by position (gathered types).
    static __device__ __forceinline__ void load(R (&v)[K], const typename E::Mem* src, const int t, const int first,
                                                const int n, R* sm, int32_t* pay = nullptr) {
        if (!kWords && !xp_wide(src)) {  // uniform: natural loads, and the region's padding
            const int i0 = rank(t) * K;
            load_tile<E, K>(v, src, first + i0, n);
            if constexpr (gathers<E>::value)
                if (pay)
                    for (int i = i0; i < i0 + K && first + i < n; ++i) pay[i] = src[first + i].data;
            put<0>(v, t, sm);
            return;
        }
        const int i0 = io_index(t), b = base<kIo, false>(t);
        // The loads first, as they come from memory, and the payloads stored
        // without a branch: a store inside the bounds test kept the loads of
        // gathered types apart (4 M stable records, W = 1024 / 2048 / 4096:
        // 68.6 / 76.7 / 83.3 -> 57.6 / 67.0 / 76.7 us).
        if (kWords && !xp_wide(src)) {
            if constexpr (kWords) {
#pragma unroll 1
                for (int q = 0; q < K; ++q) {
                    const int idx = first + i0 + 32 * q;
                    sh_st(&sm[b + io_offset(q)], idx < n ? E::from_mem(xp_ld_words(src + idx), idx) : E::pad());
                }
            }
        } else {
            typename E::Mem m[K];
            sfor<0, K>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                const int idx = first + i0 + 32 * q;
                if (idx < n) m[q] = xp_ldcs(src + idx);
            });
            sfor<0, K>([&](auto qc) {
                constexpr int q = decltype(qc)::value;
                constexpr int off = P::reg_off(P::kT.io, q);
                const int i = i0 + 32 * q, idx = first + i;
                if constexpr (gathers<E>::value)
                    if (pay) pay[i] = m[q].data;
                sh_st(&sm[b + off], idx < n ? E::from_mem(m[q], idx) : E::pad());
            });
        }
        __syncwarp();
        get<0>(v, t, sm);
    }
    // Whether the tile of a whole CTA, just loaded, is in order (uniform over
    // the CTA): each thread its elements and the first one of the next rank.
    static __device__ __forceinline__ bool in_order(const R (&v)[K], const int t, const R* sm) {
        __syncthreads();  // every part of the region is loaded
        const int r = rank(t);
        bool ok = thread_in_order<E, K>(v);
        if (r + 1 < (1 << LT)) ok &= !E::after(v[K - 1], sh_ld(&sm[base<0, false>(thread_of(r + 1))]));
        return __syncthreads_and(ok) != 0;
    }
    // Store from the natural layout.  KEEP: a later pass reads it again.
    template <bool KEEP = false>
    static __device__ __forceinline__ void store(const R (&v)[K], typename E::Mem* dst, const int t, const int first,
                                                 const int n, R* sm) {
        if (dead(t, n - first)) return;
        if (!kWords && !xp_wide(dst)) {
            store_tile<E, K>(v, dst, first + rank(t) * K, n);
            return;
        }
        put<0>(v, t, sm);
        __syncwarp();
        const int i0 = io_index(t), b = base<kIo, false>(t);
        if (kWords && !xp_wide(dst)) {
            if constexpr (kWords) {
#pragma unroll 1
                for (int q = 0; q < K; ++q) {
                    const int idx = first + i0 + 32 * q;
                    if (idx < n) xp_st_words(dst + idx, E::to_mem(sh_ld(&sm[b + io_offset(q)])));
                }
            }
            return;
        }
        sfor<0, K>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr int off = P::reg_off(P::kT.io, q);
            const int idx = first + i0 + 32 * q;
            const R x = sh_ld(&sm[b + off]);
            if (idx < n) {
                if constexpr (KEEP) xp_st(dst + idx, E::to_mem(x));
                else xp_stcs(dst + idx, E::to_mem(x));
            }
        });
    }
    // The same for gathered types: every payload is fetched (from pay when
    // set, else from src, the unsorted array) before `ready` lets any thread
    // store, because src may be dst.
    template <class Ready>
    static __device__ __forceinline__ void store_gather(const R (&v)[K], const typename E::Mem* src,
                                                        typename E::Mem* dst, const int t, const int first,
                                                        const int n, R* sm, const int32_t* pay, const Ready& ready) {
        put<0>(v, t, sm);
        __syncwarp();
        const int i0 = io_index(t), b = base<kIo, false>(t);
        typename E::Mem m[K];
        sfor<0, K>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            constexpr int off = P::reg_off(P::kT.io, q);
            const R x = sh_ld(&sm[b + off]);
            int32_t d = 0;
            if (first + i0 + 32 * q < n) d = pay ? pay[E::position(x)] : src[E::position(x)].data;
            m[q] = E::to_mem(x, d);
        });
        ready();
        const bool w = xp_wide(dst);
        sfor<0, K>([&](auto qc) {
            constexpr int q = decltype(qc)::value;
            const int idx = first + i0 + 32 * q;
            if (idx < n) {
                if (w) xp_stcs(dst + idx, m[q]);
                else dst[idx] = m[q];
            }
        });
    }
};

}  // namespace b200s
