// Ragged (CSR) batches in one persistent, length-bucketed launch.
//
// Array a occupies elements [off[a], off[a+1]) of the flat buffer.  The
// launch sequence of a plan is
//   1. reset the control block (counters, queue head),
//   2. k_bin_count   - histogram of arrays per working-length bucket,
//   3. k_bin_scatter - array ids grouped by bucket, largest bucket first
//                      (up to kBinSmall arrays: 1-3 in one launch, k_bin_small),
//   4. k_sort_ragged - persistent CTAs pull tasks from a device queue (one
//                      atomicAdd per task; no waiting on other CTAs).  A task
//                      is one CTA's worth of arrays of one bucket: the CTA
//                      splits into teams of TPA threads, one array per team,
//                      each team running the network of its bucket's tile
//                      (multi-warp teams synchronise on a named barrier).
// Tasks are ordered largest working length first, so the longest tasks start
// early and the short ones fill the tail.  The bitonic network's cost depends
// only on the working length, so all teams of a task finish together.
//
// The reference's only ragged one-launch precedent is
// SortPartitionsAdaptive_outofplace (cusort.hpp:2309-2352), a grid-stride loop
// over CSR partitions with one block shape and shared memory sized for the
// largest partition; here every bucket has its own tile shape.
#pragma once
#include <cuda_runtime.h>

#include "cta_xpose.cuh"

namespace b200s {

constexpr int kMaxBuckets = 16;
constexpr int kMaxOverflow = 4;
constexpr int kRaggedLmin = 3;  // smallest bucket: W = 8
constexpr int kBinSmall = 4096; // arrays of the largest batch that one CTA bins

struct RaggedCtl {
    int count[kMaxBuckets];    // arrays per bucket
    int cursor[kMaxBuckets];   // scatter cursors
    int base[kMaxBuckets];     // first position of each bucket's ids in the id list
    int dhead[kMaxBuckets];    // work queue heads of the dedicated bucket launches
    int head;                  // task queue head
    int too_long;              // arrays longer than every kernel (not sorted)
    int ocount[kMaxOverflow];  // arrays per cluster bucket
    int reserved[2];
};

// Binning parameters: nb buckets for the persistent kernel (W = 8 .. 8 <<
// (nb-1)); arrays with log2 W in [over_lo, over_lo + n_over) go to the
// cluster bucket log2 W - over_lo (ids at oids[bucket * stride]).
struct BinSpec {
    int nb;
    int over_lo;
    int n_over;
    int stride;
};

__device__ __forceinline__ int ceil_log2_dev(int n) { return n <= 1 ? 0 : 32 - __clz(n - 1); }

// Bucket of an array of length n >= 1: log2 of its working length, minus lmin.
__device__ __forceinline__ int bucket_of(int n, int lmin) {
    const int l = ceil_log2_dev(n);
    return (l > lmin ? l : lmin) - lmin;
}

// The binning kernels are defined in exactly one translation unit (plan.cu).
#ifdef B200S_DEFINE_BIN_KERNELS
__global__ void k_bin_count(const int* __restrict__ off, int arrays, RaggedCtl* ctl, BinSpec spec) {
    __shared__ int h[kMaxBuckets];
    __shared__ int over;
    if (threadIdx.x < kMaxBuckets) h[threadIdx.x] = 0;
    if (threadIdx.x == 0) over = 0;
    __syncthreads();
    for (int a = blockIdx.x * blockDim.x + threadIdx.x; a < arrays; a += gridDim.x * blockDim.x) {
        const int n = off[a + 1] - off[a];
        if (n <= 0) continue;
        const int b = bucket_of(n, kRaggedLmin);
        if (b < spec.nb) atomicAdd(&h[b], 1);
        else if (ceil_log2_dev(n) - spec.over_lo >= spec.n_over) atomicAdd(&over, 1);
    }
    __syncthreads();
    if (threadIdx.x < spec.nb && h[threadIdx.x]) atomicAdd(&ctl->count[threadIdx.x], h[threadIdx.x]);
    if (threadIdx.x == 0 && over) atomicAdd(&ctl->too_long, over);
}

// The whole binning of a batch of at most kBinSmall arrays in one CTA: reset,
// histogram, positions and lists, with the arrays' buckets kept in registers
// between the two halves.  One launch of about 3 us where the reset and the
// two kernels below take three launches in a row; from several thousand
// arrays on one CTA's loads and list stores take longer than that.
// (Offsets and lists of a kernel launched with programmatic stream
// serialization are not __restrict__: that would promise that they are constant
// from the kernel's start, before griddepcontrol.wait, and allow loads above it.)
__global__ void __launch_bounds__(1024) k_bin_small(const int* off, int arrays, RaggedCtl* ctl, int* ids, int* oids,
                                                    BinSpec spec) {
    constexpr int kPer = kBinSmall / 1024, kClasses = kMaxBuckets + kMaxOverflow;
    __shared__ int h[kClasses + 1], base[kMaxBuckets];  // h[kClasses]: too long for every kernel
    const int t = int(threadIdx.x), lane = t & 31;
    if (t <= kClasses) h[t] = 0;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    __syncthreads();
    int cls[kPer], pos[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int a = i * 1024 + t;
        const int n = a < arrays ? off[a + 1] - off[a] : 0;
        int c = -1;
        if (n > 0) {
            const int b = bucket_of(n, kRaggedLmin), o = ceil_log2_dev(n) - spec.over_lo;
            c = b < spec.nb ? b : o < spec.n_over ? kMaxBuckets + o : kClasses;
        }
        // one shared atomic per class and warp
        const unsigned same = __match_any_sync(0xffffffffu, c);
        int first = 0;
        if (c >= 0 && lane == __ffs(int(same)) - 1) first = atomicAdd(&h[c], __popc(same));
        first = __shfl_sync(0xffffffffu, first, __ffs(int(same)) - 1);
        cls[i] = c;
        pos[i] = first + __popc(same & ((1u << lane) - 1u));
    }
    __syncthreads();
    if (t < kMaxBuckets) {
        int s = 0;  // larger buckets come first
        for (int b = t + 1; b < spec.nb; ++b) s += h[b];
        base[t] = s;
        ctl->count[t] = h[t];
        ctl->cursor[t] = 0;
        ctl->base[t] = s;
        ctl->dhead[t] = 0;
    } else if (t < kClasses) {
        ctl->ocount[t - kMaxBuckets] = h[t];
    } else if (t == kClasses) {
        ctl->head = 0;
        ctl->too_long = h[kClasses];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int c = cls[i], a = i * 1024 + t;
        if (c >= 0 && c < kMaxBuckets) ids[base[c] + pos[i]] = a;
        else if (c >= kMaxBuckets && c < kClasses) oids[size_t(c - kMaxBuckets) * spec.stride + pos[i]] = a;
    }
}

// ids[] receives array ids grouped by bucket, largest working length first;
// arrays for the cluster kernels go to their own lists.
__global__ void k_bin_scatter(const int* __restrict__ off, int arrays, RaggedCtl* ctl, int* ids, int* oids,
                              BinSpec spec) {
    const int nb = spec.nb;
    __shared__ int base[kMaxBuckets], h[kMaxBuckets], grab[kMaxBuckets];
    if (threadIdx.x == 0) {
        int s = 0;
        for (int b = nb - 1; b >= 0; --b) {
            base[b] = s;
            if (blockIdx.x == 0) ctl->base[b] = s;  // for the launches of dedicated buckets
            s += ctl->count[b];
        }
    }
    for (int a0 = blockIdx.x * blockDim.x; a0 < arrays; a0 += gridDim.x * blockDim.x) {
        if (threadIdx.x < kMaxBuckets) h[threadIdx.x] = 0;
        __syncthreads();
        const int a = a0 + int(threadIdx.x);
        int b = -1, local = 0;
        if (a < arrays) {
            const int n = off[a + 1] - off[a];
            if (n > 0) {
                b = bucket_of(n, kRaggedLmin);
                if (b < nb) {
                    local = atomicAdd(&h[b], 1);
                } else {
                    const int ob = ceil_log2_dev(n) - spec.over_lo;
                    if (ob < spec.n_over) {
                        const int pos = atomicAdd(&ctl->ocount[ob], 1);
                        oids[size_t(ob) * spec.stride + pos] = a;
                    }
                    b = -1;
                }
            }
        }
        __syncthreads();
        if (threadIdx.x < nb && h[threadIdx.x]) grab[threadIdx.x] = atomicAdd(&ctl->cursor[threadIdx.x], h[threadIdx.x]);
        __syncthreads();
        if (b >= 0) ids[base[b] + grab[b] + local] = a;
        __syncthreads();
    }
}
#else
__global__ void k_bin_small(const int* off, int arrays, RaggedCtl* ctl, int* ids, int* oids, BinSpec spec);
__global__ void k_bin_count(const int* __restrict__ off, int arrays, RaggedCtl* ctl, BinSpec spec);
__global__ void k_bin_scatter(const int* __restrict__ off, int arrays, RaggedCtl* ctl, int* ids, int* oids,
                              BinSpec spec);
#endif  // B200S_DEFINE_BIN_KERNELS

// log2 elements per thread of bucket L (= log2 W) in a shape family with
// K = 2^LKF: K elements per thread when a whole team fits the CTA, more when
// it would not (the team never exceeds the CTA).
constexpr int family_lk(int L, int LKF, int LOGCTA) {
    const int lk = L < LKF ? L : LKF;
    return L - lk > LOGCTA ? L - LOGCTA : lk;
}

// Tile of bucket L in a shape family: one lane for W <= K, then more lanes,
// then more warps.
template <int LKF, int L, int CTA>
struct FamilyShape {
    static constexpr int LK = family_lk(L, LKF, log2_const(CTA));
    static constexpr int REST = L - LK;
    static constexpr int LG = REST < 5 ? REST : 5;
    static constexpr int LW = REST - LG;
    using type = Shape<LK, LG, LW>;
};

// Shared-memory bytes of one team of windowed bucket L, a multiple of 16.
template <class EW, int LK, int L>
constexpr size_t team_bytes() {
    return (xc_smem_bytes<EW, LK, L>() + 15) / 16 * 16;
}

// How the persistent kernel sorts bucket L of element type E (EW: the type
// its windowed and transposed networks run on, ElemRecI32G for stable records):
//   kWindows   teams of whole warps, the windowed network of win.cuh,
//   kXpose     several arrays per warp, the one-warp transposed network,
//   kBlocked   shuffles and registers (network.cuh), one of two families.
// The first two are the tiles the same lengths take in a packed batch; 16-byte
// records have no one-warp transposed tile, and int32 arrays below 256 and
// others below 64 are faster in the blocked form.
enum RaggedKind { kBlocked, kXpose, kWindows };
template <class EW>
constexpr int ragged_lk() {
    return sizeof(typename EW::Reg) == 4 ? 5 : 4;
}
template <class E, class EW>
constexpr RaggedKind ragged_kind(int L) {
    if (L >= ragged_lk<EW>() + 5) return kWindows;
    if (sizeof(typename E::Reg) != 16 && L >= (sizeof(typename E::Reg) == 4 ? 8 : 6)) return kXpose;
    return kBlocked;
}
// log2 threads per array of bucket L.
template <class E, class EW>
constexpr int ragged_log_tpa(int L, int family_k, int log_cta) {
    return L - (ragged_kind<E, EW>(L) == kBlocked ? family_lk(L, family_k, log_cta) : ragged_lk<EW>());
}

template <class E, class EW, int L, int LKF, int CTA>
__device__ __forceinline__ void ragged_task(const typename E::Mem* in, typename E::Mem* out,
                                            const int* off, const int* ids, const int count,
                                            const int local_task, unsigned char* smem_raw) {
    constexpr int LOGTPA = ragged_log_tpa<E, EW>(L, LKF, log2_const(CTA)), TPA = 1 << LOGTPA;
    static_assert(TPA <= CTA, "a team fits the CTA");
    constexpr int APT = CTA / TPA;
    const int tid = thread_index();
    const int team = tid >> LOGTPA, t = tid & (TPA - 1);
    const int idx = local_task * APT + team;
    int na = 0;
    long long start = 0;
    if (idx < count) {
        const int a = ids[idx];
        start = off[a];
        na = off[a + 1] - off[a];
    }
    if constexpr (ragged_kind<E, EW>(L) == kWindows) {
        static_assert(TPA == 32 || APT <= 15, "named barrier ids");
        using S = Shape<ragged_lk<EW>(), 5, LOGTPA - 5>;
        auto* sm = reinterpret_cast<typename EW::Reg*>(smem_raw + size_t(team) * team_bytes<EW, S::LK, L>());
        xc_sort_array<EW, S, false>(in + start, out + start, na, t, sm, TeamBarrier{1 + team, TPA});
    } else if constexpr (ragged_kind<E, EW>(L) == kXpose) {
        constexpr int LK = ragged_lk<EW>(), LG = L - LK;
        auto* sm = reinterpret_cast<typename EW::Reg*>(smem_raw) + team * xp_region<LK, LG>();
        xp_sort_array<EW, LK, LG, keys_only<EW>::value ? kXpIoStriped : kXpIoStaged>(
            in + start, out + start, na, t, sm, xp_pay<EW, LK, LG>(smem_raw, APT, team));
    } else {
        using R = typename E::Reg;
        using S = typename FamilyShape<LKF, L, CTA>::type;
        static_assert(S::LW == 0, "blocked buckets are below a warp");
        R* cur = reinterpret_cast<R*>(smem_raw);
        R* nxt = cur;
        R v[S::K];
        load_tile<E, S::K>(v, in + start, t * S::K, na);
        network<E, S>(v, t, cur, nxt, CtaBarrier{}, na);
        store_tile<E, S::K>(v, out + start, t * S::K, na);
    }
}

// NB buckets (W = 8 .. 8 << (NB-1)); a blocked bucket b uses family B (K =
// 2^LKB) when bit b of family_mask is set, else family A (K = 2^LKA); buckets
// whose bit is set in dedicated_mask are left to their own launches (their ids
// stay in the list at ctl->base[b]).  MINB: CTAs per SM the register budget is
// sized for.  A CTA's first task is its own number; the further ones come
// from the queue, each drawn while the previous task is sorted.
template <class E, class EW, int CTA, int NB, int LKA, int LKB, int MINB>
__global__ void __launch_bounds__(CTA, MINB) k_sort_ragged(const typename E::Mem* in, typename E::Mem* out,
                                                        const int* off, const int* ids, RaggedCtl* ctl,
                                                        unsigned family_mask, unsigned dedicated_mask) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_first[NB], s_tasks[NB], s_base[NB], s_count[NB];
    __shared__ int s_total, s_next[2];
    // launched with programmatic stream serialization behind the binning kernel
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (threadIdx.x < NB) {
        const int b = int(threadIdx.x), L = b + kRaggedLmin;
        const int c = ctl->count[b];
        const int log_apt = log2_const(CTA) -
                            ragged_log_tpa<E, EW>(L, ((family_mask >> b) & 1u) ? LKB : LKA, log2_const(CTA));
        s_tasks[b] = ((dedicated_mask >> b) & 1u) ? 0 : (c + (1 << log_apt) - 1) >> log_apt;
        s_count[b] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int task = 0, base = 0;
        for (int b = NB - 1; b >= 0; --b) {
            // dedicated buckets get no tasks here, but their ids still occupy
            // the list, so the bases count them
            s_first[b] = task;
            s_base[b] = base;
            task += s_tasks[b];
            base += s_count[b];
        }
        s_total = task;
    }
    __syncthreads();
    const int total = s_total;
    int task = int(blockIdx.x);
    for (int turn = 0; task < total; turn ^= 1) {
        if (threadIdx.x == 0) s_next[turn] = int(gridDim.x) + atomicAdd(&ctl->head, 1);
        int b = NB - 1;
        while (b > 0 && task >= s_first[b] + s_tasks[b]) --b;
        const int local = task - s_first[b];
        const bool fam_b = (family_mask >> b) & 1u;
        sfor<0, NB>([&](auto bc) {
            constexpr int B = decltype(bc)::value;
            constexpr int L = B + kRaggedLmin;
            if (b == B) {
                const int* list = ids + s_base[B];
                if (ragged_kind<E, EW>(L) == kBlocked && fam_b)
                    ragged_task<E, EW, L, LKB, CTA>(in, out, off, list, s_count[B], local, smem_raw);
                else
                    ragged_task<E, EW, L, LKA, CTA>(in, out, off, list, s_count[B], local, smem_raw);
            }
        });
        __syncthreads();
        task = s_next[turn];
    }
}

// Shared memory of k_sort_ragged: the largest CTA's worth of a bucket's teams.
template <class E, class EW, int CTA, int NB, int L = kRaggedLmin>
constexpr size_t ragged_smem() {
    size_t bytes = 0;
    if constexpr (ragged_kind<E, EW>(L) == kWindows)
        bytes = size_t(CTA >> (L - ragged_lk<EW>())) * team_bytes<EW, ragged_lk<EW>(), L>();
    else if constexpr (ragged_kind<E, EW>(L) == kXpose)
        bytes = xp_smem<EW, ragged_lk<EW>(), L - ragged_lk<EW>()>(CTA >> (L - ragged_lk<EW>()));
    if constexpr (L < kRaggedLmin + NB - 1) {
        const size_t rest = ragged_smem<E, EW, CTA, NB, L + 1>();
        return rest > bytes ? rest : bytes;
    } else {
        return bytes;
    }
}

// Launches over an id list: every array of the list fits the tile; one group
// per array.  With d_count null the grid strides over `count` arrays.
// Otherwise (a dedicated bucket of a ragged plan) the count and the list's
// first position are read on the device, so that a captured launch sorts
// whatever the binning put into its bucket, and the resident CTAs pull groups
// of arrays from the queue at d_head (one atomicAdd per group), which keeps
// them busy when the arrays' lengths, and so their costs, differ.
template <class E, class S, int CTA, bool SB = false>
__global__ void __launch_bounds__(CTA) k_sort_idlist(const typename E::Mem* in, typename E::Mem* out,
                                                     const int* __restrict__ off, const int* __restrict__ ids,
                                                     int count, const int* d_count, const int* d_base,
                                                     int* d_head) {
    using R = typename E::Reg;
    __shared__ int s_next;
    if (d_count) {
        count = *d_count;
        ids += *d_base;
    }
    constexpr int APC = CTA / S::TPA;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* cur = reinterpret_cast<R*>(smem_raw);
    R* nxt = SB ? cur : cur + S::W;  // the launch passes 1 or 2 buffers of W elements
    const int slot = int(threadIdx.x) / S::TPA;
    const int t = int(threadIdx.x) % S::TPA;
    long long first = (long long)blockIdx.x * APC;
    for (;;) {
        if (d_head) {
            if (threadIdx.x == 0) s_next = atomicAdd(d_head, APC);
            __syncthreads();
            first = s_next;
            __syncthreads();
        }
        if (first >= count) break;  // uniform across the CTA
        const long long g = first + slot;
        int na = 0;
        long long start = 0;
        if (g < count) {
            const int a = ids[g];
            start = off[a];
            na = off[a + 1] - off[a];
        }
        R v[S::K];
        load_tile<E, S::K>(v, in + start, t * S::K, na);
        if constexpr (SB) network<E, S>(v, t, cur, nxt, CtaBarrierSingle{}, na);
        else network<E, S>(v, t, cur, nxt, CtaBarrier{}, na);
        store_tile<E, S::K>(v, out + start, t * S::K, na);
        if (!d_head) first += (long long)gridDim.x * APC;
    }
}

}  // namespace b200s
