// Launch form 3 of the tiles of a warp and more: every comparator layer of an
// array held by a whole CTA (or one CTA's slice of a cluster's array) runs as a
// compare-exchange between two registers of one thread (win.cuh), the tile
// going through one shared region between windows.
//
// Global memory: every warp moves its own 32 * K consecutive elements with
// coalesced accesses through the region.  (One thread's K consecutive elements
// with 128-bit accesses touch 32 cache lines per instruction: at W = 4096
// records that was 22 % of the shared-memory pipe's time, and is 8 % this way.)
//
// Cluster stages (index bits above one CTA's slice) run in the slice's first
// merge window: there a warp's lanes read 32 neighbouring elements of the
// partner CTA's slice (distributed shared memory; in the natural layout they
// would be 2^LK elements apart, each read pulling a whole sector), and the
// registers hold the slice's top LK bits, so the first LK local merges follow
// without a trip.
#pragma once
#include <cooperative_groups.h>

#include "win.cuh"

namespace b200s {

// Shared-memory elements of a slice, and bytes with the payloads of gathered
// types (one CTA per array; clusters fetch payloads from global memory).
template <class E, int LK, int LOGW>
constexpr int xc_smem_elems() {
    return Win<E, LK, LOGW>::kElems;
}
template <class E, int LK, int LOGW>
constexpr size_t xc_smem_bytes() {
    return size_t(Win<E, LK, LOGW>::kElems) * sizeof(typename E::Reg) + (gathers<E>::value ? size_t(4) << LOGW : 0);
}

// Cross-CTA layer of a cluster stage, in the slice's first merge window: the
// partner of (rank, local index i) is (rank ^ cm, reflect ? i ^ (W - 1) : i).
// The slice is published at its own addresses, then read back from the
// partner CTA.
template <class E, int LK, int LT, bool REFLECT>
__device__ __forceinline__ void xc_cluster_layer(typename E::Reg (&v)[1 << LK], const int t, const int rank,
                                                 const int cm, const bool upper, typename E::Reg* sm) {
    using R = typename E::Reg;
    using W = Win<E, LK, LK + LT>;
    constexpr int K = 1 << LK, T = 1 << LT;
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    W::template put<W::kMerge>(v, t, sm);
    cluster.sync();
    const R* remote = cluster.map_shared_rank(sm, rank ^ cm);
    const int pb = W::template base<W::kMerge, false>(REFLECT ? T - 1 - t : t);
    sfor<0, K>([&](auto qc) {
        constexpr int q = decltype(qc)::value;
        constexpr int off = W::P::reg_off(W::layout(W::kMerge), REFLECT ? K - 1 - q : q);
        const R b = dsm_ld(&remote[pb + off]);
        v[q] = E::pick(v[q], b, upper);
    });
    cluster.sync();
}

// threadIdx.x, read anew at each call: a loop over arrays that uses it does
// not keep the windows' addresses in registers from one array to the next.
__device__ __forceinline__ int thread_index() {
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}

// The network of an array held by a cluster of 2^LC CTAs of 2^LT threads
// (slice of 2^(LK+LT) elements per CTA, n of them not padding): the local stages, then per cluster
// stage its cross-CTA layers and the merges of the slice.
template <class E, int LK, int LT, int LC>
__device__ __forceinline__ void xc_cluster_network(typename E::Reg (&v)[1 << LK], const int t, const int rank,
                                                   const int n, typename E::Reg* sm) {
    constexpr int LOCAL = LK + LT;
    using W = Win<E, LK, LOCAL>;
    const CtaBarrier bar{};
    W::network(v, t, n, sm, bar);
#pragma unroll 1
    for (int st = LOCAL; st < LOCAL + LC; ++st) {
        W::template move<0, W::kMerge>(v, t, sm, W::dead(t, n), bar);
        xc_cluster_layer<E, LK, LT, true>(v, t, rank, (2 << (st - LOCAL)) - 1, (rank >> (st - LOCAL)) & 1, sm);
#pragma unroll 1
        for (int j = st - 1; j >= LOCAL; --j)
            xc_cluster_layer<E, LK, LT, false>(v, t, rank, 1 << (j - LOCAL), (rank >> (j - LOCAL)) & 1, sm);
        W::merge(v, t, n, sm, bar);
    }
}

// One array by a team of S::TPA threads (bar: its barrier): load, network,
// store.  CHECK: with the sortedness test (the team is the CTA).
template <class E, class S, bool CHECK, class Bar = CtaBarrier>
__device__ __forceinline__ void xc_sort_array(const typename E::Mem* src, typename E::Mem* dst, const int n,
                                              const int t, typename E::Reg* sm, const Bar& bar = Bar()) {
    using R = typename E::Reg;
    using W = Win<E, S::LK, S::LOGW>;
    R v[S::K];
    int32_t* pay = gathers<E>::value ? reinterpret_cast<int32_t*>(sm + W::kElems) : nullptr;
    W::load(v, src, t, 0, n, sm, pay);
    bool skip = false;
    if constexpr (CHECK) skip = W::in_order(v, t, sm);
    if (!skip) W::network(v, t, n, sm, bar);
    if (skip && src == dst) return;
    if constexpr (gathers<E>::value) W::store_gather(v, src, dst, t, 0, n, sm, pay, [] {});
    else W::store(v, dst, t, 0, n, sm);
}

// One array per CTA of S::TPA threads (a batch of more arrays than a grid's
// CTAs takes several launches: a loop here would keep the windows' addresses
// in registers across arrays and spill).
template <class E, class S, int MINB, bool CHECK>
__global__ void __launch_bounds__(S::TPA, MINB)
    k_sort_packed_xc(const typename E::Mem* in, typename E::Mem* out, int n) {
    using R = typename E::Reg;
    static_assert(S::LG == 5, "tiles below a warp are xpose.cuh's");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // programmatic dependent launch (see k_sort_packed)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long off = (long long)blockIdx.x * n;
    xc_sort_array<E, S, CHECK>(in + off, out + off, n, int(threadIdx.x), reinterpret_cast<R*>(smem_raw));
}

// k_sort_idlist with the transposed network (one array per CTA): the arrays
// ids[0 .. count) of a CSR batch, count and list position read on the device
// when d_count is set, CTAs pulling arrays from the queue at d_head when set.
template <class E, class S, int MINB = 1>
__global__ void __launch_bounds__(S::TPA, MINB)
    k_sort_idlist_xc(const typename E::Mem* in, typename E::Mem* out, const int* __restrict__ off,
                     const int* __restrict__ ids, int count, const int* d_count, const int* d_base, int* d_head) {
    using R = typename E::Reg;
    static_assert(S::LG == 5, "one array per CTA");
    __shared__ int s_next;
    if (d_count) {
        count = *d_count;
        ids += *d_base;
    }
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* sm = reinterpret_cast<R*>(smem_raw);
    long long g = blockIdx.x;
    for (;;) {
        const int t = thread_index();
        if (d_head) {
            if (t == 0) s_next = atomicAdd(d_head, 1);
            __syncthreads();
            g = s_next;
            __syncthreads();
        }
        if (g >= count) break;  // uniform across the CTA
        const int a = ids[g];
        const long long start = off[a];
        const int na = off[a + 1] - off[a];
        xc_sort_array<E, S, false>(in + start, out + start, na, t, sm);
        __syncthreads();
        if (!d_head) g += gridDim.x;
    }
}

// One cluster of 2^LC CTAs per array, clusters striding over the batch, with
// the transposed network; the arguments are k_sort_cluster's (packed batch
// when ids == nullptr, else the CSR arrays ids[0 .. count)).
template <class E, int LK, int LT, int LC, int MINB = 1>
__global__ void __launch_bounds__(1 << LT, MINB)
    k_sort_cluster_xc(const typename E::Mem* in, typename E::Mem* out, int n, long long arrays, const int* off,
                      const int* ids, const int* d_count) {
    using R = typename E::Reg;
    namespace cg = cooperative_groups;
    constexpr int K = 1 << LK, W = 1 << (LK + LT);
    using Tile = Win<E, LK, LK + LT>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    R* sm = reinterpret_cast<R*>(smem_raw);
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = int(cluster.block_rank());
    const long long cid = (long long)blockIdx.x >> LC;
    const long long clusters = (long long)gridDim.x >> LC;
    const long long count = ids ? (d_count ? (long long)*d_count : arrays) : arrays;
    for (long long i = cid; i < count; i += clusters) {
        const int t = thread_index();
        long long start;
        int na;
        if (ids) {
            const int a = ids[i];
            start = off[a];
            na = off[a + 1] - off[a];
        } else {
            start = i * (long long)n;
            na = n;
        }
        R v[K];
        Tile::load(v, in + start, t, rank * W, na, sm);
        xc_cluster_network<E, LK, LT, LC>(v, t, rank, na - rank * W, sm);
        if constexpr (gathers<E>::value)
            Tile::store_gather(v, in + start, out + start, t, rank * W, na, sm, nullptr, [&] { cluster.sync(); });
        else Tile::store(v, out + start, t, rank * W, na, sm);
    }
}

}  // namespace b200s
