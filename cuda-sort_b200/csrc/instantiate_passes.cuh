// Launches of the sort in passes (passes.cuh).  Only the passes_*.cu
// translation units include this header.
#pragma once
#include <algorithm>

#include "instantiate.cuh"
#include "passes.cuh"
#include "passes_registry.h"

namespace b200s {

// Slices of 2^(LK+LT) elements (2^LT threads), then two passes per stage up to
// 2^LOGMAX elements.
template <class E, int LK, int LT, int LOGMAX>
struct Passes {
    static constexpr int LOCAL = LK + LT;
    using S = Shape<LK, 5, LT - 5>;
    using Mem = typename E::Mem;
    static constexpr long long kChunk = 1 << 20;  // arrays per round of launches (grids within 2^31)
    // Threads per SM the registers are sized for, as the packed tiles'.
    static constexpr int kSmThreads = sizeof(typename E::Reg) == 16 ? 512 : 1024;

    template <int ST>
    static cudaError_t stages(Mem* data, int n, long long arrays, int logw, int early, cudaStream_t st) {
        if constexpr (ST < LOGMAX) {
            if (ST >= logw) return cudaSuccess;
            constexpr int LOGT = ST - LK + 1, CTA = 1 << (LOGT - LK);
            static_assert(LOGT - LK >= 5, "whole warps");
            cudaError_t e = launch_pdl(k_merge_far<E, LK>, unsigned(arrays << (logw - LK - log2_const(kFarThreads))),
                                       kFarThreads, 0, st, data, n, logw, ST, early);
            if (e != cudaSuccess) return e;
            constexpr size_t SMEM = xc_smem_bytes<E, LK, LOGT>();
            constexpr int PER_SM = kSmThreads / CTA < 32 ? kSmThreads / CTA : 32;
            static std::atomic<unsigned long long> done{0};
            auto near = k_merge_near<E, LK, LOGT, PER_SM>;
            if ((e = opt_in_smem<SMEM>(reinterpret_cast<const void*>(near), done)) != cudaSuccess) return e;
            e = launch_pdl(near, unsigned(arrays << (logw - LOGT)), CTA, SMEM, st, data, n, logw, early);
            return e == cudaSuccess ? stages<ST + 1>(data, n, arrays, logw, early, st) : e;
        } else {
            return cudaSuccess;
        }
    }
    static cudaError_t launch(const void* in, void* out, int n, long long arrays, int logw, cudaStream_t st) {
        constexpr size_t SMEM = xc_smem_bytes<E, LK, LOCAL>();
        static std::atomic<unsigned long long> done{0};
        auto slices = k_sort_slices<E, S, kSmThreads / S::TPA>;
        cudaError_t e = opt_in_smem<SMEM>(reinterpret_cast<const void*>(slices), done);
        for (long long first = 0; e == cudaSuccess && first < arrays; first += kChunk) {
            const long long count = std::min(arrays - first, kChunk);
            const Mem* src = static_cast<const Mem*>(in) + first * n;
            Mem* dst = static_cast<Mem*>(out) + first * n;
            const long long ctas = count << (logw - LOCAL);
            const int early = ctas <= 64 || ctas >= (long long)sm_count() * (kSmThreads / S::TPA);  // see passes.cuh
            e = launch_pdl(slices, unsigned(ctas), S::TPA, SMEM, st, src, dst, n, logw - LOCAL, early);
            if (e == cudaSuccess) e = stages<LOCAL>(dst, n, count, logw, early, st);
        }
        return e;
    }
    static PassesEntry entry(int dtype) { return PassesEntry{dtype, LOCAL, LOGMAX, &launch}; }
};

}  // namespace b200s
