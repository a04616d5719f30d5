// Host-side registry of the sort in passes over global memory (passes.cuh).
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace b200s {

struct PassesEntry {
    int dtype;
    int log2_slice;  // elements one CTA sorts before the passes
    int log2_max;    // longest array
    // arrays of n <= 2^logw elements, logw > log2_slice; out aligned to the element
    cudaError_t (*launch)(const void* in, void* out, int n, long long arrays, int logw, cudaStream_t stream);
};

void register_passes_i32(std::vector<PassesEntry>& out);
void register_passes_rec(std::vector<PassesEntry>& out);
void register_passes_u64(std::vector<PassesEntry>& out);
void register_passes_u64rec(std::vector<PassesEntry>& out);

const std::vector<PassesEntry>& passes_registry();

}  // namespace b200s
