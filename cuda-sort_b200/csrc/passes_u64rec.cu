// {uint64 key, int32 payload} records sorted in passes: slices of 4096 and 8192.
#include "instantiate_passes.cuh"

namespace b200s {

void register_passes_u64rec(std::vector<PassesEntry>& o) {
    o.push_back(Passes<ElemRecU64, 4, 8, 16>::entry(3));
    o.push_back(Passes<ElemRecU64, 4, 9, 16>::entry(3));
}

}  // namespace b200s
