// uint64 keys sorted in passes: slices of 4096, 8192 and 16384.
#include "instantiate_passes.cuh"

namespace b200s {

void register_passes_u64(std::vector<PassesEntry>& o) {
    o.push_back(Passes<ElemU64, 4, 8, 16>::entry(2));
    o.push_back(Passes<ElemU64, 4, 9, 16>::entry(2));
    o.push_back(Passes<ElemU64, 4, 10, 16>::entry(2));
}

}  // namespace b200s
