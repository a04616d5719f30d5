// int32 keys sorted in passes: slices of 4096 (16 keys per thread, for few
// arrays) and 16384 (32 per thread).
#include "instantiate_passes.cuh"

namespace b200s {

void register_passes_i32(std::vector<PassesEntry>& o) {
    o.push_back(Passes<ElemI32, 4, 8, 17>::entry(0));
    o.push_back(Passes<ElemI32, 5, 9, 17>::entry(0));
}

}  // namespace b200s
