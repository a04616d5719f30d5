// Records in the reference tie order, sorted in passes: slices of 4096, 8192
// and 16384.
#include "instantiate_passes.cuh"

namespace b200s {

void register_passes_rec(std::vector<PassesEntry>& o) {
    o.push_back(Passes<ElemRecI32, 4, 8, 16>::entry(1));
    o.push_back(Passes<ElemRecI32, 4, 9, 16>::entry(1));
    o.push_back(Passes<ElemRecI32, 4, 10, 16>::entry(1));
}

}  // namespace b200s
