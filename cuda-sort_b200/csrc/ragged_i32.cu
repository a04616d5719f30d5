// Persistent ragged kernel for int32 keys: buckets W = 8 .. 16384, blocked
// families K = 32 (A) and K = 16 (B), 512 threads per CTA, two CTAs per SM.
#include "instantiate.cuh"

namespace b200s {

void register_ragged_i32(std::vector<RaggedEntry>& o) {
    o.push_back(Ragged<ElemI32, ElemI32, 512, 12, 5, 4, 2>::entry(0));
}

}  // namespace b200s
