// Persistent ragged kernel for uint64 keys: buckets W = 8 .. 8192, blocked
// families K = 16 (A) and K = 8 (B), 512 threads per CTA, two CTAs per SM.
#include "instantiate.cuh"

namespace b200s {

void register_ragged_u64(std::vector<RaggedEntry>& o) {
    o.push_back(Ragged<ElemU64, ElemU64, 512, 11, 4, 3, 2>::entry(2));
}

}  // namespace b200s
