// Persistent ragged kernels for {uint64 key, int32 payload} records: buckets
// W = 8 .. 4096, 256 threads per CTA (their 16-byte registers double the
// shared-memory tile), two CTAs per SM.
#include "instantiate.cuh"

namespace b200s {

void register_ragged_u64rec(std::vector<RaggedEntry>& o) {
    o.push_back(Ragged<ElemRecU64, ElemRecU64, 256, 10, 4, 3, 2>::entry(3));
    o.push_back(Ragged<ElemRecU64S, ElemRecU64S, 256, 10, 4, 3, 2>::entry(3));
}

}  // namespace b200s
