// Persistent ragged kernel for stable IntAndData records (see ragged_rec.cu).
#include "instantiate.cuh"

namespace b200s {

void register_ragged_rec_stable(std::vector<RaggedEntry>& o) {
    o.push_back(Ragged<ElemRecI32S, ElemRecI32G, 512, 11, 4, 3, 2>::entry(1));
}

}  // namespace b200s
