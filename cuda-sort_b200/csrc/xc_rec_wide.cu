// Launch form 3 of the IntAndData record tiles of several warps with 32 elements
// per thread, by request: the table's 16 per thread are faster, but a table row
// or a caller may name these.  Full batches of 4 M records, W = 2048 / 4096 /
// 8192: 54 / 66 / 78 us (blocked form 77 / 90 / 123).
#include "instantiate_xc.cuh"

namespace b200s {

void register_xc_rec_wide(std::vector<KernelEntry>& o) {
    PackedXc<ElemRecI32, 5, 1, 8, ElemRecI32L>::attach_to(o, 1);  // W = 2048
    PackedXc<ElemRecI32, 5, 2, 4, ElemRecI32L>::attach_to(o, 1);
    PackedXc<ElemRecI32, 5, 3, 2, ElemRecI32L>::attach_to(o, 1);  // W = 8192
}

}  // namespace b200s
