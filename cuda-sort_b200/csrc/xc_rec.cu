// Launch form 3 of the IntAndData record tiles of a warp and more (reference
// tie order and stable): the network of win.cuh, one array per CTA.  MINB: 64
// registers per thread; the stable records run as 64-bit words too
// (ElemRecI32G).
#include "instantiate_xc.cuh"

namespace b200s {

void register_xc_rec(std::vector<KernelEntry>& o) {
    PackedXc<ElemRecI32, 4, 0, 32, ElemRecI32L>::attach_to(o, 1);  // W = 512
    PackedXc<ElemRecI32, 4, 1, 16, ElemRecI32L>::attach_to(o, 1);
    PackedXc<ElemRecI32, 4, 2, 8, ElemRecI32L>::attach_to(o, 1);
    PackedXc<ElemRecI32, 4, 3, 4>::attach_to(o, 1);
    PackedXc<ElemRecI32, 4, 4, 2>::attach_to(o, 1);  // W = 8192
    // 32 records per thread, by request: the table's 16 per thread are faster,
    // but a table row or a caller may name these.  Full batches of 4 M records, W =
    // 2048 / 4096 / 8192: 54 / 65 / 77 us (blocked form 77 / 90 / 123).
    PackedXc<ElemRecI32, 5, 1, 8, ElemRecI32L>::attach_to(o, 1);  // W = 2048
    PackedXc<ElemRecI32, 5, 2, 4, ElemRecI32L>::attach_to(o, 1);
    PackedXc<ElemRecI32, 5, 3, 2, ElemRecI32L>::attach_to(o, 1);  // W = 8192
    PackedXc<ElemRecI32G, 4, 0, 32>::attach_to(o, 1);
    PackedXc<ElemRecI32G, 4, 1, 16>::attach_to(o, 1);
    PackedXc<ElemRecI32G, 4, 2, 8>::attach_to(o, 1);
    PackedXc<ElemRecI32G, 4, 3, 4>::attach_to(o, 1);
    PackedXc<ElemRecI32G, 4, 4, 2>::attach_to(o, 1);
}

}  // namespace b200s
