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
    PackedXc<ElemRecI32G, 4, 0, 32>::attach_to(o, 1);
    PackedXc<ElemRecI32G, 4, 1, 16>::attach_to(o, 1);
    PackedXc<ElemRecI32G, 4, 2, 8>::attach_to(o, 1);
    PackedXc<ElemRecI32G, 4, 3, 4>::attach_to(o, 1);
    PackedXc<ElemRecI32G, 4, 4, 2>::attach_to(o, 1);
}

}  // namespace b200s
