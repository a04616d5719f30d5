"""GPU test that the IntAndData record tiles of 32 elements per thread and several
warps have launch form 3 (a table row or a caller may name them), in the form of a
few arrays and in that of a full batch."""
import pytest

import b200sort as bs
import workloads
from test_gpu_parity import check, gpu_sort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log2_warps", [1, 2, 3])
def test_wide_record_tiles_have_form_3(log2_warps):
    tile = bs.Tile(5, 5, log2_warps, 0, 3, 0)
    w = 1 << (10 + log2_warps)
    assert bs.tile_info(bs.I32_I32, w, 0, tile).xpose_form == 1
    for n, arrays in ((w - 3, 2), (w // 2 + 1, 700)):
        for flags in (0, bs.SORTED_CHECK):
            data = workloads.make_packed(bs.I32_I32, n, arrays, "distinct16", seed=n, extremes=True)
            check(bs.I32_I32, 0, data, n, arrays, gpu_sort(bs.I32_I32, data, n, arrays, flags, tile))
