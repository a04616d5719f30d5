"""GPU parity of the packed launches around the limit of the latency form (four
warps per SM), with and without the sortedness check."""
import numpy as np
import pytest

import b200sort as bs
import workloads
from test_gpu_parity import check, gpu_sort

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [bs.I32_I32, bs.U64])
@pytest.mark.parametrize("n", [33, 64, 129, 256, 257, 512, 700, 1024, 1500, 2048])
def test_both_forms_around_the_limit(dtype, n):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    tile = bs.default_tile(dtype, n)
    per_warp = max(1, 32 >> tile.log2_lanes) if tile.log2_warps == 0 else 1
    limit = 4 * sms * per_warp >> tile.log2_warps
    for arrays in (3, limit, limit + 1):
        for dist in ("distinct16", "swap8", "sorted"):
            data = workloads.make_packed(dtype, n, arrays, dist, seed=n, extremes=dist != "sorted")
            plain = gpu_sort(dtype, data, n, arrays, 0)
            check(dtype, 0, data, n, arrays, plain)
            assert np.array_equal(plain, gpu_sort(dtype, data, n, arrays, bs.SORTED_CHECK))
            assert np.array_equal(plain, gpu_sort(dtype, data, n, arrays, bs.SORTED_CHECK, inplace=True))
