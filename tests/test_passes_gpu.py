"""GPU parity of batches sorted in passes over global memory (csrc/passes.cuh):
batch sizes around the rules that choose the slices, lengths at the edges of
slices and of a stage's blocks, the other forms beside them."""
import numpy as np
import pytest

import b200sort as bs
import workloads
from test_gpu_parity import check, gpu_sort

pytestmark = pytest.mark.gpu

SMS = 148


@pytest.mark.parametrize("dtype", [bs.I32, bs.I32_I32, bs.U64, bs.U64_I32])
@pytest.mark.parametrize("n", [4097, 6145, 8191, 8192, 8193, 12000, 16384, 16385, 24577, 32768, 49409, 65533, 65536,
                               65537, 131072])
def test_passes_match_the_oracle(dtype, n):
    if n > bs.max_length(dtype):
        pytest.skip("beyond this type's longest array")
    w = 1 << (n - 1).bit_length()
    counts = {1, max(1, SMS * 4096 // w), SMS * 4096 // w + 1, SMS * 8192 // w + 1, SMS * 16384 // w + 2}
    for i, arrays in enumerate(sorted(c for c in counts if c * n <= 3 << 20)):
        dist = ("distinct16", "uniform", "swap8", "sorted")[i % 4]
        data = workloads.make_packed(dtype, n, arrays, dist, seed=n + arrays, extremes=True)
        check(dtype, 0, data, n, arrays, gpu_sort(dtype, data, n, arrays, 0, inplace=i % 2 == 1))


@pytest.mark.parametrize("flags", [bs.SORTED_CHECK, bs.STABLE, bs.STABLE | bs.SORTED_CHECK])
def test_flags_keep_their_forms(flags):
    for n in (8000, 16384, 30000):
        data = workloads.make_packed(bs.I32_I32, n, 3, "distinct16", seed=n, extremes=True)
        check(bs.I32_I32, flags & bs.STABLE, data, n, 3, gpu_sort(bs.I32_I32, data, n, 3, flags))
