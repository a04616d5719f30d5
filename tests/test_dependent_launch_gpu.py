"""GPU test of the ragged kernels' programmatic dependent launch: the offsets
are written by the kernel just before the call, one that lets its successor
start early, into one buffer that holds other offsets each time."""
import numpy as np
import pytest

import b200sort as bs
import workloads
from gpu_util import empty_device, from_device, stream_handle, to_device
from test_ragged_gpu import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arrays", [1500, 4000, 6000])
def test_offsets_written_by_the_previous_kernel(arrays):
    import torch
    dtype, rounds, st = bs.I32_I32, 6, stream_handle()
    rng = np.random.default_rng(arrays)
    lengths = workloads.ragged_lengths(arrays, max_len=700, seed=arrays)
    data, _ = workloads.make_ragged(dtype, lengths, "distinct16", seed=arrays)
    d_in = to_device(data)
    offs, shuffled, outs = [], [], []
    for _ in range(rounds):
        off = np.concatenate([[0], np.cumsum(rng.permutation(lengths))]).astype(np.int32)
        offs.append(off)
        shuffled.append(torch.from_numpy(rng.permutation(off)).cuda())
        outs.append(empty_device(d_in.numel()))
    d_off = torch.from_numpy(offs[-1]).cuda()
    torch.cuda.synchronize()
    with bs.Plan(dtype, arrays) as plan:
        for src, d_out in zip(shuffled, outs):
            # the sorted offsets are the batch's offsets
            bs.sort_packed(bs.I32, src.data_ptr(), d_off.data_ptr(), arrays + 1, 1, 0, None, st)
            plan.sort(d_in.data_ptr(), d_out.data_ptr(), d_off.data_ptr(), arrays, st)
        torch.cuda.synchronize()
    for off, d_out in zip(offs, outs):
        check(dtype, 0, data, off.astype(np.int64), from_device(d_out[:data.nbytes], bs.NP_DTYPES[dtype]))
