"""GPU parity of 16-byte records in buffers that are not aligned to the record:
the lengths of the windowed tiles (packed, passes, clusters) and of the
persistent ragged kernel's windowed classes, 4, 8 and 12 bytes off."""
import numpy as np
import pytest

import b200sort as bs
import workloads
from gpu_util import empty_device, from_device, stream_handle, to_device
from test_ragged_gpu import check

pytestmark = pytest.mark.gpu

DTYPE = bs.U64_I32


def off_by(data, shift):
    buf = empty_device(data.nbytes + 16)
    if shift:
        assert buf.data_ptr() % 16 == 0
    buf[shift:shift + data.nbytes] = to_device(data)
    return buf


def sort_and_check(sort, flags, data, off, shift_in, shift_out):
    import torch
    d_in = off_by(data, shift_in)
    d_out = d_in if shift_out is None else empty_device(data.nbytes + 16)
    at = shift_in if shift_out is None else shift_out
    sort(d_in.data_ptr() + shift_in, d_out.data_ptr() + at)
    torch.cuda.synchronize()
    check(DTYPE, flags, data, off, from_device(d_out[at:at + data.nbytes].clone(), bs.NP_DTYPES[DTYPE]))


@pytest.mark.parametrize("flags", [0, bs.STABLE])
@pytest.mark.parametrize("shift_in,shift_out", [(8, 8), (4, 12), (8, 0), (0, 4), (12, None)])
def test_packed_and_ragged(flags, shift_in, shift_out):
    for n in (513, 1024, 1100, 3000, 4096, 8000, 9000, 20000):
        assert bs.default_tile(DTYPE, n, flags).persistent == 3  # a windowed tile
        data = workloads.make_packed(DTYPE, n, 5, "distinct16", seed=n, extremes=True)
        sort_and_check(lambda i, o: bs.sort_packed(DTYPE, i, o, n, 5, flags, None, stream_handle()), flags, data,
                       np.arange(6, dtype=np.int64) * n, shift_in, shift_out)
    rng = np.random.default_rng(7)
    lengths = np.concatenate([rng.integers(257, 4097, size=60), [257, 512, 513, 4096, 4097, 9000]])
    data, off = workloads.make_ragged(DTYPE, lengths, "distinct16", seed=3, extremes=True)
    d_off = to_device(off.astype(np.int32))
    with bs.Plan(DTYPE, len(lengths), flags) as plan:
        sort_and_check(lambda i, o: plan.sort(i, o, d_off.data_ptr(), len(lengths), stream_handle()), flags, data, off,
                       shift_in, shift_out)
