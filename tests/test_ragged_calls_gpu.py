"""GPU tests of a ragged plan's call paths: the one-launch binning around its
limits, direct launches for new buffers and the graph for repeated ones, calls
from two streams, record buffers that are only 4-byte aligned."""
import numpy as np
import pytest

import b200sort as bs
import workloads
from gpu_util import empty_device, from_device, stream_handle, to_device
from test_ragged_gpu import check

pytestmark = pytest.mark.gpu

TYPES = [(bs.I32, 0), (bs.I32_I32, 0), (bs.I32_I32, bs.STABLE), (bs.U64, 0), (bs.U64_I32, 0), (bs.U64_I32, bs.STABLE)]


def batch(dtype, flags, arrays, seed, longest=None):
    top = bs.ragged_max_length(dtype, flags)
    lengths = workloads.ragged_lengths(arrays, max_len=700, seed=seed)
    lengths[::7] = 0
    if arrays > 20:
        lengths[3], lengths[9], lengths[15] = 8193, 3000, 1025
    lengths[arrays // 2] = longest or min(top, 20000)
    return workloads.make_ragged(dtype, lengths, "distinct16", seed=seed, extremes=True)


def device(data, off):
    import torch
    d_in = to_device(data)
    return d_in, empty_device(d_in.numel()), torch.from_numpy(off.astype(np.int32)).cuda()


@pytest.mark.parametrize("dtype,flags", TYPES)
@pytest.mark.parametrize("arrays", [1, 33, 1023, 1025, 4096, 4097])
def test_direct_then_graph_then_new_buffers(dtype, flags, arrays):
    import torch
    st = stream_handle()
    with bs.Plan(dtype, arrays, flags) as plan:
        for seed in (1, 2):
            data, off = batch(dtype, flags, arrays, seed)
            d_in, d_out, d_off = device(data, off)
            for _ in range(4):      # direct, capture and replay, replay, replay
                d_out.zero_()
                plan.sort(d_in.data_ptr(), d_out.data_ptr(), d_off.data_ptr(), arrays, st)
                torch.cuda.synchronize()
                check(dtype, flags, data, off, from_device(d_out[:data.nbytes], bs.NP_DTYPES[dtype]))


def test_calls_alternating_between_two_streams():
    import torch
    dtype, arrays = bs.I32_I32, 2000
    sets = [batch(dtype, 0, arrays, seed) for seed in range(6)]
    bufs = [device(*s) for s in sets]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    with bs.Plan(dtype, arrays) as plan:
        for i, (d_in, d_out, d_off) in enumerate(bufs):
            plan.sort(d_in.data_ptr(), d_out.data_ptr(), d_off.data_ptr(), arrays, streams[i % 2].cuda_stream)
        torch.cuda.synchronize()
    for (data, off), (_, d_out, _) in zip(sets, bufs):
        check(dtype, 0, data, off, from_device(d_out[:data.nbytes], bs.NP_DTYPES[dtype]))


@pytest.mark.parametrize("arrays", [50, 5000])
def test_arrays_beyond_every_kernel_are_counted_and_left(arrays):
    import torch
    dtype = bs.I32_I32
    top = bs.ragged_max_length(dtype)
    data, off = batch(dtype, 0, arrays, 3, longest=top + 1)
    d_in, d_out, d_off = device(data, off)
    d_out.fill_(0xAB)
    with bs.Plan(dtype, arrays) as plan:
        plan.sort(d_in.data_ptr(), d_out.data_ptr(), d_off.data_ptr(), arrays, stream_handle())
        torch.cuda.synchronize()
        assert plan.too_long(stream_handle()) == 1
    a = arrays // 2
    got = from_device(d_out[:data.nbytes], np.uint8)
    assert np.all(got[off[a] * 8:off[a + 1] * 8] == 0xAB)


@pytest.mark.parametrize("flags", [0, bs.STABLE])
def test_records_in_a_buffer_that_is_only_word_aligned(flags):
    import torch
    dtype, arrays = bs.I32_I32, 300
    data, off = batch(dtype, flags, arrays, 4)
    d_in = torch.empty(data.nbytes + 16, dtype=torch.uint8, device="cuda")
    d_out = torch.empty_like(d_in)
    d_in[4:4 + data.nbytes] = torch.from_numpy(data.view(np.uint8).copy()).cuda()
    d_off = torch.from_numpy(off.astype(np.int32)).cuda()
    with bs.Plan(dtype, arrays, flags) as plan:
        for out in (d_out, d_in):   # out of place, then in place
            plan.sort(d_in.data_ptr() + 4, out.data_ptr() + 4, d_off.data_ptr(), arrays, stream_handle())
            torch.cuda.synchronize()
            check(dtype, flags, data, off, from_device(out[4:4 + data.nbytes].clone(), bs.NP_DTYPES[dtype]))
    for n in (3000, 700):           # packed: a windowed tile, misaligned
        arr = workloads.make_packed(dtype, n, 20, "distinct16", seed=n, extremes=True)
        d_in[4:4 + arr.nbytes] = torch.from_numpy(arr.view(np.uint8).copy()).cuda()
        bs.sort_packed(dtype, d_in.data_ptr() + 4, d_out.data_ptr() + 4, n, 20, flags, None, stream_handle())
        torch.cuda.synchronize()
        check(dtype, flags, arr, np.arange(21, dtype=np.int64) * n,
              from_device(d_out[4:4 + arr.nbytes].clone(), bs.NP_DTYPES[dtype]))


@pytest.mark.parametrize("dtype,flags", TYPES)
def test_sorted_check_sees_runs_out_of_order(dtype, flags):
    # sorted arrays whose 16- or 32-element runs trade places by a swap of two
    # bits of the run's number: every run is in order, the array is not
    import torch
    n, arrays = 2048, 11
    base = workloads.make_packed(dtype, n, arrays, "sorted", seed=5).reshape(arrays, n)
    for run in (16, 32):
        runs = np.arange(n // run)
        bits = (n // run).bit_length() - 1
        data = base.copy()
        for a in range(1, arrays):
            i, j = a % bits, (a * 3 + 1) % bits
            x = ((runs >> i) ^ (runs >> j)) & 1
            order = runs ^ (x << i) ^ (x << j)
            data[a] = base[a].reshape(-1, run)[order].reshape(-1)
        flat = data.reshape(-1)
        if dtype in (bs.I32_I32, bs.U64_I32):
            flat["data"] = np.arange(flat.shape[0])
        d_in, off = to_device(flat), np.arange(arrays + 1, dtype=np.int64) * n
        for d_out in (empty_device(d_in.numel()), d_in):
            bs.sort_packed(dtype, d_in.data_ptr(), d_out.data_ptr(), n, arrays, flags | bs.SORTED_CHECK, None,
                           stream_handle())
            torch.cuda.synchronize()
            check(dtype, flags, flat, off, from_device(d_out[:flat.nbytes], bs.NP_DTYPES[dtype]))
