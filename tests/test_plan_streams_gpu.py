"""GPU test of a plan's order between streams that share one handle: the
per-thread default stream is another stream in each host thread, so calls of
two threads that take turns on the host are on two streams."""
import threading

import numpy as np
import pytest

import b200sort as bs
import workloads
from gpu_util import empty_device, from_device, to_device
from test_ragged_gpu import check

pytestmark = pytest.mark.gpu

PER_THREAD_STREAM = 2  # cudaStreamPerThread


@pytest.mark.parametrize("flags", [0, bs.PLAN_NO_GRAPH])
def test_per_thread_streams_of_two_host_threads(flags):
    import torch
    dtype, calls = bs.I32_I32, 8
    batches, bufs = [], []
    for i in range(calls):
        # a long batch, then a short one that would overtake it
        lengths = workloads.ragged_lengths(30000 if i % 2 == 0 else 900, max_len=1500, seed=i)
        data, off = workloads.make_ragged(dtype, lengths, "distinct16", seed=i)
        d_in = to_device(data)
        batches.append((data, off))
        bufs.append((d_in, empty_device(d_in.numel()), torch.from_numpy(off.astype(np.int32)).cuda()))
    torch.cuda.synchronize()
    turn, errors = [threading.Semaphore(1), threading.Semaphore(0)], []
    with bs.Plan(dtype, 30000, flags) as plan:

        def caller(t):
            for i in range(t, calls, 2):
                turn[t].acquire()
                try:
                    d_in, d_out, d_off = bufs[i]
                    plan.sort(d_in.data_ptr(), d_out.data_ptr(), d_off.data_ptr(), d_off.numel() - 1, PER_THREAD_STREAM)
                except Exception as e:  # reported by the main thread
                    errors.append(e)
                turn[1 - t].release()

        threads = [threading.Thread(target=caller, args=(t,)) for t in range(2)]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        torch.cuda.synchronize()
    assert not errors, errors
    for (data, off), (_, d_out, _) in zip(batches, bufs):
        check(dtype, 0, data, off, from_device(d_out[:data.nbytes], bs.NP_DTYPES[dtype]))
