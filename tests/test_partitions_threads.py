"""b200s_sort_partitions from several host threads on one stream: its plan is
cached and hidden from the caller, so the calls themselves have to take turns.
On the CPU csrc/partitions.cu runs over a fake of the plan functions; on the GPU
two threads sort different batches on one stream."""
import os
import subprocess
import threading

import numpy as np
import pytest

import b200sort as bs
import workloads
from gpu_util import empty_device, from_device, stream_handle, to_device

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def test_calls_on_one_stream_take_turns(tmp_path):
    exe = str(tmp_path / "partitions_threads")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "partitions_threads.cpp"),
                    "-x", "c++", os.path.join(ROOT, "cuda-sort_b200", "csrc", "partitions.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=60).stdout
    calls, overlaps, dead, small = (int(x) for x in out.split())
    assert calls == 4 * 200
    assert (overlaps, dead, small) == (0, 0, 0)


@pytest.mark.gpu
def test_two_threads_on_one_stream():
    import torch
    from test_ragged_gpu import check
    dtype, calls, st = bs.I32_I32, 40, stream_handle()
    work = []
    for t in range(2):
        lengths = workloads.ragged_lengths(2000 + 700 * t, max_len=3000, seed=t)
        data, off = workloads.make_ragged(dtype, lengths, "distinct16", seed=t)
        d_in = to_device(data)
        outs = [empty_device(d_in.numel()) for _ in range(calls)]
        work.append((data, off, d_in, torch.from_numpy(off.astype(np.int32)).cuda(), outs))
    torch.cuda.synchronize()
    start, errors = threading.Barrier(2), []

    def caller(t):
        _, off, d_in, d_off, outs = work[t]
        try:
            start.wait()
            for d_out in outs:
                bs.sort_partitions(dtype, d_in.data_ptr(), d_out.data_ptr(), d_off.data_ptr(), len(off) - 1, 0, 0, st)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=caller, args=(t,)) for t in range(2)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not errors, errors
    for data, off, _, _, outs in work:
        for d_out in (outs[0], outs[calls // 2], outs[-1]):
            check(dtype, 0, data, off, from_device(d_out[:data.nbytes], bs.NP_DTYPES[dtype]))
        first = outs[0][:data.nbytes]
        assert all(torch.equal(first, o[:data.nbytes]) for o in outs)
    bs.lib().b200s_release_partition_plans()
