"""CPU test of the windowed network: the kernels' own code (csrc/win.cuh and
csrc/cta_xpose.cuh, single-CTA tiles and clusters) built for the host over
simulated threads, see win_network.cpp.  Results, tie order included, against the
reference's network, with warps run in several orders between barriers, lengths
that leave warps of padding, both buffers off their alignment, and in place."""
import concurrent.futures
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TESTS = os.path.join(ROOT, "tests")
TILES = {"i32": 3, "i32_check": 1, "i32_16": 1, "rec": 6, "rec_check": 1, "rec_32": 1, "rec_32_check": 1, "stable": 2,
         "stable_check": 1, "u64": 2, "u64_check": 1, "rec16": 5, "rec16_check": 1}


@pytest.fixture(scope="module")
def simulated(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("win_network")

    def part(k):
        exe = str(tmp / ("part%d" % k))
        subprocess.run(["g++", "-std=c++17", "-O1", "-DPART=%d" % k, "-fsanitize=alignment",
                        "-fno-sanitize-recover=alignment", "-I" + os.path.join(TESTS, "host_cuda"),
                        "-I" + os.path.join(ROOT, "cuda-sort_b200", "csrc"), os.path.join(TESTS, "win_network.cpp"),
                        "-o", exe], check=True, capture_output=True)
        return subprocess.run([exe], check=True, capture_output=True, text=True, timeout=300).stdout

    with concurrent.futures.ThreadPoolExecutor(8) as ex:
        out = "".join(ex.map(part, range(8)))
    return [line.split() for line in out.splitlines()]


def test_every_tile_is_simulated(simulated):
    names = [line[0] for line in simulated]
    assert {n: names.count(n) for n in set(names)} == TILES


def test_results_match_the_reference_network(simulated):
    assert [line for line in simulated if line[3] != "0"] == []
