"""CPU test of the windowed network's layout tables (csrc/win_layout.h): a host
program walks the same constexpr tables the kernels use."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def walked(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("win") / "win_layout")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "cuda-sort_b200", "csrc"),
                    os.path.join(ROOT, "tests", "win_layout.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return [tuple(int(x) for x in line.split()) for line in out.splitlines()]


def test_windows_run_the_reference_network_at_unique_addresses(walked):
    assert len(walked) == 2 * (6 + 5 + 5 + 5)
    assert all(ok for _, _, _, ok, _, _ in walked), walked


def test_bank_conflicts_stay_within_the_searched_classes(walked):
    # at most two of a tile's layouts take a second wavefront with 8- and
    # 16-byte elements; int32 tiles keep below one and a half per access
    for lk, logw, m, _, total, accesses in walked:
        assert total <= (accesses + 4 if m < 5 else accesses * 3 // 2), (lk, logw, m, total, accesses)
