"""CPU check of the kernels launched with programmatic stream serialization
(those that run griddepcontrol.wait): what they read may still be written by the
kernel before them until the wait returns, so no pointer parameter of theirs, or
of the device functions of their file, may be declared constant for the
kernel's whole life (__restrict__), and none is read through the read-only path."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-sort_b200", "csrc")


def functions(text, kind):
    """(name, parameters, body) of the definitions that `kind` introduces."""
    for m in re.finditer(kind, text):
        head = re.compile(r"\b(\w+)\(((?:[^()]|\([^()]*\))*)\)\s*\{").search(text, m.end())
        stop = re.compile(r"[;{]").search(text, m.end())
        if not head or not stop or stop.group() == ";" or stop.start() != head.end() - 1:
            continue
        depth, i = 1, head.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield head.group(1), head.group(2), text[head.end():i]


def sources():
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cuh", ".cu")):
            with open(os.path.join(CSRC, f)) as fh:
                out[f] = re.sub(r"//[^\n]*", "", fh.read())
    return out


def kernels():
    return [(f, name, params, body) for f, text in sources().items()
            for name, params, body in functions(text, r"__global__ void") if "griddepcontrol.wait" in body]


def test_the_dependent_kernels_are_found():
    names = {k[1] for k in kernels()}
    assert names >= {"k_bin_small", "k_sort_ragged", "k_sort_packed", "k_sort_packed_xc", "k_sort_xpose",
                     "k_sort_slices", "k_merge_far", "k_merge_near"}


@pytest.mark.parametrize("kernel", kernels(), ids=lambda k: k[1])
def test_nothing_is_declared_constant_before_the_wait(kernel):
    f, name, params, body = kernel
    assert "__restrict__" not in params, (f, name)
    assert not re.search(r"__ldg\(|ld\.global\.nc", body), (f, name)


def test_device_functions_that_read_the_offsets():
    found = {name: params for name, params, _ in functions(sources()["ragged.cuh"], r"__device__ __forceinline__ void")}
    assert "__restrict__" not in found["ragged_task"]
