"""CPU check of the launch rules that depend on the size of the GPU: they ask the
device for its SMs (sm_count) and hold no SM count of their own."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cuda-sort_b200", "csrc")


def test_no_rule_holds_an_sm_count():
    for f in sorted(os.listdir(CSRC)):
        with open(os.path.join(CSRC, f)) as fh:
            code = re.sub(r"//[^\n]*", "", fh.read())
        if f == "capi.cu":  # sm_count itself, where no device answers
            code = re.sub(r"int sm_count\(\) \{.*?\n\}", "", code, flags=re.S)
        # 148 SMs, and small multiples of them
        for m in re.finditer(r"(?<![\w.])(\d+)(?![\w.])", code):
            assert int(m.group(1)) not in {148 * k for k in (1, 2, 3, 4, 8, 16)}, (f, m.group(0))
