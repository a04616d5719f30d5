"""CPU test of the tuner's choice of a packed row: the fastest tile on a full batch,
or one a little slower that is faster on a batch of a few arrays, as the shipped
table's rows record it."""
import os
import re

import b200sort as bs
import tune_b200

TABLE = os.path.join(os.path.dirname(bs.LIB_PATH), "tune", "b200_table.csv")


def pick(full, few):
    order = sorted(range(len(full)), key=lambda i: full[i])
    k = tune_b200.pick_row([(full[i], 0.0, i) for i in order], lambda tile: few[tile])
    return order[k]


def test_fastest_unless_a_near_one_has_less_latency():
    assert pick([10.0, 10.5], [4.0, 3.9]) == 0       # near, but no faster on a few arrays
    assert pick([10.0, 10.5], [4.0, 3.5]) == 1
    assert pick([10.0, 11.0], [4.0, 2.0]) == 0       # not near
    assert pick([10.5, 10.0, 10.2], [2.0, 4.0, 3.0]) == 0
    assert pick([10.0], [4.0]) == 0


def test_the_shipped_rows_kept_for_a_few_arrays_follow_the_rule():
    kept = re.compile(r"# ([\d.]+) us; kept over \S+ at ([\d.]+):.* takes ([\d.]+) us instead of ([\d.]+)")
    with open(TABLE) as f:
        rows = [[float(x) for x in m.groups()] for m in map(kept.search, f) if m]
    assert rows
    for own, fastest, own_few, fastest_few in rows:
        assert pick([fastest, own], [fastest_few, own_few]) == 1
