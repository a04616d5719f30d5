"""Rows of the tile table and the sort in passes: a row without the passes column
is run as it stands for every batch, the shipped rows allow the passes."""
import os

import numpy as np
import pytest

import b200sort as bs
import workloads

SHIPPED = os.path.join(os.path.dirname(bs.LIB_PATH), "tune", "b200_table.csv")
KEYED = [bs.I32, bs.I32_I32, bs.U64, bs.U64_I32]


@pytest.fixture
def table(tmp_path):
    def load(*rows):
        p = tmp_path / "rows.csv"
        p.write_text("\n".join(rows) + "\n")
        return bs.load_tile_table(str(p))

    yield load
    bs.load_tile_table(SHIPPED)


def row(dtype, tile, form, *more):
    return ",".join(str(x) for x in (dtype, 0, sum(tile.as_tuple()), tile.log2_items, tile.log2_lanes,
                                     tile.log2_warps, form) + more)


def tiles_of(dtype, w, clusters):
    return [t for t in bs.tiles(dtype) if sum(t.as_tuple()) == w and (t.log2_ctas > 0) == clusters]


@pytest.mark.parametrize("dtype", KEYED)
def test_shipped_rows_allow_the_passes(dtype):
    top = bs.max_length(dtype)
    assert bs.packed_slice(dtype, top, 1) > 0 and bs.packed_slice(dtype, top, 256) > 0
    assert bs.packed_slice(dtype, 5000, 1) > 0       # one array of one CTA's length, spread over many
    assert bs.packed_slice(dtype, 5000, 4000) == 0   # many of them: their tile
    assert bs.packed_slice(dtype, 4096, 1) == 0
    for n in (5000, top):
        assert bs.packed_slice(dtype, n, 1, bs.STABLE) == (0 if dtype in (bs.I32_I32, bs.U64_I32) else
                                                            bs.packed_slice(dtype, n, 1))


@pytest.mark.parametrize("dtype", KEYED)
def test_a_row_is_run_as_it_stands(table, dtype):
    for w, clusters in ((15, True), (16, True), (13, False)):
        for tile in tiles_of(dtype, w, clusters):
            more = (tile.log2_ctas,) if tile.log2_ctas else ()
            assert table(row(dtype, tile, 3, *more)) == 1
            assert bs.default_tile(dtype, 1 << w).as_tuple() == tile.as_tuple()
            assert [bs.packed_slice(dtype, 1 << w, a) for a in (1, 64, 4096)] == [0, 0, 0]
            if 2 << w <= bs.max_length(dtype):
                assert bs.packed_slice(dtype, (1 << w) + 1, 1) > 0   # the next length keeps its row
            table(row(dtype, tile, 3, tile.log2_ctas, 0))
            assert bs.packed_slice(dtype, 1 << w, 1) == 0
            table(row(dtype, tile, 3, tile.log2_ctas, 1))
            assert bs.packed_slice(dtype, 1 << w, 1) > 0


def test_bad_column(table):
    tile = tiles_of(bs.I32_I32, 13, False)[0]
    with pytest.raises(bs.B200SortError):
        table(row(bs.I32_I32, tile, 3, 0, 2))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", KEYED)
def test_rows_sort_like_the_oracle(table, dtype):
    from test_gpu_parity import check, gpu_sort
    for w, clusters in ((15, True), (13, False)):
        tile = tiles_of(dtype, w, clusters)[0]
        n = (1 << w) - 77
        for arrays in (1, 5):
            data = workloads.make_packed(dtype, n, arrays, "distinct16", seed=n, extremes=True)
            outs = []
            for passes in (0, 1):
                table(row(dtype, tile, 3, tile.log2_ctas, passes))
                outs.append(gpu_sort(dtype, data, n, arrays, 0))
                check(dtype, 0, data, n, arrays, outs[-1])
            assert np.array_equal(*outs)
