"""Block maps of the batched engine (no GPU needed): every tile and group that a batch can
have must come back from the word that names it."""

import pytest

import native_build


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return native_build.load("batch_maps", tmp_path_factory.mktemp("native"))


@pytest.mark.parametrize("spn", [1, 32, 33, 2048, 2049, 4097, 8192, 131072])
@pytest.mark.parametrize("rows", [1, 17, 2048])
def test_tail_tiles_come_back(lib, spn, rows):
    cols = lib.bm_tail_cols(spn)
    assert cols == -(-spn // 32)
    row_tiles = -(-rows // 16)
    for rt in {0, row_tiles // 2, row_tiles - 1}:
        for ct in {0, 63, 64, 127, cols - 1}:
            if ct >= cols:
                continue
            tile = lib.bm_tail_tile(rt, ct)
            assert (lib.bm_tail_row(tile), lib.bm_tail_col(tile)) == (rt, ct)


def test_tail_tiles_beyond_the_map_are_refused(lib):
    assert lib.bm_tail_cols(131073) == -1
