"""Block maps of the batched engine (no GPU needed): every tile and group that a batch can
have must come back from the word that names it."""

import ctypes as C

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


@pytest.mark.parametrize("single", [0, 1])
@pytest.mark.parametrize("level0", [0, 1])
@pytest.mark.parametrize("spn", [1, 3, 64, 1024, 1025, 4096, 4097, 8192])
def test_group_width_names_every_problem(lib, single, level0, spn):
    """8192 problems of a structure fit in both precisions, with or without a lone problem
    of another structure, on launches that leave SMs idle and on those that do not."""
    for others in ([], [1]):
        for blocks in (1, 1000):
            probs = (C.c_int * (1 + len(others)))(spn, *others)
            rows = (C.c_int * len(probs))(*([blocks] * len(probs)))
            gs = lib.bm_pat_group(single, level0, 148, len(probs), probs, rows)
            most, usual = (4, 4 if single else 2) if level0 else (8, 8 if single else 4)
            assert 1 <= gs <= most and -(-spn // gs) <= lib.bm_max_groups(level0)
            if -(-spn // usual) <= lib.bm_max_groups(level0):
                assert gs <= usual
            if blocks == 1000 and -(-spn // usual) <= lib.bm_max_groups(level0):
                assert gs == usual   # every SM has a block
