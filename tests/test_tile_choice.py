"""The index lists of a step's prompt portions, by what a mixer asks for (engine/batch.py), and which attention kernel gets them."""
import pytest
import torch

from gollmgo_b200.cache import CacheManager, PagedKVNeed
from gollmgo_b200.engine import BatchBuilder, StepEntry
from gollmgo_b200.parts.attention import TILES_TC, TILES_TC_X, Attention
from gollmgo_b200.parts.context import QueryTiles


def step(lens, held, lists):
    pages = sum(-(-(a + b) // 16) for a, b in zip(lens, held)) + 1
    cm = CacheManager([PagedKVNeed(1, 64, None)], 16, pages, len(lens), dtype=torch.bfloat16, device="cpu")
    for i, h in enumerate(held):
        cm.admit(i)
        if h:
            cm.append(i, h)
    return BatchBuilder(cm, "cpu", query_tiles=lists).build([StepEntry(i, [0] * n, [0]) for i, n in enumerate(lens)])


def pairs(tiles):
    return list(zip(tiles.seq.tolist(), tiles.q0.tolist()))[:tiles.count]


@pytest.mark.parametrize("lens,held,some", [([144], [0], False), ([145], [0], True), ([2, 30], [143, 0], True), ([2, 30], [142, 0], False),
                                            ([1, 16], [4000, 0], False), ([300, 1, 7], [0, 9, 0], True)])
def test_tiles_only_beyond_so_many_keys(lens, held, some):
    """A portion decides for the step; a decoded token's keys do not count."""
    batch = step(lens, held, [TILES_TC, TILES_TC_X])
    assert pairs(batch.tiles[TILES_TC_X]) == (pairs(batch.tiles[TILES_TC]) if some else [])


def test_lists_of_one_height_are_lists_of_their_own():
    lists = [QueryTiles(128), QueryTiles(128, at_least=256), QueryTiles(128, beyond_keys=1000), TILES_TC]
    assert len(set(lists)) == 4
    batch = step([300, 40], [0, 0], lists)
    assert [batch.tiles[x].count for x in lists] == [4, 3, 0, 4]


@pytest.mark.parametrize("lens,held,tc", [([32] * 32, [0] * 32, False), ([32] * 32, [100] * 32, False), ([160] * 8, [0] * 8, True),
                                          ([256], [0], False), ([257], [0], True), ([512, 16], [0, 0], True)])
def test_many_short_portions_with_options_stay_on_mma(lens, held, tc):
    batch = step(lens, held, [TILES_TC_X])
    layer = Attention.__new__(Attention)
    layer._mma_x, layer.nh, layer.num_sms, layer.window = True, 32, 148, None
    assert bool(layer.long_tiles(batch)) == tc


@pytest.mark.parametrize("window,chunk,lens,tc", [(64, 0, [2048], False), (128, 0, [2048], True), (128, 0, [300], False), (257, 0, [300], True),
                                                  (None, 64, [2048], False), (None, 512, [300], True), (1024, 0, [2048], True),
                                                  (1024, 100, [2048], False), (0, 0, [300], True)])
def test_short_windows_and_chunks_stay_on_mma(window, chunk, lens, tc):
    batch = step(lens, [0] * len(lens), [TILES_TC_X])
    layer = Attention.__new__(Attention)
    layer._mma_x, layer.nh, layer.num_sms, layer.window, layer.chunk = True, 32, 148, window, chunk
    assert bool(layer.long_tiles(batch)) == tc
