"""The first level of the multigrid's cluster tail: its shared memory holds every level from there on, also on thin strips."""
import ctypes

import pytest

from difffea_b200 import _lib
from difffea_b200.multigrid import COARSEST_NODES, _coarser

NODE_BYTES = 6 * 16 + 36 * 8          # five vectors, 1 / D and the node's nine 2 x 2 blocks
LIMIT = 227 * 1024 - 2048             # what a block may take beside a static buffer of 2 KB
TAIL_NODES = 6000


def _hierarchy(gx, gy):
    levels = [(gx, gy)]
    while (levels[-1][0] + 1) * (levels[-1][1] + 1) > COARSEST_NODES or len(levels) < 2:
        levels.append((_coarser(levels[-1][0]), _coarser(levels[-1][1])))
    mg = _lib.Mg()
    mg.n_levels = len(levels)
    for l, (a, b) in enumerate(levels):
        mg.level[l].n = 2 * (a + 1) * (b + 1)
    return mg, [(a + 1) * (b + 1) for a, b in levels]


def _bytes(nodes, blocks):
    size = 1
    while 2 * size <= blocks and size * 64 < nodes[0]:
        size *= 2
    return sum(-(-n // size) * NODE_BYTES for n in nodes)


GRIDS = [(2945, 6), (5889, 12), (4793, 1), (4793, 2), (3827, 4), (11777, 24), (6000, 10), (3000, 6), (64, 64), (256, 256),
         (1500, 1500), (5, 3), (20000, 1)]


@pytest.mark.parametrize("gx,gy", GRIDS)
@pytest.mark.parametrize("blocks", [16, 8, 1])
def test_the_tail_fits_from_its_first_level_and_from_none_before(gx, gy, blocks):
    mg, nodes = _hierarchy(gx, gy)
    t = _lib.load().dfea_mg_tail_level(ctypes.byref(mg), blocks, LIMIT)
    assert 1 <= t < len(nodes)                                     # the coarsest level always fits
    fits = [nodes[l] <= TAIL_NODES and _bytes(nodes[l:], blocks) <= LIMIT for l in range(len(nodes))]
    assert fits[t] and not any(fits[1:t])


def test_square_grids_keep_their_first_small_level():
    for n in (64, 128, 256, 384, 1024):
        mg, nodes = _hierarchy(n, n)
        t = _lib.load().dfea_mg_tail_level(ctypes.byref(mg), 16, LIMIT)
        assert t == next(l for l in range(1, len(nodes)) if nodes[l] <= TAIL_NODES)


def test_no_room_and_bad_arguments():
    mg, nodes = _hierarchy(64, 64)
    lib = _lib.load()
    assert lib.dfea_mg_tail_level(ctypes.byref(mg), 16, 100) == mg.n_levels
    assert lib.dfea_mg_tail_level(None, 16, LIMIT) == -1
    assert lib.dfea_mg_tail_level(ctypes.byref(mg), 0, LIMIT) == -1
