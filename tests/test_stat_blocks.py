"""Room for the statistics' partial sums, on the CPU: one block writes one partial, and
the room a solver is created with covers every launch that a step of it can be -- on
the whole grid or as a z-slab (two planes fewer), with a mask or without.  Fewer planes
can give more blocks, since a block then takes a shorter run of them."""
import ctypes as C
import random

import pytest

from myfluidsimulation_b200 import _lib


class Cfg(C.Structure):
    _fields_ = [("blocks", C.c_int), ("threads", C.c_int)]


EVEN, ODD = Cfg(148 * 8, 256), Cfg(148 * 12, 256)


def funcs():
    L = _lib.lib()
    room, grid = L._ZN3lbm14aa_stat_blocksEiiiiNS_9LaunchCfgES0_, L._ZN3lbm11aa_odd_gridEiilbiNS_9LaunchCfgE
    room.restype = grid.restype = C.c_int64
    room.argtypes = [C.c_int] * 4 + [Cfg, Cfg]
    grid.argtypes = [C.c_int, C.c_int, C.c_int64, C.c_bool, C.c_int, Cfg]
    return room, grid


def sizes():
    r = random.Random(5)
    yield from [(64, 256, 167), (64, 512, 57), (128, 256, 56), (256, 128, 56), (64, 128, 333), (64, 192, 222), (1, 1, 3), (1, 1, 1),
                (600000, 3, 3)]
    for _ in range(4000):
        yield tuple(int(2 ** r.uniform(0, 9.5)) for _ in range(3))


@pytest.mark.parametrize("storage", [0, 1, 2, 3])
def test_partials_cover_every_launch(storage):
    room, grid = funcs()
    for nx, ny, nz in sizes():
        have = room(nx, ny, nz, storage, EVEN, ODD)
        assert have >= EVEN.blocks
        for planes in {nz, max(nz - 2, 1)}:
            for mask in (False, True):
                assert grid(nx, ny, planes, mask, storage, ODD) <= have, (nx, ny, nz, planes, mask)
