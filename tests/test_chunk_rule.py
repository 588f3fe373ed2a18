"""The tile passes' chunk length (tile_layout.h, host build): states of one
tile, whose chunks no length changes, do not decide it."""

import ctypes

import pytest

from qmprs_gb300 import build as qb

BLOCKS, PER_STATE, TILE_QUBITS = 4 * 152, 256, 11


@pytest.fixture(scope="module")
def tiles():
    lib = ctypes.CDLL(str(qb.build_hostcheck()))
    return lambda ns: lib.hc_chunk_tiles((ctypes.c_int * len(ns))(*ns), len(ns))


@pytest.mark.parametrize("large", [[12], [18], [20], [20, 17, 13], [22] * 3])
@pytest.mark.parametrize("small", [1, 600, 5000])
def test_small_states_change_nothing(tiles, large, small):
    assert tiles([8] * small + large + [11]) == tiles(large)


@pytest.mark.parametrize("ns", [[2], [11] * 1000, [12], [16] * 40, [20], [20] * 6, [22], [14, 17, 20, 21]])
def test_fewest_tiles_of_one_wave(tiles, ns):
    def chunks(t):
        return [-(-2 ** (n - TILE_QUBITS) // t) for n in ns if n > TILE_QUBITS] or [0]

    def fits(t):
        return sum(chunks(t)) <= BLOCKS and max(chunks(t)) <= PER_STATE
    assert tiles(ns) == next((t for t in range(1, 17) if fits(t)), 32)
