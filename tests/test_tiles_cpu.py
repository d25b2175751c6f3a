"""Index arithmetic of the flat tiles (tile_cells, set_flat and step_grid in
openlb_b200/csrc/aa_kernels.cuh), restated: the division by nz is exact wherever
it is used, and the blocks of a plane cover every cell once."""
from __future__ import annotations

import numpy as np
import pytest


def flat_constants(nz: int):
    s = 0
    while (1 << s) < nz:
        s += 1
    return ((1 << 32) * ((1 << s) - nz)) // nz + 1, s


def divide(n: np.ndarray, mul: int, shift: int) -> np.ndarray:
    """32-bit: (mulhi(n, mul) + n) >> shift."""
    n = n.astype(np.uint64)
    return (((n * np.uint64(mul) >> np.uint64(32)) + n) & np.uint64(0xFFFFFFFF)) >> np.uint64(shift)


@pytest.mark.parametrize("nz", [1, 2, 3, 5, 7, 31, 32, 33, 75, 150, 255, 256, 257, 1000, 4095, 65535, 65537,
                                (1 << 20) + 1, (1 << 30) - 1, 1 << 30, (1 << 31) - 1, 1 << 31])
def test_division_is_exact_below_2_31(nz):
    mul, shift = flat_constants(nz)
    assert 0 < mul < 1 << 32
    rng = np.random.default_rng(nz & 0xFFFF)
    top = (1 << 31) - 1
    q = rng.integers(0, top // nz + 1, 2000, dtype=np.int64)
    n = np.concatenate([q * nz, q * nz - 1, q * nz + nz - 1, rng.integers(0, top, 2000), [0, 1, top - 1, top]])
    n = n[(n >= 0) & (n <= top)]
    assert np.array_equal(divide(n, mul, shift).astype(np.int64), n // nz)


@pytest.mark.parametrize("threads", [64, 256])
@pytest.mark.parametrize("cells_per_thread", [1, 2])
@pytest.mark.parametrize("ny,nz", [(1, 1), (1, 63), (8, 8), (5, 13), (16, 16), (257, 1), (1, 257), (61, 75), (173, 150)])
def test_blocks_cover_a_plane_once(threads, cells_per_thread, ny, nz):
    mul, shift = flat_constants(nz)
    tile = threads * cells_per_thread
    blocks = (ny * nz + tile - 1) // tile
    seen = np.zeros((ny, nz), int)
    for b in range(blocks):
        for k in range(cells_per_thread):
            n = (b * cells_per_thread + k) * threads + np.arange(threads)
            n = n[n < ny * nz]          # other lanes are given y = ny and skipped
            y = divide(n, mul, shift).astype(int)
            z = n - y * nz
            assert np.all((y < ny) & (z >= 0) & (z < nz))
            np.add.at(seen, (y, z), 1)
    assert np.all(seen == 1)
