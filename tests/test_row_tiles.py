"""Row bounds of the tiles of CTA pairs (csrc/row_tiles.cuh), compiled for the CPU: up to the largest sizes that the library takes."""

import ctypes
import shutil
import subprocess

import pytest

from triturus_b200 import build

SIZES = [1, 31, 32, 33, 192, 193, 385, 1000, 3_640_000, 3_700_001, 4_000_000, 2**24 + 5, 2**30 - 7, 2**30]


@pytest.fixture(scope="module")
def row_tile(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    tmp = tmp_path_factory.mktemp("row_tiles")
    src = tmp / "row_tiles.cpp"
    src.write_text(
        f'#include "{build.CSRC / "row_tiles.cuh"}"\n'
        'extern "C" void row_tile(int units, int tiles, int t, int* out) {\n'
        "  const tb200::RowTile r = tb200::row_tile(units, tiles, t);\n  out[0] = r.first, out[1] = r.units;\n}\n"
    )
    subprocess.run([cxx, "-O1", "-std=c++17", "-shared", "-fPIC", "-o", str(tmp / "row_tiles.so"), str(src)], check=True)
    lib = ctypes.CDLL(str(tmp / "row_tiles.so"))

    def call(units, tiles, t):
        out = (ctypes.c_int * 2)()
        lib.row_tile(units, tiles, t, out)
        return out[0], out[1]

    return call


@pytest.mark.parametrize("rows", SIZES)
def test_tiles_cover_the_rows(row_tile, rows):
    """Contiguous, all units once, one to six units each and no two sizes further apart than one: at both ends, and around
    every tile where a 32-bit product of tile and unit counts would wrap."""
    units = (rows + 31) // 32
    tiles = (units + 5) // 6
    largest = -(-units // tiles)
    around = {0, tiles - 1, *(k * 2**31 // units + d for k in range(1, min(8, units * tiles // 2**31 + 1)) for d in (-1, 0, 1))}
    for t in sorted(x for x in {y + d for y in around for d in (-1, 0, 1)} if 0 <= x < tiles):
        first, n = row_tile(units, tiles, t)
        assert max(1, largest - 1) <= n <= largest <= 6
        assert 0 <= first and t * (units // tiles) <= first <= t * largest
        assert first + n == (units if t == tiles - 1 else row_tile(units, tiles, t + 1)[0])
    assert row_tile(units, tiles, 0)[0] == 0
