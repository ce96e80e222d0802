"""Order of the CTA-pair kernel's tiles in groups of many row tiles, on the host with the kernel's own functions."""
import ctypes as C

import pytest

from ccfuser_b200 import native as N


@pytest.mark.parametrize("swiglu", [0, 1])
@pytest.mark.parametrize("row_tiles", [1, 15, 16, 17, 18, 31, 33, 49, 56, 64, 241])
def test_row_blocks_cover_every_tile_once(row_tiles, swiglu):
    rows = [row_tiles * 256 - 3, 0, 300]
    cols = 9
    n = cols * (128 if swiglu else 256)
    arr = lambda v: (C.c_int * len(v))(*v)  # noqa: E731
    base, total = [], 0
    for r in rows:
        base.append(total)
        total += (r + 127) // 128 * 128
    want = (row_tiles + 2) * cols
    out = (C.c_int * (5 * want))()
    zero = arr([0, 0, 0])
    got = N.load().ccf_debug_pair_tile_order(arr(base), arr(rows), zero, zero, 3, n, 512, 0, swiglu, out, want)
    assert got == want
    tiles = [(out[5 * t], (out[5 * t + 1] - base[out[5 * t]]) // 256, out[5 * t + 2] // (n // cols)) for t in range(want)]
    assert set(tiles) == {(0, i, j) for i in range(row_tiles) for j in range(cols)} | {(2, i, j) for i in range(2) for j in range(cols)}
    # 16 consecutive tiles of the first group never touch more than two blocks of rows, each at most 16 high
    blocks = (row_tiles + 15) // 16
    per = (row_tiles + blocks - 1) // blocks
    assert per <= 16
    for t in range(row_tiles * cols - 1):
        a, b = tiles[t][1] // per, tiles[t + 1][1] // per
        assert b in (a, a + 1)
