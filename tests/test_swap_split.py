"""Whole tiles of the kernel with the weights on the M side (csrc/swap_shape.h), on the host with the kernel's own functions: one pair sums
all k-blocks of a tile, and a stage of the pipeline holds it. What becomes of the last round's tiles is test_swap_items.py's."""
import ctypes as C
import random

import pytest

from ccfuser_b200 import native as N


def _segments(rows, n, k, kseg, wide, pairs):
    lib = N.load()
    arr = (C.c_int * len(rows))(*rows)
    cap = 20000
    out = (C.c_int * (9 * cap))()
    cnt = lib.ccf_debug_swap_segments(arr, len(rows), n, k, kseg, int(wide), pairs, out, cap)
    assert 0 <= cnt <= cap
    return [tuple(out[9 * i:9 * i + 9]) for i in range(cnt)]


@pytest.mark.parametrize("wide", [False, True])
def test_every_k_block_of_every_tile_is_summed_once(wide):
    rng = random.Random(5 + wide)
    for _ in range(400):
        groups = rng.choice([1, 2, 3, 8, 16, 64])
        top = rng.choice([1, 2, 17, 128, 129, 160, 161, 256, 257, 320, 321, 700])
        rows = [rng.randint(0, top) for _ in range(groups)]
        n, k = 32 * rng.randint(1, 40), 8 * rng.randint(1, 300)
        kseg, pairs = rng.choice([1, 2]), rng.choice([1, 2, 66, 74])
        kb = kseg * ((k + 63) // 64)
        cap = 128 if wide else 256 if max(rows) <= 256 else 320
        tiles = sum((r + cap - 1) // cap for r in rows) * ((n + 255) // 256)
        seen = {}
        for pair, tile, k0, k1, first, sharers, half, stages, total in _segments(rows, n, k, kseg, wide, pairs):
            assert 0 <= tile < tiles and 0 <= k0 < k1 <= kb and 0 <= pair < pairs
            assert half % 16 == 0 and half <= 160 and 2 <= stages <= 12
            seen.setdefault(tile, []).append((k0, k1, pair, first, sharers))
            assert total == tiles and pair == tile % pairs      # the pairs take the tiles in turns
        assert len(seen) == tiles
        for runs in seen.values():
            assert len(runs) == 1                               # no tile is shared
            k0, k1, pair, first, sharers = runs[0]
            assert (k0, k1) == (0, kb) and first == pair and sharers == 1
