"""What the CTA pairs of the kernel with the weights on the M side work on (csrc/swap_shape.h), the pieces of its last round among it, on
the host with the kernel's own functions."""
import ctypes as C
import random

import pytest

from ccfuser_b200 import native as N


def _items(rows, n, wide, pairs):
    arr, cap = (C.c_int * len(rows))(*rows), 40000
    out = (C.c_int * (12 * cap))()
    cnt = N.load().ccf_debug_swap_items(arr, len(rows), n, 512, 1, int(wide), pairs, out, cap)
    assert 0 <= cnt <= cap
    return [tuple(out[12 * i:12 * i + 12]) for i in range(cnt)]


def _cases():
    rng = random.Random(11)
    for _ in range(600):
        groups = rng.choice([1, 2, 3, 4, 8, 16, 64])
        top = rng.choice([17, 64, 127, 128, 129, 160, 256, 257, 300, 320, 321, 700])
        skew = rng.choice([0, 0, 1])        # a few popular experts and many rows of one digit beside them
        rows = [rng.randint(0, top) if not skew or rng.random() < 0.3 else rng.randint(0, 40) for _ in range(groups)]
        yield rows, 32 * rng.randint(1, 40), rng.choice([1, 2, 5, 66, 74])
    yield [300, 20, 17, 9], 1024, 74
    yield [256, 40, 17], 1024, 74
    yield [320, 64, 193, 129, 257], 512, 74


@pytest.mark.parametrize("wide", [False, True])
def test_every_row_and_feature_is_worked_on_once(wide):
    cut = 0
    for rows, n, pairs in _cases():
        seen, zeros, last = {}, {}, {}
        for pair, item, whole, g, row, tokens, zero, n0, parts, np_, half, have in _items(rows, n, wide, pairs):
            assert 0 < tokens and row + tokens <= rows[g] and n0 % 256 == 0 and n0 < n
            assert parts in (1, 2) and np_ % 16 == 0 and tokens <= parts * np_ and half <= have      # a stage holds it
            seen.setdefault((g, n0), []).append((row, row + tokens))
            if zero:
                assert row + tokens == rows[g]           # they lie behind the group's last row
                zeros[(g, n0)] = zeros.get((g, n0), 0) + zero
            if item >= whole:
                last.setdefault(pair, []).append(item)
                cut += tokens < rows[g]
        assert set(seen) == {(g, n0) for g, r in enumerate(rows) if r for n0 in range(0, n, 256)}
        for (g, _), runs in seen.items():
            runs.sort()
            assert runs[0][0] == 0 and runs[-1][1] == rows[g] and all(a[1] == b[0] for a, b in zip(runs, runs[1:]))
        for (g, n0) in seen:
            assert zeros.get((g, n0), 0) == -rows[g] % 64
        assert all(len(v) == 1 for v in last.values())
    assert cut > 500


@pytest.mark.parametrize("wide", [False, True])
def test_pieces_have_64_rows(wide):
    """A piece streams the tile's weights again: no tile comes in pieces of fewer rows, whatever the largest tile of the launch has."""
    for rows, n, pairs in _cases():
        tile_cap = 128 if wide else 256 if max(rows) <= 256 else 320
        for pair, item, whole, g, row, tokens, zero, n0, parts, np_, half, have in _items(rows, n, wide, pairs):
            mt = (rows[g] + tile_cap - 1) // tile_cap
            per = ((rows[g] + mt - 1) // mt + 15) // 16 * 16
            tile = min(per, rows[g] - row // per * per)
            assert tokens == tile or (item >= whole and tokens >= 64)
