"""The split of a product's row tiles, and of the k of left-over ones, among CTAs: every k tile of every row tile exactly once."""
import ctypes

import pytest

from tileinfer_b200.ops import lib


@pytest.mark.parametrize("n_tiles,KB,skew", [(640, 272, 60), (639, 272, 0), (640, 96, 12), (4352, 80, 147), (2060, 80, 100), (1, 8, 3),
                                             (149, 600, 5), (447, 321, 1), (148, 544, 7), (146, 600, 90), (74, 1200, 0)])
def test_parts_cover_a_product_once(n_tiles, KB, skew):
    seen, out, busy, ncta = {}, (ctypes.c_int * 7)(), [], 148
    for cta in range(ncta):
        assert lib.lib().ti_gemv_stream_part(n_tiles, KB, skew, cta, ncta, out) == 0
        first, count, tile, kt0, kt1, two, slices = out
        for t in range(first, first + count):
            seen.setdefault(t, []).append((0, KB))
        if tile >= 0:
            for t in range(tile, tile + two):
                seen.setdefault(t, []).append((kt0, kt1))
        busy.append(count * KB + (two * (kt1 - kt0) if tile >= 0 else 0))
    assert sorted(seen) == list(range(n_tiles))
    for r in seen.values():
        r.sort()
        assert r[0][0] == 0 and r[-1][1] == KB and all(u[1] == v[0] for u, v in zip(r, r[1:]))
    if slices > 1:                               # a left-over tile costs a slice of two, not a whole one
        assert max(busy) - n_tiles // ncta * KB <= 2 * (KB // slices + 1)
