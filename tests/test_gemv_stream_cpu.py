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


def _form(wt, M, products):
    """Ring stages, rows the kernel is built for and bytes of staged rows of a launch of (N, K, xmode) products; zeros: the other form."""
    from tileinfer_b200.ops import functional as F
    c, out = lib.ChainParams(), (ctypes.c_int * 3)()
    c.n_ops = len(products)
    for p, (N, K, xmode) in zip(c.op, products):
        p.M, p.N, p.n_tiles, p.K, p.KB, p.xmode, p.tp = M, N, -(-N // 8), K, K // (64 if wt == F.W_INT8 else 32), xmode, 1
    assert lib.lib().ti_gemv_stream_plan(ctypes.byref(c), wt, 148, out) == 0
    return tuple(out)


@pytest.mark.parametrize("bf16,M,N,K,norm,rows", [
    (0, 1, 8, 64, 1, 1), (0, 1, 5120, 20480, 0, 1), (1, 1, 248320, 5120, 1, 1),                          # one row that registers hold
    (0, 1, 2352, 20544, 0, 0), (0, 1, 2361, 20544, 0, 8), (1, 1, 2368, 20512, 1, 8), (1, 1, 2352, 20512, 1, 0), (1, 1, 1192, 24576, 0, 8),
    (0, 1, 2368, 65536, 0, 8), (0, 1, 2368, 65600, 0, 0),                                                                # a longer one
    (0, 2, 1192, 64, 0, 0), (0, 8, 16480, 5120, 1, 0), (1, 2, 32768, 2048, 1, 0), (1, 2, 32768, 2048, 0, 0),                # several
    (1, 2, 5120, 12256, 0, 0), (1, 2, 5120, 12288, 0, 8), (1, 2, 5120, 12288, 1, 0), (1, 8, 1192, 3072, 0, 8), (1, 8, 1184, 3072, 0, 0),
    (1, 9, 16480, 5120, 0, 0)])
def test_form_of_a_product(bf16, M, N, K, norm, rows):
    assert _form(bf16, M, [(N, K, norm)])[1] == rows


def test_form_of_a_chain():
    """Every product has to be of the form, and the longest rows decide what a launch's kernel is built for."""
    layer = [(5120, 6144, 0), (34816, 5120, 1), (5120, 17408, 0), (16480, 5120, 1)]
    assert _form(0, 1, layer)[1] == 1 and _form(0, 2, layer)[1] == 0
    stages, rows, x_bytes = _form(0, 1, [(5120, 6144, 0), (43008, 5120, 1), (5120, 21504, 0), (16480, 5120, 1)])
    assert rows == 8 and x_bytes >= 2 * 21504 and stages >= 4
    assert _form(1, 4, [(2048, 8192, 0), (8192, 6176, 0)])[1] == 8 and _form(1, 4, [(2048, 8192, 0), (8192, 2048, 1)])[1] == 0
