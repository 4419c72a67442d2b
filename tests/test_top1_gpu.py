"""The arg-max form of the top-k kernels (k = 1): ties, rows of -inf and of the lowest float, NaN, ragged vocabularies, the merge of
candidates in any order, and the static entry point; the oracle is the radix selection's order (float bits mapped to ascending integers, smallest id first)."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _key(v):
    u = v.view(torch.int32).long() & 0xFFFFFFFF
    return torch.where(u >= 1 << 31, 0xFFFFFFFF - u, u + (1 << 31)).clamp_min(1)


def _expect(row):
    k = _key(row)
    return int((k == k.max()).nonzero()[0])


@pytest.mark.parametrize("V", [1, 255, 256, 257, 4097, 15616, 131071, 248320])
def test_top1(V):
    from tileinfer_b200.ops import functional as F
    F.L()
    g = torch.Generator().manual_seed(V)
    rows = [torch.randn(V, generator=g), torch.full((V,), float("-inf")), torch.full((V,), torch.finfo(torch.float32).min),
            torch.randint(-3, 3, (V,), generator=g).float(), torch.randn(V, generator=g), torch.zeros(V), -torch.zeros(V)]
    rows[4][V // 2:] = float("nan")
    rows[5][V // 3:] = -0.0
    x = torch.stack(rows)
    d = x.cuda()
    M, chunks_of = len(rows), -(-V // 128)
    cs = max(256, -(-chunks_of // 256) * 256)
    chunks = -(-V // cs)
    ws_v, ws_i = torch.empty(M, chunks, device="cuda"), torch.empty(M, chunks, dtype=torch.int32, device="cuda")
    out_v, out_i = torch.empty(M, 1, device="cuda"), torch.empty(M, 1, dtype=torch.int32, device="cuda")
    p = F.TopkParams()
    p.logits, p.ws_val, p.ws_idx, p.out_val, p.out_idx = (t.data_ptr() for t in (d, ws_v, ws_i, out_v, out_i))
    p.M, p.V, p.ld, p.k, p.chunks, p.chunk_size, p.vocab_start, p.tp = M, V, V, 1, chunks, cs, 1000, 1
    F.topk(p)
    torch.cuda.synchronize()
    want = [_expect(r) for r in rows]
    assert (out_i[:, 0].cpu() - 1000).tolist() == want
    assert torch.equal(out_v[:, 0].cpu().view(torch.int32), x[torch.arange(M), want].view(torch.int32))
    # the merge alone: candidates of which some chunks have none
    ws_i[0, 1:] = -1
    F.topk_merge(p)
    torch.cuda.synchronize()
    assert int(out_i[0]) == 1000 + _expect(rows[0][:cs])
    ws_i[0] = -1
    F.topk_merge(p)
    torch.cuda.synchronize()
    assert int(out_i[0]) == -1 and float(out_v[0]) == float("-inf")
    if V <= 524288:
        from tileinfer_b200.ops import build
        fn = ctypes.CDLL(build.LIB).ti_topk_static
        fn.restype, fn.argtypes = ctypes.c_int, [ctypes.c_void_p] + [ctypes.c_int] * 5 + [ctypes.c_void_p] * 3
        assert fn(d.data_ptr(), M, V, V, 1, 0, out_v.data_ptr(), out_i.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        assert out_i[:, 0].cpu().tolist() == want


@pytest.mark.parametrize("chunks", [2, 148, 600])
def test_merge_of_candidates_in_any_order(chunks):
    """Equal candidates whose ids do not ascend with their places (the arg-max epilogue of the vocabulary product deals columns
    to CTAs by ticket): the smallest id wins, with its value, wherever it stands.  The last row has places without a candidate."""
    from tileinfer_b200.ops import functional as F
    F.L()
    g = torch.Generator().manual_seed(chunks)
    ids = torch.stack([torch.arange(chunks - 1, -1, -1), torch.randperm(chunks, generator=g), torch.randperm(chunks, generator=g),
                       torch.arange(chunks).roll(1), torch.randperm(chunks, generator=g)]) * 3
    val = torch.stack([torch.full((chunks,), 2.5), torch.randint(0, 2, (chunks,), generator=g).float(), torch.randn(chunks, generator=g),
                       torch.full((chunks,), float("-inf")), torch.full((chunks,), torch.finfo(torch.float32).min)])
    ids[4, torch.randperm(chunks, generator=g)[:chunks // 2]] = -1
    want = [min((int(i) for i, v, k in zip(r, x, _key(x)) if i >= 0 and k == _key(x)[r >= 0].max()), default=-1) for r, x in zip(ids, val)]
    M = len(val)
    ws_v, ws_i = val.cuda(), ids.int().cuda()
    out_v, out_i = torch.empty(M, 1, device="cuda"), torch.empty(M, 1, dtype=torch.int32, device="cuda")
    p = F.TopkParams()
    p.ws_val, p.ws_idx, p.out_val, p.out_idx = (t.data_ptr() for t in (ws_v, ws_i, out_v, out_i))
    p.M, p.V, p.ld, p.k, p.chunks, p.chunk_size, p.vocab_start, p.tp = M, 3 * chunks, 0, 1, chunks, 0, 1000, 1
    F.topk_merge(p)
    torch.cuda.synchronize()
    assert (out_i[:, 0].cpu() - 1000).tolist() == want
    assert torch.equal(out_v[:, 0].cpu(), torch.stack([x[r >= 0].max() for r, x in zip(ids, val)]))
