"""Prefill attention on pairs of CTAs (neighbouring heads of one KV head): contexts whose last tile of 128 keys lies in the first
CTA's half, just past it, and around its end; query tiles of one to 128 rows; windows that start inside a tile; groups of heads
that cannot be paired beside groups that can.  Against softmax attention in fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("D,hq,hkv", [(256, 24, 4), (128, 16, 4), (256, 2, 1), (128, 2, 2), (128, 9, 3), (256, 12, 2)])
@pytest.mark.parametrize("window", [0, 70])
def test_pair_attention(D, hq, hkv, window):
    from tileinfer_b200.ops import functional as F
    F.L()
    g = torch.Generator(device="cuda").manual_seed(D + hq)
    # (cached tokens, new tokens)
    seqs = [(0, 1), (0, 63), (0, 64), (0, 65), (0, 128), (0, 129), (63, 1), (63, 2), (100, 29), (127, 130), (500, 17), (1000, 300)]
    need = [(c + n + 15) // 16 for c, n in seqs]
    T, nb = sum(n for _, n in seqs), sum(need) + 3
    perm = torch.randperm(nb).tolist()
    bt = torch.zeros(len(seqs), max(need), dtype=torch.int32)
    kc, vc = torch.zeros(nb, hkv, 16, D, dtype=BF16, device="cuda"), torch.zeros(nb, hkv, D, 16, dtype=BF16, device="cuda")
    kv, at, tiles, pos, t = [], 0, [], [], 0
    for s, (c, n) in enumerate(seqs):
        blocks = perm[at:at + need[s]]
        at += need[s]
        bt[s, :need[s]] = torch.tensor(blocks, dtype=torch.int32)
        k, v = (torch.randn(need[s] * 16, hkv, D, generator=g, device="cuda").to(BF16) for _ in range(2))
        kc[blocks], vc[blocks] = k.view(-1, 16, hkv, D).permute(0, 2, 1, 3), v.view(-1, 16, hkv, D).permute(0, 2, 3, 1)
        kv.append((k[:c + n].float(), v[:c + n].float()))
        pos += range(c, c + n)
        tiles += [(s, a, min(128, t + n - a)) for a in range(t, t + n, 128)]
        t += n
    q = (2.0 * torch.randn(T, hq, D, generator=g, device="cuda")).to(BF16)
    proj = torch.randn(T, hq * 2 * D, generator=g, device="cuda").to(BF16)
    out = torch.zeros(T, hq * D, dtype=BF16, device="cuda")
    tl = torch.tensor(tiles, dtype=torch.int32).t().contiguous().cuda()
    status = F._STATUS = torch.zeros(4, dtype=torch.int32, device="cuda")
    F.attn_prefill(q, kc, vc, nb, bt.cuda(), torch.tensor(pos, dtype=torch.int32, device="cuda"), tl, proj, out, hq=hq, hkv=hkv, D=D,
                   max_blocks=max(need), ld=proj.stride(0), window=window)
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    t = 0
    for (c, n), (k, v) in zip(seqs, kv):
        i, j = torch.arange(c, c + n, device="cuda")[:, None], torch.arange(c + n, device="cuda")[None]
        dead = (j > i) | ((j <= i - window) if window else False)
        sc = torch.einsum("tkgd,lkd->kgtl", q[t:t + n].float().view(n, hkv, hq // hkv, D), k) * D ** -0.5
        ref = torch.einsum("kgtl,lkd->tkgd", sc.masked_fill(dead, -float("inf")).softmax(-1), v).reshape(n, hq, D)
        ref = ref * torch.sigmoid(proj[t:t + n].float().view(n, hq, 2, D)[:, :, 1])
        # weights and outputs are rounded to bf16 (2^-9 each); a weighted sum keeps the relative size of its terms' errors
        assert float((out[t:t + n].float().view(n, hq, D) - ref).norm() / ref.norm()) < 2.0 ** -7
        t += n
