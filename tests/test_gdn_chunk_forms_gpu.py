"""Forms of the chunk-parallel DeltaNet prefill that its dispatch chooses between: projection rows that can and cannot be
read in vectors, one v-head per CTA (few chunks) and all v-heads of a k-head per CTA (many), chunks of every fill."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _run(F, chunked, proj, conv_w, neg, dt_bias, norm_w, state, cs, slots, cu_l, hk, hv, d):
    S, T = len(cu_l) - 1, cu_l[-1]
    state, cs = state.clone(), cs.clone()
    out = torch.zeros(T, hv * d, dtype=BF16, device="cuda")
    cu = torch.tensor(cu_l, dtype=torch.int32, device="cuda")
    p = F.GdnChunkParams() if chunked else F.GdnParams()
    for name, t in (("proj", proj), ("conv_w", conv_w), ("neg_a_exp", neg), ("dt_bias", dt_bias), ("norm_w", norm_w),
                    ("state", state), ("conv_state", cs), ("slots", slots), ("cu", cu), ("out", out)):
        setattr(p, name, t.data_ptr())
    p.ld, p.hk, p.hv, p.eps = proj.stride(0), hk, hv, 1e-6
    if chunked:
        ck, seq_ck = (t.cuda() for t in F.gdn_chunk_table(cu_l))
        p.ck_seq, p.ck_tok0, p.ck_ntok, p.ck_snap = (ck[i].data_ptr() for i in range(4))
        p.seq_ck, p.nc = seq_ck.data_ptr(), ck.shape[1]
        ws = F.GdnChunkWorkspace("cuda").get(ck.shape[1] * hv, d, d)
        p.wf, p.qf, p.mf, p.kf, p.u, p.gamma = (b.data_ptr() for b in ws)
        F.gdn_chunked(p, S, T, d, d, False)
    else:
        F.gdn_step(p, S, d, d, False)
    torch.cuda.synchronize()
    return out, state, cs


# pad: extra columns of a projection row.  heads: 2 * hk * d + 2 * hv * d + 2 * hv columns, so pad 0 gives rows of a multiple of 4
# (d = 128) or 2 (d = 64) values, pad 1 rows of an odd number of them.  `long`: at least 296 (chunk, k-head) pairs.
@pytest.mark.parametrize("d,hk,hv,pad,lens", [
    (128, 4, 12, 0, [1, 64, 65, 127, 19]),
    (128, 4, 12, 1, [1, 64, 65, 127, 19]),
    (128, 4, 12, 0, [4000, 1, 700, 63]),
    (128, 4, 12, 3, [4000, 1, 700, 63]),
    (128, 8, 8, 0, [2400]),
    (64, 4, 8, 0, [5, 4800]),
    (64, 4, 8, 1, [5, 130]),
    (128, 1, 10, 0, [300, 2]),               # more v-heads per k-head than one CTA takes
])
def test_chunked_forms_match_the_serial_kernel(d, hk, hv, pad, lens):
    from tileinfer_b200.ops import functional as F
    F.L()
    g = torch.Generator(device="cuda").manual_seed(7)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    cu_l = [0]
    for n in lens:
        cu_l.append(cu_l[-1] + n)
    S, T, rep = len(lens), cu_l[-1], hv // hk
    proj = rnd(T, 2 * hk * d + 2 * hv * d + 2 * hv + pad).to(BF16)
    conv_w = rnd(2 * hk * d + hv * d, 4) * 0.5
    neg, dt_bias, norm_w = -torch.exp(rnd(hv) * 0.5), rnd(hv) * 0.5, 1 + 0.1 * rnd(d)
    state = rnd(S + 1, hv, d, d) * 0.1
    hist = rnd(S + 1, 3, 2 * hk * d + hv * d).to(BF16)
    q, k, v = (x.reshape(S + 1, 3, -1, d) for x in hist.split((hk * d, hk * d, hv * d), -1))
    cs = torch.cat([q.repeat_interleave(rep, 2), k.repeat_interleave(rep, 2), v], -1).transpose(1, 2).contiguous()
    slots = torch.randperm(S + 1)[:S].int().cuda()
    args = (proj, conv_w, neg, dt_bias, norm_w, state, cs, slots, cu_l, hk, hv, d)
    out, st, c = _run(F, True, *args)
    out1, st1, c1 = _run(F, False, *args)
    assert torch.equal(c, c1)
    # every operand of the chunk products is rounded to bf16 once (2^-9 relative): 1 % of the whole in the 2-norm
    for got, want in ((out, out1), (st, st1)):
        assert float((got.float() - want.float()).norm() / want.float().norm()) < 1e-2
        assert torch.isfinite(got.float()).all()
