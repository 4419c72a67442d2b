"""Products of one row on one GPU, whose weights a CTA streams through one ring: sizes around a CTA's share of row tiles (none, a
lone tile, left-over tiles cut along k, an odd number of those), k tiles around the 16 of a stage, every epilogue, and chains whose rows
go from product to product as packets, or behind a grid barrier; the same sizes with 2 and 8 rows, which take the other form except for
bf16 rows too long to stage.  Against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _F():
    from tileinfer_b200.ops import functional as F
    F.L()
    return F


def _weight(F, N, K, quant, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    W = F.LinearW(torch.randn(N, K, generator=g, device="cuda") * K ** -0.5, quant)
    if not quant:
        return W, W.dense().double()
    from tileinfer_b200.models.weights import untile_int8
    return W, (untile_int8(W.tiles).double() * W.scale.double()[:, None])[:N]


def _bound(x, w, quant):
    """int8: a row is stored to half a unit, at most max |x| 2^-15; bf16: fp32 sums of exact products."""
    a = x.double().abs()
    if quant:
        return a.amax(1, keepdim=True) * 2.0 ** -15 * w.abs().sum(1) + 2.0 ** -21 * (a @ w.abs().t()) + 1e-6
    return (x.shape[1] / 16 + 16) * 2.0 ** -23 * (a @ w.abs().t()) + 1e-6


# (N, K): 8 rows; one tile for some CTAs; 148 tiles and one more; an odd last tile; left-over pairs cut along k (of an even and an odd
# number of tiles); k tiles 1, 15, 16, 17, 33 and a k that one row's staging does not hold in registers
SHAPES = [(8, 64), (64, 1024), (1184, 960), (1192, 1088), (2376, 2112), (5120, 17408), (5112, 17408), (3576, 20544), (35008, 512)]


@pytest.mark.parametrize("quant", [True, False])
@pytest.mark.parametrize("N,K", SHAPES)
@pytest.mark.parametrize("M", [1, 2, 8])
def test_shapes(M, N, K, quant):
    F = _F()
    if F.plan_gemv(F.W_INT8 if quant else F.W_BF16, F.XNORM, M, N // 8, K // (64 if quant else 32)) is None:
        pytest.skip("rows do not fit")
    W, w = _weight(F, N, K, quant, N + K)
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K + 8, generator=g, device="cuda").to(BF16)[:, :K]
    ws = F.GemvWorkspace()
    y = F.gemv(W, x, epi=F.EPI_F32, ws=ws)
    assert not bool(((y.double() - x.double() @ w.t()).abs() > _bound(x, w, quant)).any())
    for _ in range(3):
        assert torch.equal(y, F.gemv(W, x, epi=F.EPI_F32, ws=ws))
    assert int(ws.counters.abs().sum()) == 0 and int(ws.sched[1]) == 0 and int(ws.sched[2]) == 0
    r = torch.randn(M, N, generator=g, device="cuda").to(BF16)
    out = F.gemv(W, x, epi=F.EPI_ROWPAR, resid=r, ws=ws)
    assert torch.equal(out, (r.float() + y).to(BF16))


@pytest.mark.parametrize("quant", [True, False])
@pytest.mark.parametrize("M,alias", [(1, "none"), (1, "resid_shifted"), (1, "skip"), (2, "none")])
def test_chain(M, alias, quant):
    """Four dependent products in one launch, many times, against the same ones launched one by one: bit by bit."""
    F = _F()
    H, I, KO, NI = 5120, 2048, 1536, 1048
    wt = F.W_INT8 if quant else F.W_BF16
    Wo, Wgu, Wd = (_weight(F, n, k, quant, s)[0] for n, k, s in ((H, KO, 1), (2 * I, H, 2), (H, I, 3)))
    Wi = _weight(F, NI, H, quant, 4)[0]
    g = torch.Generator(device="cuda").manual_seed(5)
    nw = (torch.randn(H, generator=g, device="cuda") * 0.1).to(BF16)
    ws = F.GemvWorkspace()

    def run(seed, chained):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x, h0 = torch.randn(M, KO, generator=g, device="cuda").to(BF16), torch.randn(M, H, generator=g, device="cuda").to(BF16)
        h1 = torch.zeros(M + 1, H, dtype=BF16, device="cuda")
        h2, act, proj = torch.zeros(M, H, dtype=BF16, device="cuda"), torch.zeros(M, I, dtype=BF16, device="cuda"), torch.zeros(M, NI, dtype=BF16, device="cuda")
        resid = h1.view(-1)[8:8 + M * H].view(M, H) if alias == "resid_shifted" else h1[:M]      # (the shifted one reads behind a barrier)
        last = h1[:M] if alias == "skip" else h2
        ps = [F.make_gemv_params(Wo, x, h1[:M], M, xmode=F.XGLOBAL, epi=F.EPI_ROWPAR, resid=h0, ws=ws),
              F.make_gemv_params(Wgu, h1[:M], act, M, xmode=F.XNORM, epi=F.EPI_SWIGLU, norm_w=nw, ws=ws),
              F.make_gemv_params(Wd, act, h2, M, xmode=F.XGLOBAL, epi=F.EPI_ROWPAR, resid=resid, ws=ws),
              F.make_gemv_params(Wi, last, proj, M, xmode=F.XNORM, epi=F.EPI_STORE, norm_w=nw, ws=ws)]
        if chained:
            F.gemv_chain_launch(ps, wt)
        else:
            for p in ps:
                F.gemv_launch(p, wt)
        return h1, act, h2, proj

    for seed in range(6):
        a, b = run(seed, False), run(seed, True)
        assert all(torch.equal(u, v) for u, v in zip(a, b)), seed
    assert int(ws.sched[:3].abs().sum()) == 0


@pytest.mark.parametrize("M", [1, 3])
def test_argmax(M):
    F = _F()
    N, K = 9472, 512                                     # 1184 tiles: 8 per CTA
    W, _ = _weight(F, N, K, False, 9)
    x = torch.randn(M, K, device="cuda").to(BF16)
    logits = F.gemv(W, x, epi=F.EPI_F32)
    val, idx = torch.zeros(M, F.NUM_SMS, device="cuda"), torch.zeros(M, F.NUM_SMS, dtype=torch.int32, device="cuda")
    p = F.make_gemv_params(W, x, val, M, epi=F.EPI_ARGMAX, out_idx=idx)
    F.gemv_launch(p, F.W_BF16)
    best = val.argmax(1)
    assert torch.equal(val.amax(1), logits.amax(1))
    assert torch.equal(idx.gather(1, best[:, None])[:, 0].long(), logits.argmax(1))


@pytest.mark.parametrize("N", [64, 4744])
def test_sums_of_a_long_row_fit_in_32_bits(N):
    """K beyond 65536: low limbs of 255 beside weights of 127 add up to more than 2^31.  Every weight is 1, one activation (64) sets the
    row's unit to 2^-8, all others are 255 units."""
    F = _F()
    K = 72000
    W = F.LinearW(torch.ones(N, K, device="cuda"), True)
    x = torch.full((1, K), 255 / 256, dtype=BF16, device="cuda")
    x[0, 7] = 64.0
    y = F.gemv(W, x, epi=F.EPI_F32).double()
    want = x.double().sum() * 127 * W.scale[:N].double()
    # exact integer sums, their two parts added in fp32 and scaled: a few roundings of 2^-24
    assert not bool(((y[0] - want).abs() > 2.0 ** -21 * want).any())
