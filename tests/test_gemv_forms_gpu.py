"""Both forms of the GEMV where one of them is rarely taken: widths that are no multiple of 4, rows with infinities and NaN, a long row within
a chain, a workspace too small for cut tiles and packets (gemv_stream.cuh), and gemv_body with few rows (between ranks).  Against fp64."""
import ctypes

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


def _stages(F, ps, wt):
    out = (ctypes.c_int * 3)()
    F.L().ti_gemv_stream_plan(ctypes.byref(F.make_chain(ps)), wt, F.NUM_SMS, out)
    return out[0]


class _Ranks:
    """A communicator of two ranks.  Products that send nothing are served by gemv_body all the same."""
    tp, rank, m_cap, timeout_ns, ll_ptrs, step_ptr, status_ptr = 2, 0, 16, 10 ** 9, [0, 0], 0, 0


@pytest.mark.parametrize("quant", [True, False])
@pytest.mark.parametrize("N,K", [(2, 64), (1034, 1024), (1038, 960), (5118, 17408)])
def test_widths(N, K, quant):
    """Remainders of 2 and 6 in the last tile, one of them in a tile that is cut along k."""
    F = _F()
    W, w = _weight(F, N, K, quant, N)
    x = torch.randn(1, K, device="cuda").to(BF16)
    guard = torch.full((1, N + 8), 7.0, device="cuda")
    y = F.gemv(W, x, out=guard[:, :N], epi=F.EPI_F32)
    assert not bool(((y.double() - x.double() @ w.t()).abs() > _bound(x, w, quant)).any()) and bool((guard[:, N:] == 7.0).all())
    r = torch.randn(1, N, device="cuda").to(BF16)
    assert torch.equal(F.gemv(W, x, epi=F.EPI_ROWPAR, resid=r), (r.float() + y).to(BF16))
    assert torch.equal(F.gemv(W, x), y.to(BF16))


@pytest.mark.parametrize("N", [1032, 1034])
def test_residual_of_an_earlier_product(N):
    """The residual comes from a product whose row is nobody's input: as packets, or, of a width that has none, behind the barrier."""
    F = _F()
    Wa, Wb = (_weight(F, N, 1024, True, s)[0] for s in (1, 2))
    ws = F.GemvWorkspace()
    for seed in range(10):
        g = torch.Generator(device="cuda").manual_seed(seed)
        xa, xb = (torch.randn(1, 1024, generator=g, device="cuda").to(BF16) for _ in range(2))
        h0 = torch.randn(1, N, generator=g, device="cuda").to(BF16)

        def run(chained):
            a, b = torch.zeros_like(h0), torch.zeros_like(h0)
            ps = [F.make_gemv_params(Wa, xa, a, 1, epi=F.EPI_ROWPAR, resid=h0, ws=ws), F.make_gemv_params(Wb, xb, b, 1, epi=F.EPI_ROWPAR, resid=a, ws=ws)]
            if chained:
                F.gemv_chain_launch(ps, F.W_INT8)
            else:
                for p in ps:
                    F.gemv_launch(p, F.W_INT8)
            return a, b
        assert all(torch.equal(u, v) for u, v in zip(run(False), run(True))), seed


@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("quant", [True, False])
@pytest.mark.parametrize("bad", [float("inf"), -float("inf"), float("nan")])
def test_rows_that_are_not_finite(bad, quant, norm):
    """What gemv_body makes of such a row: the same values, infinities and NaN in the same places."""
    F = _F()
    N, K = 1192, 1024
    W, _ = _weight(F, N, K, quant, 3)
    x = torch.randn(1, K, device="cuda").to(BF16)
    x[0, 77] = bad
    nw = (torch.randn(K, device="cuda") * 0.1).to(BF16) if norm else None
    kw = dict(xmode=F.XNORM if norm else F.XGLOBAL, epi=F.EPI_F32, norm_w=nw)
    a, b = F.gemv(W, x, **kw), F.gemv(W, x, comm=_Ranks, **kw)
    torch.testing.assert_close(a, b, rtol=2.0 ** -20, atol=1e-6, equal_nan=True)


@pytest.mark.parametrize("quant", [True, False])
def test_long_row_in_a_chain(quant):
    """A row longer than registers hold: the whole chain runs behind grid barriers."""
    F = _F()
    H, I = 2560, 21504
    Ws = [_weight(F, n, k, quant, i) for i, (n, k) in enumerate(((H, 1024), (2 * I, H), (H, I), (H, H)))]
    nw = (torch.randn(H, device="cuda") * 0.1).to(BF16)
    ws = F.GemvWorkspace()
    for _ in range(3):
        x, h0 = torch.randn(1, 1024, device="cuda").to(BF16), torch.randn(1, H, device="cuda").to(BF16)
        h1, h2, act, proj = (torch.zeros(1, n, dtype=BF16, device="cuda") for n in (H, H, I, H))
        ps = [F.make_gemv_params(Ws[0][0], x, h1, 1, epi=F.EPI_ROWPAR, resid=h0, ws=ws),
              F.make_gemv_params(Ws[1][0], h1, act, 1, xmode=F.XNORM, epi=F.EPI_SWIGLU, norm_w=nw, ws=ws),
              F.make_gemv_params(Ws[2][0], act, h2, 1, epi=F.EPI_ROWPAR, resid=h1, ws=ws),
              F.make_gemv_params(Ws[3][0], h2, proj, 1, epi=F.EPI_STORE, ws=ws)]
        assert _stages(F, ps, Ws[0][0].wt) >= 4
        F.gemv_chain_launch(ps, Ws[0][0].wt)
        for got, base, xx, (_, w) in ((h1, h0, x, Ws[0]), (h2, h1, act, Ws[2]), (proj, None, h2, Ws[3])):
            ref = xx.double() @ w.t() + (0 if base is None else base.double())
            assert not bool(((got.double() - ref).abs() > _bound(xx, w, quant) + 2.0 ** -8 * ref.abs()).any())
        want = F.gemv(Ws[1][0], h1, xmode=F.XNORM, epi=F.EPI_SWIGLU, norm_w=nw, ws=ws)
        # the norm's sum of squares may be added in another order: an ulp of a normed value, a unit of an int8 row's limbs
        assert float((act.double() - want.double()).norm() / want.double().norm()) < 2.0 ** -8
    assert int(ws.sched[:3].abs().sum()) == 0 and int(ws.counters.abs().sum()) == 0


@pytest.mark.parametrize("quant", [True, False])
def test_small_workspace(quant):
    """No room for cut tiles and packets: whole tiles, and grid barriers between the products."""
    F = _F()
    H, I = 5120, 8192
    Ws = [_weight(F, n, k, quant, i)[0] for i, (n, k) in enumerate(((H, 1024), (2 * I, H), (H, I)))]
    ws = F.GemvWorkspace(max_units=64, max_tiles=64)
    nw = (torch.randn(H, device="cuda") * 0.1).to(BF16)
    for seed in range(4):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x, h0 = torch.randn(1, 1024, generator=g, device="cuda").to(BF16), torch.randn(1, H, generator=g, device="cuda").to(BF16)

        def run(chained):
            h1, h2, act = (torch.zeros(1, n, dtype=BF16, device="cuda") for n in (H, H, I))
            ps = [F.make_gemv_params(Ws[0], x, h1, 1, epi=F.EPI_ROWPAR, resid=h0, ws=ws),
                  F.make_gemv_params(Ws[1], h1, act, 1, xmode=F.XNORM, epi=F.EPI_SWIGLU, norm_w=nw, ws=ws),
                  F.make_gemv_params(Ws[2], act, h2, 1, epi=F.EPI_ROWPAR, resid=h1, ws=ws)]
            assert not ps[0].ws and not ps[0].counters
            if chained:
                F.gemv_chain_launch(ps, Ws[0].wt)
            else:
                for p in ps:
                    F.gemv_launch(p, Ws[0].wt)
            return h1, act, h2
        assert all(torch.equal(u, v) for u, v in zip(run(False), run(True))), seed
    assert int(ws.sched[:3].abs().sum()) == 0 and int(ws.ws.abs().sum()) == 0


@pytest.mark.parametrize("quant", [True, False])
@pytest.mark.parametrize("M,N,K", [(1, 1192, 2048), (1, 5120, 6144), (3, 1192, 2112), (3, 5120, 6144), (8, 5112, 2176)])
def test_few_rows_between_ranks(M, N, K, quant):
    F = _F()
    W, w = _weight(F, N, K, quant, N + M)
    x = torch.randn(M, K + 8, device="cuda").to(BF16)[:, :K]
    p = F.make_gemv_params(W, x, torch.empty(M, N, device="cuda"), M, epi=F.EPI_F32, comm=_Ranks)
    assert _stages(F, [p], W.wt) == 0
    y = F.gemv(W, x, epi=F.EPI_F32, comm=_Ranks)
    assert not bool(((y.double() - x.double() @ w.t()).abs() > _bound(x, w, quant)).any())
    x = x.contiguous()
    nw = (torch.randn(K, device="cuda") * 0.1).to(BF16)
    y = F.gemv(W, x, xmode=F.XNORM, epi=F.EPI_F32, norm_w=nw, comm=_Ranks)
    xd = x.double()
    xn = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * (1 + nw.double())
    # the normed row is rounded to bf16: 2^-9 of each value, signs at random (six standard deviations of the sum)
    tol = 6 * 2.0 ** -9 * (xn.square() @ w.square().t()).sqrt() + (_bound(xn, w, True) if quant else 0) + 1e-5
    assert not bool(((y.double() - xn @ w.t()).abs() > tol).any())


@pytest.mark.parametrize("M,N,K", [(2, 1192, 12288), (4, 1192, 6176), (8, 1192, 3072), (8, 2376, 3104), (7, 5118, 5152), (6, 16480, 5120), (1, 1192, 24576)])
def test_bf16_rows_read_once(M, N, K):
    """Several bf16 rows through one ring: those that gemv_body does not stage.  A tile more than there are CTAs, an odd number, left-over
    tiles cut along k with a remainder of columns."""
    F = _F()
    W, w = _weight(F, N, K, False, N + K)
    x = torch.randn(M, K + 8, device="cuda").to(BF16)[:, :K]
    ws = F.GemvWorkspace()
    out = torch.empty(M, N, device="cuda")
    assert _stages(F, [F.make_gemv_params(W, x, out, M, epi=F.EPI_F32, ws=ws)], F.W_BF16) >= 4
    y = F.gemv(W, x, out=out, epi=F.EPI_F32, ws=ws)
    assert not bool(((y.double() - x.double() @ w.t()).abs() > _bound(x, w, False)).any())
    for _ in range(3):
        assert torch.equal(y, F.gemv(W, x, epi=F.EPI_F32, ws=ws))
    r = torch.randn(M, N, device="cuda").to(BF16)
    assert torch.equal(F.gemv(W, x, epi=F.EPI_ROWPAR, resid=r, ws=ws), (r.float() + y).to(BF16))
    val, idx = torch.zeros(M, F.NUM_SMS, device="cuda"), torch.zeros(M, F.NUM_SMS, dtype=torch.int32, device="cuda")
    F.gemv_launch(F.make_gemv_params(W, x, val, M, epi=F.EPI_ARGMAX, out_idx=idx, ws=ws), F.W_BF16)
    best = val.argmax(1, keepdim=True)
    assert torch.equal(val.amax(1), y.amax(1)) and torch.equal(idx.gather(1, best)[:, 0].long(), y.argmax(1))
    assert int(ws.counters.abs().sum()) == 0 and int(ws.sched[:3].abs().sum()) == 0
