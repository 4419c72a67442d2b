"""What orders the parts of a chain of products through one ring per CTA (gemv_stream.cuh)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _chain(F, shapes, M, quant, seed=1):
    """[(N, K, epilogue)] -> a function that runs the chain, or its products one by one, from fresh inputs.  The residual of a product
    is the output of the one two before it, as in a layer; there are two hidden buffers, so that the third product's output is the
    first one's residual buffer."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    Ws = [F.LinearW(torch.randn(n, k, generator=g, device="cuda") * k ** -0.5, quant) for n, k, _ in shapes]
    nws = [(torch.randn(k, generator=g, device="cuda") * 0.1).to(BF16) for _, k, _ in shapes]
    ws = F.GemvWorkspace()

    def run(seed, chained):
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn(M, shapes[0][1], generator=g, device="cuda").to(BF16)
        hidden = [torch.randn(M, shapes[0][0], generator=g, device="cuda").to(BF16) for _ in range(2)]
        cur, ps, outs = 0, [], []
        for (n, k, epi), W, nw in zip(shapes, Ws, nws):
            if epi == F.EPI_ROWPAR:
                out = hidden[1 - cur]
                ps.append(F.make_gemv_params(W, x, out, M, epi=epi, resid=hidden[cur], ws=ws))
                cur = 1 - cur
            else:
                out = torch.zeros(M, n // 2 if epi == F.EPI_SWIGLU else n, dtype=BF16, device="cuda")
                ps.append(F.make_gemv_params(W, x, out, M, xmode=F.XNORM, epi=epi, norm_w=nw, ws=ws))
            outs.append(out)
            x = out
        if chained:
            F.gemv_chain_launch(ps, Ws[0].wt)
        else:
            for p in ps:
                F.gemv_launch(p, Ws[0].wt)
        return outs
    return run, ws


def _agree(F, shapes, M, quant, times):
    F.status_ptr()
    before = F._STATUS.clone()
    run, ws = _chain(F, shapes, M, quant)
    for seed in range(times):
        a, b = run(seed, False), run(seed, True)
        assert all(torch.equal(u, v) for u, v in zip(a, b)), seed
    assert torch.equal(F._STATUS, before)                      # no wait ran out
    assert int(ws.sched[:3].abs().sum()) == 0 and int(ws.counters.abs().sum()) == 0


@pytest.mark.parametrize("quant", [True, False])
def test_ctas_without_work(quant):
    """Products with fewer row tiles than there are CTAs: some have nothing to do but to poll for rows, and the launch's tag must not
    move on before they have read it."""
    from tileinfer_b200.ops import functional as F
    F.L()
    _agree(F, [(64, 128, F.EPI_ROWPAR), (256, 64, F.EPI_SWIGLU), (64, 128, F.EPI_ROWPAR), (136, 64, F.EPI_STORE)], 1, quant, 40)
