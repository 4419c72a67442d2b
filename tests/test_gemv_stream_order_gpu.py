"""What orders the parts of a chain of products through one ring per CTA (gemv_stream.cuh)."""
import ctypes

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
        cur, ps, outs, first = 0, [], [], x                    # (the parameters hold addresses: the input has to outlive the launch)
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
        del first
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


@pytest.mark.parametrize("quant", [True, False])
def test_split_products_in_a_row(quant):
    """Four products whose left-over tiles are cut along k: each uses the partial sums and counters of the one before again, with nothing
    but the packets in between, and the third overwrites the first one's residual."""
    from tileinfer_b200.ops import functional as F
    F.L()
    shapes = [(5120, 8192, F.EPI_ROWPAR), (16384, 5120, F.EPI_SWIGLU), (5120, 8192, F.EPI_ROWPAR), (8192, 5120, F.EPI_STORE)]
    out = (ctypes.c_int * 7)()
    for n, k, _ in shapes:
        F.L().ti_gemv_stream_part(n // 8, k // (64 if quant else 32), 0, 0, F.NUM_SMS, out)
        assert out[6] > 1
    _agree(F, shapes, 1, quant, 12)


def test_a_long_kernel_before_the_launch():
    """The launch starts early and fills its ring beside the kernel before it.  That one may take longer than the 2 s after which this
    launch's waits give up (here: the packets of a second rank never come, which it notices after 2.3 s): the limit counts from its end."""
    from tileinfer_b200.ops import functional as F
    F.L()
    N, K, ms = 1184 * 8, 4096, 2300                            # eight row tiles and 16 stages per CTA: more than the ring holds
    g = torch.Generator(device="cuda").manual_seed(3)
    W, W0 = (F.LinearW(torch.randn(n, k, generator=g, device="cuda") * k ** -0.5, True) for n, k in ((N, K), (64, 64)))
    x, x0 = (torch.randn(1, k, generator=g, device="cuda").to(BF16) for k in (K, 64))
    want = F.gemv(W, x, epi=F.EPI_F32)

    class Comm:
        tp, rank, m_cap, timeout_ns = 2, 0, 1, ms * 10 ** 6
    boxes = [torch.zeros(2 * 2 * 32 * 16, dtype=torch.uint8, device="cuda") for _ in range(2)]       # this rank's packets, the other's
    ctrl = torch.tensor([1, 0, 0, 0], dtype=torch.int32, device="cuda")
    comm = Comm()
    comm.ll_ptrs, comm.step_ptr, comm.status_ptr = [b.data_ptr() for b in boxes], ctrl.data_ptr(), ctrl.data_ptr() + 4
    h, resid, out = torch.zeros(1, 64, dtype=BF16, device="cuda"), torch.zeros(1, 64, dtype=BF16, device="cuda"), torch.zeros(1, N, device="cuda")
    ws = [F.GemvWorkspace(), F.GemvWorkspace()]
    before = F.make_gemv_params(W0, x0, h, 1, epi=F.EPI_ROWPAR, resid=resid, ws=ws[0], comm=comm)
    after = F.make_gemv_params(W, x, out, 1, epi=F.EPI_F32, ws=ws[1])
    F.status_ptr()
    status = F._STATUS.clone()
    torch.cuda.synchronize()
    F.gemv_launch(before, F.W_INT8)
    F.gemv_launch(after, F.W_INT8)
    torch.cuda.synchronize()
    assert int(ctrl[1]) == 1                                   # the kernel before did wait that long
    assert torch.equal(F._STATUS, status) and torch.equal(out, want)


@pytest.mark.parametrize("M", [2, 8])
def test_several_rows_behind_a_grid_barrier(M):
    """bf16 rows that do not fit in 48 KB without a norm: the products of a chain are separated by grid barriers."""
    from tileinfer_b200.ops import functional as F
    F.L()
    H = 24576 // M
    g = torch.Generator(device="cuda").manual_seed(M)
    Ws = [F.LinearW(torch.randn(H, H, generator=g, device="cuda") * H ** -0.5, False) for _ in range(3)]
    ws = F.GemvWorkspace()
    for seed in range(10):
        x = torch.randn(M, H, generator=g, device="cuda").to(BF16)

        def run(chained):
            a, b = torch.zeros_like(x), torch.zeros_like(x)
            ps = [F.make_gemv_params(Ws[0], x, a, M, ws=ws), F.make_gemv_params(Ws[1], a, b, M, ws=ws),
                  F.make_gemv_params(Ws[2], b, a, M, epi=F.EPI_ROWPAR, resid=x, ws=ws)]
            if chained:
                F.gemv_chain_launch(ps, F.W_BF16)
            else:
                for p in ps:
                    F.gemv_launch(p, F.W_BF16)
            return a, b
        assert all(torch.equal(u, v) for u, v in zip(run(False), run(True))), seed
    assert int(ws.sched[:3].abs().sum()) == 0 and int(ws.counters.abs().sum()) == 0
