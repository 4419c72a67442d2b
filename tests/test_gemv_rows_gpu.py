"""bf16 GEMV: rows staged in shared memory with and without a norm, at the size where rows without one stop being staged (48 KB),
with one row (its own form) and up to 16, and a k that one row's form does not take.  Against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("M,K", [(1, 32), (1, 2048), (1, 20480), (1, 20512), (1, 24544), (1, 24576), (2, 12256), (2, 12288), (3, 8192), (8, 3040),
                                 (9, 2720), (16, 1504), (16, 1536)])
def test_rows(M, K):
    from tileinfer_b200.ops import functional as F
    F.L()
    g = torch.Generator(device="cuda").manual_seed(M * 31 + K)
    N = 1032
    W = F.LinearW(torch.randn(N, K, generator=g, device="cuda") * K ** -0.5, False)
    w = W.dense().double()
    x = torch.randn(M, K + 8, generator=g, device="cuda").to(BF16)[:, :K]           # rows with a pitch of their own
    y = F.gemv(W, x, epi=F.EPI_F32)
    # fp32 sums of K exact products over warps' slices: K / 16 additions, each off by at most 2^-23 of the magnitudes' sum
    bound = (K / 16 + 16) * 2.0 ** -23 * (x.double().abs() @ w.abs().t()) + 1e-6
    assert not bool(((y.double() - x.double() @ w.t()).abs() > bound).any())
    if F.plan_gemv(F.W_BF16, F.XNORM, M, W.n_tiles, W.KB) is None:
        return
    nw = (torch.randn(K, generator=g, device="cuda") * 0.1).to(BF16)
    y = F.gemv(W, x, xmode=F.XNORM, epi=F.EPI_F32, norm_w=nw)
    xd = x.double()
    xn = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * (1 + nw.double())
    # the normed row is rounded to bf16: 2^-9 of each value, signs at random (six standard deviations of the sum)
    tol = 6 * 2.0 ** -9 * (xn.square() @ w.square().t()).sqrt() + 1e-5
    assert not bool(((y.double() - xn @ w.t()).abs() > tol).any())
