"""Products of a few hundred tokens with few weight tiles: tiles of 64 tokens where those of 128 would leave pairs of CTAs without work,
at the sizes where one or the other is taken (74 tiles of 64 are one round), with remainders of tokens and rows.  Against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("M,N,K", [(65, 5120, 2048), (128, 9472, 2048), (128, 9728, 2048), (129, 2056, 2048), (192, 6152, 4096), (300, 3784, 2048),
                                   (577, 2048, 2048), (130, 5120, 17408)])
@pytest.mark.parametrize("quant", [True, False])
def test_products(M, N, K, quant):
    from tileinfer_b200.ops import functional as F
    F.L()
    g = torch.Generator(device="cuda").manual_seed(M + N)
    W = F.LinearW(torch.randn(N, K, generator=g, device="cuda") * K ** -0.5, quant)
    x = torch.randn(M, K, generator=g, device="cuda").to(BF16)
    r = torch.randn(M, N, generator=g, device="cuda").to(BF16)
    if quant:
        from tileinfer_b200.models.weights import untile_int8
        w = (untile_int8(W.tiles).double() * W.scale.double()[:, None])[:N]
        y = F.gemm_w8a16(W, F.quant_rows(x), epi=F.GEPI_ROWPAR, resid=r)
    else:
        w = W.dense().double()
        y = F.gemm_bf16(W, x, epi=F.GEPI_ROWPAR, resid=r)
    ref = r.double() + x.double() @ w.t()
    a = x.double().abs()
    # activations to half a unit (2^-15 of the row's largest), fp32 sums, the result rounded to bf16
    tol = (a.amax(1, keepdim=True) * 2.0 ** -15 * w.abs().sum(1) if quant else 0) + K * 2.0 ** -24 * (a @ w.abs().t()) + 2.0 ** -8 * ref.abs() + 1e-5
    assert not bool(((y.double() - ref).abs() > tol).any())
