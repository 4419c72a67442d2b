"""The persistent products (pairs of CTAs): edges of tiles in every direction, odd numbers of tiles, half
stages of k, every epilogue that stores through another path, against fp64 products of the same operands."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16

# (tokens, weight rows, k): the last token / weight tile full, one short, one over; fewer k stages than the ring holds;
# k with a half stage; more tiles than pairs of SMs, not a multiple of them; a last round cut along k in two to four slices,
# the last slice shorter; nothing but cut tiles; tiles of 32 and 64 tokens, full, nearly empty and one over; a short k with many
# tiles; the last batch of bf16 decodes with one tile per CTA and the first on pairs
SHAPES = [(256, 16384, 512), (129, 16480, 576), (257, 19200, 320), (4095, 1000, 1152), (2176, 2568, 64), (1060, 5120, 4160),
          (3000, 1160, 128), (8200, 520, 2048), (128, 5120, 17408), (70, 5128, 8256), (200, 4096, 6144), (1300, 5120, 6144),
          (1, 2048, 2048), (5, 5120, 6144), (17, 16480, 5120), (32, 5120, 17408), (33, 5120, 17408), (50, 1000, 4096), (64, 34816, 2048),
          (64, 30976, 320), (8, 34816, 1024), (9, 34816, 1024)]


def _operands(M, N, K, quantize):
    from tileinfer_b200.models.weights import untile_int8
    from tileinfer_b200.ops import functional as F
    F.L()
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N)
    W = F.LinearW(torch.randn(N, K, generator=g, device="cuda") * 0.05, quantize)
    x = torch.randn(M, K, generator=g, device="cuda").to(BF16)
    w = (untile_int8(W.tiles).double() * W.scale.double()[:, None])[:N] if quantize else W.dense().double()
    return F, W, x, w


@pytest.mark.parametrize("quantize", [True, False])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_pair_products(M, N, K, quantize):
    F, W, x, w = _operands(M, N, K, quantize)
    g = torch.Generator(device="cuda").manual_seed(5)
    resid = torch.randn(M, N, generator=g, device="cuda").to(BF16)
    limbs = F.quant_rows(x) if quantize else None
    run = lambda **kw: F.gemm_w8a16(W, limbs, **kw) if quantize else F.gemm_bf16(W, x, **kw)  # noqa: E731
    ref = x.double() @ w.t()
    # int8: a row's limbs are off by at most half a unit of 2^(e-14), e the exponent of its largest value.  bf16: K / 16
    # additions in fp32 that truncate, each off by at most 2^-23 of a partial sum, which is at most the sum of the magnitudes.
    # Stored as bf16 (relative 2^-9), or fp32.
    unit = 2.0 ** (torch.floor(torch.log2(x.double().abs().amax(1, keepdim=True))) - 14)
    noise = 6 * unit * w.norm(dim=1) / 12 ** 0.5 if quantize else (K / 16 + 2) * 2.0 ** -23 * (x.double().abs() @ w.abs().t())
    noise = noise + 1e-6 * ref.abs()

    def near(got, want, extra):
        assert got.shape == want.shape
        bad = (got.double() - want).abs() > extra + (2.0 ** -8) * want.abs() * (got.dtype == BF16)
        assert not bool(bad.any()), float((got.double() - want).abs().max())

    near(run(), ref, noise)
    near(run(epi=F.GEPI_ROWPAR, resid=resid), ref + resid.double(), noise)
    out = torch.empty(M, N, dtype=torch.float32, device="cuda")
    near(run(out=out, epi=F.GEPI_F32), ref, noise)
    if N % 16 == 0:
        gate, up = ref[:, 0::2], ref[:, 1::2]
        got = run(epi=F.GEPI_SWIGLU).double()
        want = torch.nn.functional.silu(gate) * up
        # gate and up are rounded to bf16 before the product: three roundings of 2^-9, the gate's times silu's slope (< 1.1)
        tol = (2.0 ** -7) * want.abs() + (noise[:, 0::2] + 2.0 ** -9 * gate.abs()) * 1.1 * up.abs() + \
            (noise[:, 1::2] + 2.0 ** -9 * up.abs()) * torch.nn.functional.silu(gate).abs() + 1e-6
        assert not bool(((got - want).abs() > tol).any())
    # same products twice: the same bits
    assert torch.equal(run(), run())


def test_pair_products_into_padded_rows():
    """Output rows longer than the product (a shared projection buffer): nothing past column N is written."""
    F, W, x, w = _operands(300, 16400, 640, True)
    buf = torch.full((300, 16480), 7.0, dtype=BF16, device="cuda")
    F.gemm_w8a16(W, F.quant_rows(x), out=buf)
    assert bool((buf[:, 16400:] == 7.0).all())
    ref = x.double() @ w.t()
    assert float((buf[:, :16400].double() - ref).norm() / ref.norm()) < 2.0 ** -8


# Stages of k from one to more than the ring has (6 to 10 of them; 121 weight tiles, so that some pairs run one tile and some two):
# the commits that a copying warp waits for before its CTA leaves are those of the last ring fill, whole or not, of one tile or two.
@pytest.mark.parametrize("quantize", [True, False])
@pytest.mark.parametrize("M", [20, 50, 100, 300])
@pytest.mark.parametrize("stages", [1, 2, 3, 5, 6, 7, 9, 10, 11, 13])
def test_last_ring_fill(stages, M, quantize):
    F, W, x, w = _operands(M, 30976, stages * (128 if quantize else 64), quantize)
    limbs = F.quant_rows(x) if quantize else None
    F.status_ptr()
    before = F._STATUS.clone()
    run = lambda: F.gemm_w8a16(W, limbs) if quantize else F.gemm_bf16(W, x)  # noqa: E731
    got, ref = [run() for _ in range(4)], x.double() @ w.t()
    assert float((got[0].double() - ref).norm() / ref.norm()) < 2.0 ** -8          # stored as bf16: 2^-9 at most
    assert all(torch.equal(got[0], o) for o in got[1:])
    assert torch.equal(F._STATUS, before)                      # no wait ran out
