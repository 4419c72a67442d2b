"""Token tiles of the products that pairs of CTAs take: 64 up to one round of 74 tiles, not where the larger tiles are better cut along k."""
import pytest


@pytest.mark.parametrize("bf16,M,N,K,tokens", [
    (0, 32, 5120, 6144, 32), (0, 33, 5120, 6144, 64), (0, 64, 34816, 5120, 64),                            # batched decode
    (0, 65, 9472, 2048, 64), (0, 65, 9480, 2048, 128), (0, 192, 5120, 6144, 64), (0, 193, 5120, 6144, 128),    # one round of 64
    (0, 65, 18944, 2048, 128), (0, 128, 5120, 17408, 128), (0, 129, 5120, 17408, 64), (0, 4096, 5120, 6144, 128),
    (1, 65, 5120, 17408, 128), (1, 128, 5120, 6144, 64), (1, 129, 5120, 6144, 64),
    (1, 129, 5120, 17408, 256), (1, 192, 5120, 17408, 256), (1, 129, 5120, 14208, 256), (1, 129, 4096, 14336, 256),    # 256, cut along k
    (1, 129, 5120, 14144, 64), (1, 129, 5120, 6272, 64), (1, 256, 2048, 8192, 64), (1, 300, 2048, 6144, 64),            # 64 although 256 would be
    (1, 129, 34816, 5120, 256), (1, 4096, 34816, 5120, 256), (1, 4096, 5120, 6144, 256)])
def test_tokens(bf16, M, N, K, tokens):
    from tileinfer_b200.ops import functional as F
    stages = -(-K * (2 if bf16 else 1) // 128)
    assert F.L("base").ti_gemm_pair_tokens(bf16, M, -(-N // 8), stages, 1) == tokens


def test_without_a_workspace():
    """Nothing is cut without one: the tiles of 64 come back."""
    from tileinfer_b200.ops import functional as F
    assert F.L("base").ti_gemm_pair_tokens(1, 129, 640, 272, 0) == 64 and F.L("base").ti_gemm_pair_tokens(0, 128, 640, 136, 0) == 64
