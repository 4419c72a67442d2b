"""The scheduling counters of the GEMV between launches: zero.  Left to run, the counter of finished CTAs wraps around after
2^31 / 148 launches, out of step with their ends."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 9])
def test_counters_are_zero_between_launches(M):
    from tileinfer_b200.ops import functional as F
    F.L()
    W = F.LinearW(torch.randn(64, 512, device="cuda"), True)
    ws = F.GemvWorkspace()
    F.gemv(W, torch.randn(M, 512, device="cuda").to(torch.bfloat16), ws=ws)
    assert int(ws.sched[:3].abs().sum()) == 0
