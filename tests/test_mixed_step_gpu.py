"""Running sequences (one token each) beside prompts in one step: the decode kernels advance the former, the chunk kernels the
latter, and each leaves the other's states, convolution inputs and output rows alone.  Oracle: the CPU executor."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# first: tokens of every sequence's first step; second: the step under test (1: a running sequence).  40 running sequences of 8
# heads are more than the 296 (head, sequence) pairs up to which the decode step takes one block per pair.
@pytest.mark.parametrize("first,second", [([20, 33, 0], [1, 1, 50]), ([0, 17, 40, 5], [64, 1, 65, 1]), ([3, 0], [1, 129]),
                                          ([2] * 40 + [0], [1] * 40 + [35])])
def test_one_token_sequences_beside_prompts(first, second):
    from tileinfer_b200.models.config import TINY_HYBRID
    from tileinfer_b200.models.hybrid_b200 import B200HybridModel
    from tileinfer_b200.models.reference_cpu import Batch, TorchHybridModel
    from tileinfer_b200.models.weights import RandomWeights
    S = len(first)
    src = RandomWeights(TINY_HYBRID, 0)
    g = torch.Generator().manual_seed(S)
    per = 16
    gpu, cpu = B200HybridModel(TINY_HYBRID, src, quant="w8a16"), TorchHybridModel(TINY_HYBRID, src, quant="w8a16")
    slots = torch.randperm(S + 2, generator=g)[:S].tolist()
    for m in (gpu, cpu):
        m.alloc_cache(S * per, 16, S + 2)
    ids = [torch.randint(0, 1000, (a + b,), generator=g) for a, b in zip(first, second)]

    def batch(lens, starts):
        live = [s for s in range(S) if lens[s]]
        cu = [0]
        for s in live:
            cu.append(cu[-1] + lens[s])
        pos = torch.cat([torch.arange(starts[s], starts[s] + lens[s]) for s in live])
        at = torch.cat([torch.arange(starts[s], starts[s] + lens[s]) + s * per * 16 for s in live])
        return Batch(torch.cat([ids[s][starts[s]:starts[s] + lens[s]] for s in live]), pos, cu, [starts[s] + lens[s] for s in live],
                     [list(range(s * per, (s + 1) * per)) for s in live], at, [slots[s] for s in live])

    for lens, starts in ((first, [0] * S), (second, first)):
        b = batch(lens, starts)
        got, want = gpu.logits(gpu.forward(b)).float().cpu(), cpu.logits(cpu.forward(b))
    assert float((got - want).abs().max()) < 0.05          # the tolerance of the engine's own comparison with this oracle
    for s in slots:
        a, w = gpu.rec[:, s].float().cpu(), cpu.rec_state[:, s]
        assert float((a - w).norm() / w.norm()) < 2e-2
    assert gpu.peer_status() == 0
