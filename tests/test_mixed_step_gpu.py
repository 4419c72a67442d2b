"""Running sequences (one token each) beside prompts in one step: the decode kernels advance the former, the chunk kernels the
latter, and each leaves the other's states, convolution inputs and output rows alone.  Oracle: the CPU executor."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _heads(cfg, conv):
    """[.., channels, 3] of the CPU executor -> [.., v-heads, 3, q | k | v of the head], as the GPU's state cache keeps them."""
    hk, hv, dk, dv = cfg.gdn_num_k_heads, cfg.gdn_num_v_heads, cfg.gdn_head_k_dim, cfg.gdn_head_v_dim
    q, k, v = conv.transpose(-1, -2).split((hk * dk, hk * dk, hv * dv), -1)
    rep = lambda x: x.unflatten(-1, (hk, dk)).repeat_interleave(hv // hk, dim=-2)  # noqa: E731
    return torch.cat([rep(q), rep(k), v.unflatten(-1, (hv, dv))], -1).transpose(-2, -3)


def _near(got, want, tol=2e-2):
    assert got.shape == want.shape
    assert float((got.float().cpu() - want).norm() / want.norm()) < tol


# first: tokens of every sequence's first step; second: the step under test (1: a running sequence); a step of one token for all
# follows, which starts from the states and convolution inputs that the second left.  40 running sequences of 8 heads are more
# than the 296 (head, sequence) pairs up to which the decode step takes one block per pair.  snap: {sequence: tokens of the second
# step after which its state is captured}; a one-token sequence with a capture stays a chunk.
@pytest.mark.parametrize("first,second,snap", [([20, 33, 0], [1, 1, 50], {}), ([0, 17, 40, 5], [64, 1, 65, 1], {}), ([3, 0], [1, 129], {}),
                                               ([2] * 40 + [0], [1] * 40 + [35], {}), ([15, 31, 9, 16], [1, 1, 1, 80], {0: [1], 3: [16, 64]}),
                                               ([7, 14, 30], [40, 2, 1], {0: [9], 1: [1, 2]})])
@pytest.mark.parametrize("state", ["fp32", "bf16"])
def test_one_token_sequences_beside_prompts(first, second, snap, state):
    from tileinfer_b200.models.config import TINY_HYBRID
    from tileinfer_b200.models.hybrid_b200 import B200HybridModel
    from tileinfer_b200.models.reference_cpu import Batch, TorchHybridModel
    from tileinfer_b200.models.weights import RandomWeights
    S = len(first)
    src = RandomWeights(TINY_HYBRID, 0)
    g = torch.Generator().manual_seed(S)
    per = 16
    gpu, cpu = B200HybridModel(TINY_HYBRID, src, quant="w8a16"), TorchHybridModel(TINY_HYBRID, src, quant="w8a16")
    gpu.state_bf16 = state == "bf16"                        # rounds a state by 2^-9 a step, well inside the tolerance
    perm = torch.randperm(S + 2, generator=g).tolist()
    slots, unused = perm[:S], perm[S:]
    for m in (gpu, cpu):
        m.alloc_cache(S * per, 16, S + 2)
    for u in unused:
        gpu.rec[:, u].normal_()
        gpu.conv[:, u].normal_()
    kept = gpu.rec[:, unused].clone(), gpu.conv[:, unused].clone()
    ids = [torch.randint(0, 1000, (a + b + 1,), generator=g) for a, b in zip(first, second)]

    def batch(lens, starts, snap):
        live = [s for s in range(S) if lens[s]]
        cu = [0]
        for s in live:
            cu.append(cu[-1] + lens[s])
        pos = torch.cat([torch.arange(starts[s], starts[s] + lens[s]) for s in live])
        at = torch.cat([torch.arange(starts[s], starts[s] + lens[s]) + s * per * 16 for s in live])
        return Batch(torch.cat([ids[s][starts[s]:starts[s] + lens[s]] for s in live]), pos, cu, [starts[s] + lens[s] for s in live],
                     [list(range(s * per, (s + 1) * per)) for s in live], at, [slots[s] for s in live],
                     [[starts[s] + n for n in snap.get(s, [])] for s in live])

    for lens, starts, pts in ((first, [0] * S, {}), (second, first, snap), ([1] * S, [a + b for a, b in zip(first, second)], {})):
        b = batch(lens, starts, pts)
        got, want = gpu.logits(gpu.forward(b)).float().cpu(), cpu.logits(cpu.forward(b))
        assert float((got - want).abs().max()) < 0.05          # the tolerance of the engine's own comparison with this oracle
        for s in range(S):
            if starts[s] + lens[s]:
                _near(gpu.rec[:, slots[s]], cpu.rec_state[:, slots[s]])
                _near(gpu.conv[:, slots[s]], _heads(TINY_HYBRID, cpu.conv_state[:, slots[s]]))
        assert torch.equal(gpu.rec[:, unused], kept[0]) and torch.equal(gpu.conv[:, unused], kept[1])
        a, w = gpu.take_snapshots(), cpu.take_snapshots()
        assert sorted(a) == sorted(w) and len(a) == sum(map(len, pts.values()))
        for key in a:
            _near(a[key][0], w[key][0])
            _near(a[key][1], _heads(TINY_HYBRID, w[key][1]))
    assert gpu.peer_status() == 0


def test_captured_steps_without_a_wait_between_them():
    """Two captured steps in a row, the second prepared while the first may still be copying its inputs: each gives what it
    gives alone."""
    from tileinfer_b200.models.config import TINY_HYBRID
    from tileinfer_b200.models.hybrid_b200 import B200HybridModel
    from tileinfer_b200.models.reference_cpu import Batch
    from tileinfer_b200.models.weights import RandomWeights
    m = B200HybridModel(TINY_HYBRID, RandomWeights(TINY_HYBRID, 0), quant="w8a16")
    S, per = 8, 8
    m.alloc_cache(S * per, 16, S + 1)
    m.capture_decode_graphs(S, S, 128, S)
    g = torch.Generator().manual_seed(1)
    ids = torch.randint(0, 1000, (40, S), generator=g)
    busy = torch.zeros(64 << 20, device="cuda")

    def run(wait):
        for s in range(S):
            m.zero_state(s)
        out = []
        for t in range(len(ids)):
            order = torch.randperm(S, generator=torch.Generator().manual_seed(t)).tolist()      # other rows, slots and tables each time
            if not wait:
                busy.add_(1)                                   # the device is behind: copies of earlier steps are still queued
            out.append(m.step_logits(Batch(ids[t][order], torch.full((S,), t), list(range(S + 1)), [t + 1] * S,
                                           [list(range(s * per, (s + 1) * per)) for s in order],
                                           torch.tensor([s * per * 16 + t for s in order]), order)))
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return torch.stack(out)

    assert torch.equal(run(True), run(False))
    assert m.peer_status() == 0
