"""Rows that a step returns or samples (`Batch.out_rows`, `sample_rows`): any integers that index a list, negative ones included;
others are an error on the host, before anything is launched.  The runtime's own code runs here on host tensors; the GPU test
compares whole steps."""
import numpy as np
import pytest
import torch

from tileinfer_b200.models.reference_cpu import Batch
from tileinfer_b200.models.runtime_b200 import DeviceRuntime


class _Stop(Exception):
    pass


class _Host(DeviceRuntime):
    """A step whose layers give back the numbers of the rows."""
    dev, hkv, host_steps, graphs, v_local, tp, peer = torch.device("cpu"), 1, 0, {}, 3, 1, None

    def _alloc_ctx(self, *sizes):
        return self._alloc_inputs(*sizes)

    def _run_layers(self, x):
        return torch.arange(x.T, dtype=torch.float32)[:, None].expand(x.T, 3)

    def logits(self, hidden):
        self.asked = hidden[:, 0].tolist()
        return hidden


def _batch(lens, out_rows=None):
    cu = np.cumsum([0] + lens).tolist()
    return Batch(torch.zeros(cu[-1], dtype=torch.long), torch.cat([torch.arange(n) for n in lens]), cu, list(lens),
                 [[s] for s in range(len(lens))], torch.arange(cu[-1]), list(range(len(lens))), out_rows=out_rows)


@pytest.mark.parametrize("kind", [list, tuple, np.array, torch.tensor])
@pytest.mark.parametrize("rows", [[0], [-1], [5, -6, 2, 2], [0, 1, 2, 3, 4, 5], [-6, -5, -4, -3, -2, -1], list(range(5, -1, -1))])
def test_rows_of_a_step(rows, kind):
    want = [r % 6 for r in rows]
    assert _Host().forward(_batch([3, 1, 2], kind(rows)))[:, 0].tolist() == want
    assert _Host().step_logits(_batch([3, 1, 2], kind(rows)))[:, 0].tolist() == want


def test_rows_by_default_and_none():
    assert _Host().forward(_batch([3, 1, 2]))[:, 0].tolist() == [2, 3, 5]
    assert _Host().forward(_batch([0, 0, 2, 1]))[:, 0].tolist() == [2, 2, 1, 2]
    assert _Host().step_logits(_batch([3, 1, 2], [])).shape == (0, 3)


@pytest.mark.parametrize("rows", [[6], [-7], [0, 100]])
def test_rows_out_of_range(rows):
    for call in (_Host().forward, _Host().step_logits):
        with pytest.raises(IndexError):
            call(_batch([3, 1, 2], rows))


@pytest.mark.parametrize("rows,want", [([-1, 0], [5, 2]), ([0, 1, 2], [2, 3, 5]), ([1], [3]), ([-3, -2, -1], [2, 3, 5])])
def test_rows_to_sample(rows, want, monkeypatch):
    from tileinfer_b200.models import runtime_b200

    def stop(*_):
        raise _Stop
    h = _Host()
    monkeypatch.setattr(h, "_topk_rows", stop)
    with pytest.raises(_Stop):
        h.forward_and_sample(_batch([3, 1, 2]), rows, 1)
    assert h.asked == want
    monkeypatch.setattr(runtime_b200.DeviceRuntime, "_topk_rows", stop)
    with pytest.raises(IndexError):
        h.forward_and_sample(_batch([3, 1, 2]), [3], 1)


@pytest.mark.gpu
def test_rows_on_the_device():
    """A prompt step and a captured decode step (three sequences in a bucket of four): rows from the end give what the same rows
    from the front give."""
    from tileinfer_b200.models.config import TINY_HYBRID
    from tileinfer_b200.models.hybrid_b200 import B200HybridModel
    from tileinfer_b200.models.weights import RandomWeights
    m = B200HybridModel(TINY_HYBRID, RandomWeights(TINY_HYBRID, 0), quant="w8a16")
    m.alloc_cache(8, 16, 5)
    m.capture_decode_graphs(4, 4, 64, 4)

    def step(lens, rows, start=0):
        cu = np.cumsum([0] + lens).tolist()
        pos = torch.cat([torch.arange(start, start + n) for n in lens])
        at = torch.cat([torch.arange(start, start + n) + s * 32 for s, n in enumerate(lens)])
        for s in range(len(lens)):
            m.zero_state(s)
        ids = torch.arange(cu[-1]) % 1000
        return m.step_logits(Batch(ids, pos, cu, [start + n for n in lens], [[2 * s, 2 * s + 1] for s in range(len(lens))], at,
                                   list(range(len(lens))), out_rows=rows))

    for lens, start in (([20, 1, 7], 0), ([1, 1, 1], 5)):
        T = sum(lens)
        want = step(lens, [T - 1, 0, T - 2], start)
        assert torch.equal(step(lens, [-1, -T, -2], start), want)
        assert torch.equal(step(lens, list(range(T)), start)[[T - 1, 0, T - 2]], want)
    assert m.peer_status() == 0
