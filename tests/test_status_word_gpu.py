"""The error bits of every kernel of a hybrid step go to the executor's own status word, which travels to the host with the tokens."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quant", ["w8a16", "bf16"])
def test_every_launch_of_a_step_reports_to_the_executor(quant, monkeypatch):
    """Prompts long and short (tensor-core products and attention, both DeltaNet forms, mixed steps), one and several decodes, eager and
    captured: no launch falls back to the process-wide word, which nothing of this executor reads."""
    from tileinfer_b200.engine.llm import LLM
    from tileinfer_b200.engine.sampling_params import SamplingParams
    from tileinfer_b200.ops import functional as F
    F.L()

    def fallback():
        raise AssertionError("a launch without the executor's status word")
    monkeypatch.setattr(F, "status_ptr", fallback)
    seen = []
    make = F.make_gemv_params

    def record(*a, **kw):
        p = make(*a, **kw)
        seen.append(p.status)
        return p
    monkeypatch.setattr(F, "make_gemv_params", record)
    llm = LLM("preset:tiny-hybrid", quantization=quant, num_kvcache_blocks=128, max_num_seqs=4, max_model_len=512)
    sp = SamplingParams(temperature=0.0, max_tokens=6, ignore_eos=True)
    out = llm.generate_token_ids([list(range(1, 301)), [5, 9, 200], list(range(7, 47))], sp) + llm.generate_token_ids([[4, 8, 15]], sp)
    assert [len(o) for o in out] == [6] * 4
    model = llm.model_runner.model
    assert seen and set(seen) == {model.ctrl.data_ptr() + 4} == {model._status_ptr()}
    assert model.peer_status() == 0
