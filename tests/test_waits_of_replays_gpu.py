"""A bounded wait that runs out inside a replayed pass is an error of the step whose tokens it spoils (the word that a kernel would
set is set by the test)."""

import pytest
import torch

import tiny

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


class AtCall:
    """Observer: before the given forward pass's tokens are read, a wait has run out."""

    def __init__(self, call):
        self.call, self.calls, self.passes = call, 0, []

    def after_forward(self, rids, tokens, logits):
        from mini_infer_b200.ops import functional as F
        self.calls += 1
        self.passes.append(list(tokens))
        if self.calls == self.call:
            F.wait_status(torch.device(DEV)).fill_(37)

    def settled(self, note, kept):
        pass


@pytest.mark.parametrize("dtype,hidden", [("float32", 512), ("float32", 64)])
@pytest.mark.parametrize("call", [3, 6])
def test_decode_replays(tmp_path, dtype, hidden, call):
    from mini_infer_b200.engine.llm import LLM
    from mini_infer_b200.ops import functional as F
    from mini_infer_b200.ops.library import KernelError
    from mini_infer_b200.sampling import SamplingParams
    cfg = dict(tiny.CONFIG_A, hidden_size=hidden)
    tiny.make_folder(str(tmp_path), cfg, seed=5)
    llm = LLM(str(tmp_path), dtype=dtype, max_seq_len=64, max_running=2)
    prompts, params = [[1, 2, 3, 4, 5], [6, 7, 8]], SamplingParams(greedy=True, max_new_tokens=8)
    first = [o.token_ids for o in llm.generate(prompts, params)]
    assert llm.runner.graph_replays > 0
    observer = AtCall(call)
    llm.executor.observer = observer
    if hidden < F.library().mi_f32_tc_min_inner():     # nothing in the passes waits: nothing is looked at
        llm.generate(prompts, params)
        F.wait_status(torch.device(DEV)).zero_()
        return
    with pytest.raises(KernelError, match="code 37"):
        llm.generate(prompts, params)
    assert observer.passes[call - 1] == [1, 1]
    llm.executor.observer = None
    again = LLM(str(tmp_path), dtype=dtype, max_seq_len=64, max_running=2)
    assert [o.token_ids for o in again.generate(prompts, params)] == first
