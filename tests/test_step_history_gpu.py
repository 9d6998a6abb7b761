"""What a step computes does not depend on the steps before it: on which of them was captured, on their contexts, on the stream
they ran on; and what it returned stays what it was where it is the caller's."""
import numpy as np
import pytest
import torch

import helpers

pytestmark = pytest.mark.gpu


def runner_of(name, dtype, graphs, max_requests=8):
    from railgun_b200.engine.runner import ModelRunner
    cfg, _, page = helpers.TINY[name]
    return ModelRunner(helpers.model_dir(name), dtype=dtype, page_size=page, max_tokens=8192, max_requests=max_requests,
                       use_graphs=graphs), helpers.prompts(cfg["vocab_size"], [960, 950, 940, 40], seed=5)


def portions_beside(runner, toks, contexts, portion=8):
    """Steps of one layout: a new request's portion beside one of the requests that hold ``contexts`` tokens, in turn."""
    from railgun_b200.engine.batch import StepEntry
    out = []
    for i, n in enumerate(contexts):
        if not runner.alloc.has(n):
            runner.step([StepEntry(n, toks[n % 3][:n], [])])
        fed = runner.alloc.num_computed(n)
        out.append(runner.step([StepEntry(n, [toks[n % 3][fed]], [0]), StepEntry(5000 + i, toks[3][i:i + portion], [0, portion - 1])]))
        runner.end([5000 + i])
    return out


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_short_steps_keep_their_logits(dtype):
    runner, toks = runner_of("C", dtype, True)
    plain, _ = runner_of("C", dtype, False)
    contexts = [520] * 9
    got, want = portions_beside(runner, toks, contexts), portions_beside(plain, toks, contexts)      # none read before all have run
    assert len(runner._short_steps.graphs) == 1
    assert len({t.data_ptr() for t in got}) == len(got)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_steps_of_one_layout_and_other_parts_of_contexts(dtype):
    """A portion beside one single token: 520 and 600 keys make three parts, 780 and 800 four, all in tables of one width."""
    runner, toks = runner_of("C", dtype, True)
    plain, _ = runner_of("C", dtype, False)
    contexts = [520] * 6 + [780, 600, 800] + [780] * 5 + [520, 780]
    got, want = portions_beside(runner, toks, contexts), portions_beside(plain, toks, contexts)
    assert len(runner._short_steps.graphs) == (2 if dtype == "bfloat16" else 1)             # 32-bit attention is in one part
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), (i, contexts[i])


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_single_tokens_after_longer_and_shorter_ones(dtype):
    """A request of 100 tokens decodes alone, and behind one and three steps of one with 880."""
    from railgun_b200.engine.batch import StepEntry
    results = []
    for between in ([], [[0]], [[0]] * 3):
        runner, toks = runner_of("C", dtype, True)
        for rid, n in ((0, 880), (1, 100)):
            runner.step([StepEntry(rid, toks[rid][:n], [])])
        for who in between:
            runner.step([StepEntry(rid, [toks[rid][runner.alloc.num_computed(rid)]], [0]) for rid in who])
        steps = {}
        for _ in range(6):
            at = runner.alloc.num_computed(1)
            steps[at] = runner.step([StepEntry(1, [toks[1][at]], [0])]).clone()
        results.append(steps)
    for other in results[1:]:
        for at in set(other) & set(results[0]):
            assert torch.equal(other[at], results[0][at]), at
