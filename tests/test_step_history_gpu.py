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
                       use_graphs=graphs), helpers.prompts(cfg["vocab_size"], [900, 700, 600, 40], seed=5)


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
