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


@pytest.mark.parametrize("kind", ["portions", "single tokens"])
def test_steps_on_several_streams(kind):
    """Steps that share a captured step, on two streams in turn, the first of which is busy when its step is launched."""
    from railgun_b200.engine.batch import StepEntry
    runner, toks = runner_of("C", "bfloat16", True, max_requests=32)
    plain, _ = runner_of("C", "bfloat16", True, max_requests=32)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    entries = {"portions": lambda r, i: [StepEntry(10 + i, toks[i % 3][i:i + 9], [8])],
               "single tokens": lambda r, i: [StepEntry(i % 2, [toks[i % 2][r.alloc.num_computed(i % 2)]], [0])]}[kind]
    for r in (runner, plain):
        for rid in (0, 1):
            r.step([StepEntry(rid, toks[rid][:50 + 10 * rid], [])])
        for i in range(6):                                              # captured
            r.step(entries(r, i))
    want = [plain.step(entries(plain, i)).clone() for i in range(6, 14)]
    torch.cuda.synchronize()
    got = []
    for i in range(6, 14):
        with torch.cuda.stream(streams[i % 2]):
            if i % 2 == 0:
                torch.cuda._sleep(4_000_000)                            # some two milliseconds
            got.append(runner.step(entries(runner, i)).clone())
    torch.cuda.synchronize()
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), i


@pytest.mark.parametrize("B", [1, 24])
def test_steps_that_are_packed_while_the_one_before_runs(B):
    """No results are read in between and the stream is busy, so that the host packs as soon as a step has read its numbers; 24
    requests in tables of 64 pages are more numbers than one block reads."""
    from railgun_b200.engine.batch import StepEntry
    logits = []
    for wait in (True, False):
        runner, toks = runner_of("C", "bfloat16", True, max_requests=32)
        runner.step([StepEntry(rid, toks[rid % 3][rid:rid + 150], []) for rid in range(B)])
        ids, out = np.arange(B), []
        for i in range(12):
            tokens = np.array([toks[(rid + i) % 3][i + rid] for rid in range(B)], dtype=np.int32)
            if not wait and i > 2:
                torch.cuda._sleep(400_000)
            out.append(runner.decode_step_flat(ids, tokens).clone())
            out.append(runner.last_greedy.clone())
            if wait:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        logits.append(out)
    for i, (a, b) in enumerate(zip(*logits)):
        assert torch.equal(a, b), i


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 4 * 256 * 592 + 5])
@pytest.mark.parametrize("at", [0, 1])
def test_a_result_goes_where_the_step_says(n, at):
    from railgun_b200 import ops
    src = torch.randn(n, device="cuda")
    room = torch.full((n + at + 1,), 7.0, device="cuda")
    where = torch.tensor([0, room[at:].data_ptr()], dtype=torch.int64, device="cuda").view(torch.int32)
    ops.step_result(src, where[:2])
    assert bool((room == 7.0).all())
    ops.step_result(src, where[2:])
    assert torch.equal(room[at:at + n], src) and bool((room[:at] == 7.0).all()) and float(room[-1]) == 7.0
    with pytest.raises(ops.KernelError):
        ops.step_result(src, where[1:3])
