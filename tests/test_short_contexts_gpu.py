"""Single tokens on short contexts, which have a captured step of their own: contexts that grow across its edge, and steps whose
requests' contexts are far longer or shorter than those of the step before, alone and together."""
import pytest

import helpers
from test_replay_gpu import compare, oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("name", ["B", "C"])
def test_steps_across_the_edge(name, dtype, tmp_path):
    from railgun_b200.engine.runner import SHORT_CONTEXT, ModelRunner
    from railgun_b200.replay import Replayer
    cfg, _, page = helpers.TINY[name]
    reqs, logits = oracle(name)
    by_length = sorted(reqs, key=lambda r: len(reqs[r]))
    long, grows = by_length[-1], by_length[-2]
    small = next(r for r in by_length if 40 <= len(reqs[r]) <= 100)
    start = {long: len(reqs[long]) - 8, grows: SHORT_CONTEXT - 6, small: 30}
    assert len(reqs[grows]) > SHORT_CONTEXT and len(reqs[long]) > SHORT_CONTEXT + 8
    # who decodes in each step: the small one alone, the long one directly behind it and before it, both, all three
    turns = [[grows]] * 4 + [[small], [long], [small], [small, long], [grows, small], [grows], [small], [grows, small, long], [small]]
    steps, fed = [], dict(start)
    tokens = {r: reqs[r] for r in (long, grows, small)}
    steps.append({"step": 0, "entries": [{"id": r, "tokens": t[:start[r]], "want": list(range(start[r]))} for r, t in tokens.items()],
                  "end": []})
    for i, who in enumerate(turns):
        entries = []
        for r in who:
            if fed[r] < len(tokens[r]):
                entries.append({"id": r, "tokens": [tokens[r][fed[r]]], "want": [0]})
                fed[r] += 1
        steps.append({"step": i + 1, "entries": entries, "end": []})
    steps[-1]["end"] = list(tokens)
    runner = ModelRunner(helpers.model_dir(name), dtype=dtype, page_size=page, max_tokens=helpers.peak_tokens(steps, 64),
                         max_requests=4)
    rp = Replayer(runner, tmp_path)
    for s in steps:
        rp.feed(s)
    reaches = {st.batch.max_context_len for st in runner._static.values()}
    assert SHORT_CONTEXT in reaches and 1024 in reaches
    runner.check_device_errors()
    runner.alloc.check()
    rows = helpers.collect(steps, tmp_path, cfg["vocab_size"])
    seen = {r: reqs[r][:fed[r]] for r in tokens}
    compare(rows, seen, {r: logits[r][:fed[r]] for r in tokens}, dtype, f"short contexts {name} {dtype}")
