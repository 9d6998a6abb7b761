"""Decode steps whose tokens are given, launched one behind the other without a wait of the host: every step's logits are
those of steps that are waited for, on one stream and on two in turn, whatever the number of requests does in between."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def runner_for(folder, dtype):
    from railgun_b200.config.llama import LlamaConfig
    from railgun_b200.engine.runner import ModelRunner
    from railgun_b200.weights.random_init import write_random_model
    cfg = LlamaConfig.from_dict(dict(
        architectures=["LlamaForCausalLM"], hidden_size=64, num_attention_heads=4, num_key_value_heads=2, head_dim=16,
        num_hidden_layers=2, intermediate_size=96, vocab_size=150, rope_theta=10000.0, tie_word_embeddings=True,
        max_position_embeddings=256))
    write_random_model(cfg, 3, folder, std=0.1)
    return ModelRunner(folder, dtype=dtype, max_tokens=2048, max_requests=8)


def steps(runner, wait, streams):
    """Twelve steps of four, three or one request(s), with the given tokens; the logits of each, or with several streams of
    the last (which reads what all steps wrote: a step's logits are overwritten by the next step, on whatever stream)."""
    from railgun_b200.engine.batch import StepEntry
    runner.step([StepEntry(i, [5 + i, 9, 20 + i], []) for i in range(4)])
    torch.cuda.synchronize()
    out = []
    for k in range(12):
        with torch.cuda.stream(streams[k % len(streams)]):
            n = (4, 4, 3, 4, 1, 4)[k % 6]
            logits = runner.step([StepEntry(i, [(7 * k + 31 * i) % 150], [0]) for i in range(n)])
            if len(streams) == 1 or k == 11:
                out.append(logits.clone())
        if wait:
            torch.cuda.synchronize()
    torch.cuda.synchronize()
    runner.end(range(4))
    return out


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_steps_launched_without_a_wait(tmp_path, dtype):
    runner = runner_for(str(tmp_path), dtype)
    here = torch.cuda.current_stream()
    steps(runner, True, [here])                                   # graphs are captured
    want = steps(runner, True, [here])
    for streams in ([here], [torch.cuda.Stream(), torch.cuda.Stream()]):
        got = steps(runner, False, streams)
        assert all(torch.equal(a, b) for a, b in zip(got[::-1], want[::-1]))
    runner.check_device_errors()
