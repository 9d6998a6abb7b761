"""Retention's and the delta rule's recurrences in chunks against the token-by-token loop in 64 bits, where they can go
wrong: portions of one token to several chunks, chunks of one token, requests that continue or have no slot, heads that share
keys, sizes that fill no tile, decays of 0 and 1, keys that point the same way."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

from test_mepatar_gpu import dev, rel, step_batch

pytestmark = pytest.mark.gpu
# 32-bit sums of up to 64 + 128 terms, through at most five chunks: about 1e-6 is seen; and what the token-by-token kernel
# is held to
BOUND = 2e-5


def loop(q, k, v, S, g, beta=None):
    o = np.zeros_like(v)
    for t in range(q.shape[0]):
        S *= g[t]
        S += np.outer(k[t], v[t] if beta is None else beta[t] * (v[t] - S.T @ k[t]))
        o[t] = S.T @ q[t]
    return o


SIZES = [(4, 4, 32, 16), (4, 2, 16, 8), (3, 1, 8, 24), (5, 5, 12, 20), (2, 2, 128, 128), (4, 2, 64, 136), (2, 1, 100, 72),
         (1, 1, 4, 4)]
LENGTHS = [[64, 1, 65], [63, 128, 200], [129], [300, 2]]


@pytest.mark.parametrize("rule", ["retention", "delta"])
@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("H,Hqk,d,dv", SIZES)
def test_chunks_against_the_loop(H, Hqk, d, dv, lengths, rule):
    from railgun_b200 import ops
    rng = np.random.default_rng(H * d + dv + lengths[0])
    R, T = len(lengths), sum(lengths)
    q, k = rng.normal(size=(2, T, Hqk, d)) * 0.3
    v = rng.normal(size=(T, H, dv))
    if rule == "delta":
        k += rng.normal(size=(1, Hqk, d)) * 0.6                       # keys that partly point the same way
        k /= np.linalg.norm(k, axis=-1, keepdims=True)
        loga = -rng.exponential(size=(T, H)) * np.logspace(-4, 0.5, H)
        beta = rng.uniform(0.05, 1.0, size=(T, H))
    else:
        decay = np.linspace(0.9, 1.0, H) if H != 3 else np.array([0.0, 0.5, 1.0])
        loga = np.broadcast_to(np.log(np.maximum(decay, 1e-300)), (T, H))
        beta = None
    v_type = torch.bfloat16 if d == 128 else torch.float32
    v = torch.tensor(v, dtype=v_type).double().numpy()
    slots = [R - 1 - r for r in range(R)]
    starts = [0 if r == 1 else 7 for r in range(R)]
    state0 = rng.normal(size=(R + 1, H, dv, d))
    f32 = lambda a: dev(np.ascontiguousarray(a), torch.float32)
    state = f32(state0)
    rows = torch.cat([f32(q.reshape(T, -1)), f32(k.reshape(T, -1)), torch.zeros(T, 4, device=state.device)], 1)   # views
    qv, kv = rows[:, :Hqk * d], rows[:, Hqk * d:2 * Hqk * d]
    vv = dev(v.reshape(T, -1), v_type)
    batch = step_batch(lengths, starts, slots)
    if rule == "delta":
        got = ops.delta_chunk_scan(qv, kv, vv, state, batch, H, d, dv, f32(loga), f32(beta))
    else:
        got = ops.decay_chunk_scan(qv, kv, vv, state, batch, H, d, dv, f32(decay).double().log())
    got, state = got.cpu().double().numpy(), state.cpu().double().numpy()
    assert np.isfinite(got).all()
    g = np.exp(loga) if rule == "delta" else np.broadcast_to(f32(decay).double().cpu().numpy(), (T, H))
    lo = 0
    for r, n in enumerate(lengths):
        for h in range(H):
            S = state0[slots[r], h].T.copy() if starts[r] else np.zeros((d, dv))
            span, hq = slice(lo, lo + n), h // (H // Hqk)
            ref = loop(q[span, hq], k[span, hq], v[span, h], S, g[span, h], beta[span, h] if rule == "delta" else None)
            assert rel(got[span, h], ref) < BOUND and rel(state[slots[r], h], S.T) < BOUND, (r, h)
        lo += n
    assert np.array_equal(state[R], state0[R].astype(np.float32))     # nobody's slot


@pytest.mark.parametrize("rule", ["retention", "delta"])
def test_no_slot_and_cut_portions(rule):
    """A row without a slot reads zeros and writes nothing; a prompt in two portions is what it is in one."""
    from railgun_b200 import ops
    H, d, dv, T = 2, 32, 32, 210
    gen = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (0.2 * torch.randn(T, H * d, device="cuda", generator=gen) for _ in range(3))
    k = torch.nn.functional.normalize(k.view(T, H, d), dim=-1).reshape(T, H * d)
    loga = -torch.rand(T, H, device="cuda", generator=gen) * 0.1
    beta = torch.rand(T, H, device="cuda", generator=gen)
    log_decay = torch.tensor([-0.01, -0.2], dtype=torch.float64, device="cuda")

    def run(lo, hi, state, start, slot):
        batch, part = step_batch([hi - lo], [start], [slot]), slice(lo, hi)
        if rule == "delta":
            return ops.delta_chunk_scan(q[part], k[part], v[part], state, batch, H, d, dv, loga[part].contiguous(), beta[part].contiguous())
        return ops.decay_chunk_scan(q[part], k[part], v[part], state, batch, H, d, dv, log_decay)

    state = torch.full((1, H, dv, d), 9.0, device="cuda")
    whole = run(0, T, state, 0, 0)
    kept = state.clone()
    assert rel(run(0, T, state, 5, -1), whole.cpu().double().numpy()) < 1e-6 and torch.equal(state, kept)
    two = torch.cat([run(0, 77, state, 0, 0), run(77, T, state, 77, 0)])
    assert rel(two, whole.cpu().double().numpy()) < BOUND and rel(state, kept.cpu().double().numpy()) < BOUND


def test_what_it_refuses():
    from railgun_b200 import ops
    state = torch.zeros(1, 1, 4, 6, device="cuda")
    assert not ops.delta_chunk_ok(torch.zeros(2, 6, device="cuda"), state, 6, 4)
    assert not ops.delta_chunk_ok(torch.zeros(2, 132, device="cuda"), torch.zeros(1, 1, 4, 132, device="cuda"), 132, 4)
    assert not ops.delta_chunk_ok(torch.zeros(2, 9, device="cuda")[:, 1:], torch.zeros(1, 1, 4, 8, device="cuda"), 8, 4)


@pytest.mark.parametrize("rule", ["retention", "delta"])
def test_each_request_by_its_own_length(rule):
    """Long portions run in chunks and the others token by token, as they would in a step of their own."""
    from railgun_b200 import ops
    least = ops.DECAY_CHUNK_MIN_TOKENS if rule == "retention" else ops.DELTA_CHUNK_MIN_TOKENS
    lengths = [1, least + 70, least - 1, 1, least, 3]
    starts, slots = [9, 0, 4, 0, 7, 2], [2, 0, 5, 1, -1, 4]
    H, d, dv, T = 4, 64, 32, sum(lengths)
    gen = torch.Generator(device="cuda").manual_seed(8)
    q, k, v = (0.2 * torch.randn(T, H * n, device="cuda", generator=gen) for n in (d, d, dv))
    k = torch.nn.functional.normalize(k.view(T, H, d), dim=-1).reshape(T, H * d)
    loga, beta = -torch.rand(T, H, device="cuda", generator=gen), torch.rand(T, H, device="cuda", generator=gen)
    decay = torch.tensor([0.5, 0.9, 0.99, 1.0], device="cuda")
    state0 = torch.randn(6, H, dv, d, device="cuda", generator=gen)

    def step(part, lengths, starts, slots, scan, chunks):
        batch, state = step_batch(lengths, starts, slots), state0.clone()
        batch.max_query_len, batch.layout = max(lengths), (tuple(lengths),)
        a, b, more = loga[part].contiguous(), beta[part].contiguous(), scan and chunks
        args, o = (q[part], k[part], v[part], state, batch, H, d, dv), None
        if scan:
            below = least if more else 0
            o = ops.state_scan(*args, decay=decay, below=below) if rule == "retention" else \
                ops.state_scan(*args, g=a.exp(), beta=b, below=below)
        if chunks:
            own = dict(least=least, o=o) if more else {}
            o = ops.decay_chunk_scan(*args, decay.double().log(), **own) if rule == "retention" else \
                ops.delta_chunk_scan(*args, a, b, **own)
        return o, state

    whole = slice(0, T)
    assert ops.scan_split(SimpleNamespace(max_query_len=max(lengths), layout=(tuple(lengths),)), least) == (
        -(-(least + 70) // 64) + -(-least // 64), True)
    got, state = step(whole, lengths, starts, slots, True, True)
    want, scanned = step(whole, lengths, starts, slots, True, False)
    lo = 0
    for r, n in enumerate(lengths):
        part = slice(lo, lo + n)
        if n >= least:
            alone, after = step(part, [n], starts[r:r + 1], slots[r:r + 1], False, True)
        else:
            alone, after = want[part], scanned
        assert torch.equal(got[part], alone), r
        if slots[r] >= 0:
            assert torch.equal(state[slots[r]], after[slots[r]]), r
        lo += n
    assert torch.equal(state[3], state0[3])                             # nobody's slot


@pytest.mark.parametrize("rule", ["retention", "delta", "delta that forgets"])
def test_no_further_off_than_token_by_token(rule):
    """Both forms against 64 bits, over the decays that models have: sums of 128 products in one chain, as the chunks once made
    them, were 1.4 to 2.2 times as far off as the token-by-token kernel; sums of fours are 0.6 to 0.99 times."""
    from railgun_b200 import ops
    H, d, T = 4, 128, 400
    rng = np.random.default_rng(11)
    unit = lambda a: a / np.linalg.norm(a, axis=-1, keepdims=True)   # noqa: E731
    q, k, v = unit(rng.normal(size=(T, H, d))), unit(rng.normal(size=(T, H, d))), rng.normal(size=(T, H, d))
    q, k, v = (a.astype(np.float32) for a in (q, k, v))
    loga = (rng.uniform(size=(T, H)) * (-2.0 if rule == "delta that forgets" else -0.01)).astype(np.float32)
    beta = rng.uniform(size=(T, H)).astype(np.float32)
    decay = np.array([1.0 - 2.0 ** (-5 - 0.8 * i) for i in range(H)], dtype=np.float32)
    batch, rows = step_batch([T], [0], [0]), [dev(a.reshape(T, -1)) for a in (q, k, v)]
    state = lambda: torch.zeros(1, H, d, d, device="cuda")           # noqa: E731
    if rule == "retention":
        scan = ops.state_scan(*rows, state(), batch, H, d, d, decay=dev(decay))
        chunks = ops.decay_chunk_scan(*rows, state(), batch, H, d, d, dev(decay).double().log())
        g = np.broadcast_to(decay.astype(np.float64), (T, H))
    else:
        scan = ops.state_scan(*rows, state(), batch, H, d, d, g=dev(loga).exp(), beta=dev(beta))
        chunks = ops.delta_chunk_scan(*rows, state(), batch, H, d, d, dev(loga), dev(beta))
        g = np.exp(loga.astype(np.float64))
    ref = np.stack([loop(*(a[:, h].astype(np.float64) for a in (q, k, v)), np.zeros((d, d)), g[:, h],
                         None if rule == "retention" else beta[:, h].astype(np.float64)) for h in range(H)], 1)
    off = lambda a: np.linalg.norm(a.cpu().double().numpy() - ref)    # noqa: E731
    assert off(chunks) < 1.05 * off(scan)


@pytest.mark.parametrize("rule", ["retention", "delta"])
@pytest.mark.parametrize("at", [3, 37, 64, 130])
def test_a_later_tokens_infinity_stays_out_of_earlier_outputs(rule, at):
    """Within a chunk a token's weight for a later one is left out, not multiplied by zero."""
    from railgun_b200 import ops
    H, d, dv, T = 2, 32, 36, 200
    gen = torch.Generator(device="cuda").manual_seed(at)
    q, k, v = (0.2 * torch.randn(T, H * n, device="cuda", generator=gen) for n in (d, d, dv))
    loga, beta = -torch.rand(T, H, device="cuda", generator=gen) * 0.1, torch.rand(T, H, device="cuda", generator=gen) + 0.1
    log_decay, batch = torch.tensor([-0.01, -0.2], dtype=torch.float64, device="cuda"), step_batch([T], [0], [0])

    def run(v):
        args = (q, k, v, torch.zeros(1, H, dv, d, device="cuda"), batch, H, d, dv)
        return ops.delta_chunk_scan(*args, loga, beta) if rule == "delta" else ops.decay_chunk_scan(*args, log_decay)

    want = run(v)
    v[at, 5] = float("inf")
    got = run(v)
    assert torch.equal(got[:at], want[:at]) and not torch.isfinite(got[at, 0, 5])
