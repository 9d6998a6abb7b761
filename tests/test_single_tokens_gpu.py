"""The kernels that single-token steps of the mixers take where sizes and addresses allow: the streamed product with a bias and
over several inputs at once, the convolution that moves its state on itself, norms over all heads several numbers at a time."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def rel(a, b):
    return float((a.double() - b.double()).abs().max() / b.double().abs().max())


@pytest.mark.parametrize("M", [1, 7, 16, 17])
@pytest.mark.parametrize("N,K", [(2576, 2048), (16, 8), (50, 264), (9520, 128), (40000, 64), (2048, 4104)])
def test_product_with_a_bias(M, N, K):
    """Every launch shape of the product, ragged last tiles; 17 rows are the library's."""
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + N)
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = torch.randn(N, K, device=DEV, generator=g).bfloat16()
    b = torch.randn(N, device=DEV, generator=g).bfloat16() * K ** 0.5
    exact = x.double() @ w.double().T + b.double()
    got = ops.linear(x, w, bias=b)
    # one rounding to bfloat16 of a sum that is off by K 2^-24 of its terms at most
    assert (got.double() - exact).abs().max() <= (2.0 ** -8 + 2.0 ** -14) * exact.abs().max()
    assert torch.equal(ops.linear(x, w, bias=b), got)
    if M <= 16:
        assert torch.equal(ops.linear(x, w, bias=torch.zeros_like(b)), ops.linear(x, w))


@pytest.mark.parametrize("M", [4, 48])
def test_products_that_stay_the_librarys(M):
    """With a bias, of several inputs, and logits of 41 to 64 rows: a matrix elsewhere is refused, one off a 16-byte boundary is
    taken, and derivatives and maps go through the product."""
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M)
    N, K = (64, 128) if M <= 16 else (5 * 148 * 128 + 64, 64)
    flat = torch.randn(N * K + 1, device=DEV, generator=g).bfloat16()
    w, odd = flat[:N * K].view(N, K), flat[1:].view(N, K)
    x, b = torch.randn(M, K, device=DEV, generator=g).bfloat16(), torch.randn(N, device=DEV, generator=g).bfloat16()
    bias, out_dtype = (b, None) if M <= 16 else (None, torch.float32)
    calls = [lambda x, w, b: ops.linear(x, w, out_dtype, bias=bias if b is None else b)]
    if M <= 16:
        calls.append(lambda x, w, b: ops.linear_groups(x[None], w[None])[0])
    for call in calls:
        exact = lambda w: x.double() @ w.double().T + (b.double() if call is calls[0] and M <= 16 else 0.0)  # noqa: E731
        # one rounding to bfloat16 at most, of a sum that is off by K 2^-24 of its terms at most
        assert (call(x, odd, None).double() - exact(odd)).abs().max() <= (2.0 ** -8 + 2.0 ** -14) * exact(odd).abs().max()
        with pytest.raises(RuntimeError):
            call(x, w.cpu(), None)
        with pytest.raises(RuntimeError):
            call(x.cpu(), w, None)
    if M <= 16:
        with pytest.raises(RuntimeError):
            ops.linear(x, w, bias=b.cpu())
        xg, wg, bg = (t.clone().requires_grad_() for t in (x, w, b))
        ops.linear(xg, wg, bias=bg).float().sum().backward()
        assert torch.allclose(bg.grad.float(), torch.full((N,), float(M), device=DEV))
        assert rel(wg.grad, x.double().sum(0).expand_as(w)) < 2.0 ** -7 and rel(xg.grad, w.double().sum(0).expand_as(x)) < 2.0 ** -7
        moved = torch.func.jvp(lambda a: ops.linear(a, w, bias=b), (x,), (torch.ones_like(x),))[1]
        assert rel(moved, w.double().sum(1).expand(M, N)) < 2.0 ** -7
        maps = torch.vmap(lambda m: ops.linear(x, m, bias=b))(torch.stack([w, 2 * w]))
        assert rel(maps[1], 2 * x.double() @ w.double().T + b.double()) < 2.0 ** -7


@pytest.mark.parametrize("M,G,N,K", [(1, 4, 1024, 2048), (16, 4, 64, 48), (5, 3, 32, 8), (8, 2, 2400, 72), (17, 4, 64, 64), (3, 4, 48, 64)])
def test_products_of_several_inputs(M, G, N, K):
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(N)
    x = torch.randn(G, M, K, device=DEV, generator=g).bfloat16()
    w = torch.randn(G, N, K, device=DEV, generator=g).bfloat16()
    exact = x.double() @ w.double().transpose(1, 2)
    got = ops.linear_groups(x, w)
    assert got.dtype == torch.float32 and got.shape == (G, M, N)
    assert rel(got, exact) < K * 2.0 ** -24 + 1e-6
    assert rel(ops.linear_groups(x.float(), w.float()), exact) < K * 2.0 ** -24 + 1e-6


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C,K", [(48, 4), (1536, 4), (40, 2), (37, 3), (1032, 6)])
def test_convolution_moves_its_state_on(C, K, dtype):
    """Single tokens: new requests, requests with a past, padding rows without a slot, against the two kernels one after the
    other (the same bits)."""
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(C)
    R = 5
    x = torch.randn(R, C + 8, device=DEV, generator=g).to(dtype)
    taps = torch.randn(K, C, device=DEV, generator=g)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(cu_seqlens=i32(list(range(R + 1))), req_of_token=i32(list(range(R))), start_pos=i32([3, 0, 1, 900, 0]),
                            state_slots=i32([4, 0, -1, 2, -1]), num_requests=R, decode_only=True)
    state = torch.randn(6, K - 1, C, device=DEV, generator=g)
    one, two = state.clone(), state.clone()
    got = ops.causal_conv(x, 8, taps, one, batch, dtype, silu=True, update=True)
    want = ops.causal_conv(x, 8, taps, two, batch, dtype, silu=True)
    ops.conv_state_update(x, 8, two, batch)
    assert torch.equal(got, want) and torch.equal(one, two) and not torch.equal(one, state)


@pytest.mark.parametrize("types", [("float32", "float32"), ("bfloat16", "bfloat16"), ("float32", "bfloat16")])
@pytest.mark.parametrize("H,G,d,dims", [(8, 2, 128, 64), (20, 4, 96, 8), (3, 1, 24, 0), (40, 8, 64, 64)])
@pytest.mark.parametrize("T", [6, 149])
@pytest.mark.parametrize("whole", [True, False])
def test_prepare_several_numbers_at_a_time(H, G, d, dims, types, T, whole):
    """A head a warp (few tokens) and four (more tokens than SMs), normed over all heads or each alone, against the form that takes
    one number at a time."""
    from railgun_b200 import ops
    from railgun_b200.parts.latent_attention import rotary_frequencies
    a, o = (getattr(torch, t) for t in types)
    g = torch.Generator(device=DEV).manual_seed(H * d)
    page, n = 4, (H + 2 * G) * d
    x = torch.randn(T, n, device=DEV, generator=g).to(a)
    odd = torch.zeros(T, n + 1 + n % 2, dtype=a, device=DEV)[:, :n]       # rows that only the one-number form takes
    odd.copy_(x)
    freq = rotary_frequencies(dims, 1e4).to(DEV) if dims else torch.zeros(1, dtype=torch.float64, device=DEV)
    pos = torch.randint(0, 70000, (T,), device=DEV, generator=g, dtype=torch.int32)
    slots = torch.arange(T, dtype=torch.int32, device=DEV)
    slots[1] = -1
    qn, kn = (torch.rand(h * d if whole else d, device=DEV, generator=g) + 0.5 for h in (H, G))
    got = []
    for rows in (x, odd):
        cache = torch.full((T // page + 1, 2, G, page, d), 7.0, dtype=o, device=DEV)
        q = ops.attention_prepare(rows, cache, qn, kn, 1e-5, freq, dims, not whole, pos, slots, None, H, G, d, d, d,
                                  norm_whole=whole, out_dtype=o)
        got.append((q, cache))
    # 32-bit: a root mean square added up in another order; bfloat16: one unit where that tips a rounding
    tol = 2e-6 if o == torch.float32 else 2.0 ** -7
    assert rel(got[0][0], got[1][0]) <= tol and rel(got[0][1], got[1][1]) <= tol
    assert torch.equal(got[0][1] == 7.0, got[1][1] == 7.0)


@pytest.mark.parametrize("types", [("float32", "float32"), ("bfloat16", "bfloat16"), ("float32", "bfloat16")])
@pytest.mark.parametrize("H,dv", [(8, 128), (1, 4), (3, 24), (16, 128), (33, 124), (33, 128)])
@pytest.mark.parametrize("whole", [False, True])
def test_norm_and_gate(H, dv, types, whole):
    """Rows of up to and above what a block keeps in registers; heads of up to and above a warp's width."""
    from railgun_b200 import ops
    a, o = (getattr(torch, t) for t in types)
    g = torch.Generator(device=DEV).manual_seed(H * dv)
    T = 3
    x = torch.randn(T, H, dv, device=DEV, generator=g)
    z = torch.randn(T, H * dv + 8, device=DEV, generator=g).to(a)[:, 8:]
    w = torch.rand(H * dv, device=DEV, generator=g) + 0.5
    for kind, weight in (("silu", w), ("sigmoid", None)):
        y = x.double() / (x.double().pow(2).mean((1, 2) if whole else 2, keepdim=True) + 1e-5).sqrt()
        y = y.flatten(1) * (1.0 if weight is None else weight.double())
        s = torch.sigmoid(z.double())
        exact = y * (s if kind == "sigmoid" else s * z.double()) * 0.7
        got = ops.head_norm_gate(x, z, weight, 1e-5, o, whole=whole, gate_kind=kind, out_scale=0.7)
        assert rel(got, exact) < (2e-6 if o == torch.float32 else 2.0 ** -8)


@pytest.mark.parametrize("T,H", [(1, 4), (3, 4096), (592, 2048), (593, 2048), (149, 4100), (2, 16384), (160, 16384), (2, 16388), (150, 32768), (2, 32772)])
def test_rows_kept_in_registers(T, H):
    """One, two and four pieces a thread, and rows that are too wide for that; rows picked out; nothing pending."""
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(H)
    x, w = torch.randn(T, H, device=DEV, generator=g), torch.rand(H, device=DEV, generator=g) + 0.5
    unit = lambda v: v / (v.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()
    for pending in (torch.randn(T, H, device=DEV, generator=g).bfloat16(), torch.randn(T, H, device=DEV, generator=g), None):
        resid = x.clone()
        new = x if pending is None else x + pending.float()
        for dt in (torch.float32, torch.bfloat16):
            r = x.clone()
            got = ops.add_rmsnorm(r, pending, w, 1e-5, dt)
            assert torch.equal(r, new) and rel(got, unit(new.double()) * w.double()) < (2e-6 if dt == torch.float32 else 2.0 ** -8)
        rows = torch.tensor([T - 1, 0], dtype=torch.int32, device=DEV)
        got = ops.add_rmsnorm(resid, pending, w, 1e-5, torch.float32, rows=rows)
        assert torch.equal(resid, x) and rel(got, (unit(new.double()) * w.double())[rows.long()]) < 2e-6


@pytest.mark.parametrize("T,H,groups", [(2, 8192, 1), (593, 2048, 4), (3, 4096, 1), (150, 1024, 1), (5, 4096, 32), (2, 36864, 9), (7, 20, 5)])
def test_groups_kept_in_registers(T, H, groups):
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(H)
    x, w1, w2 = torch.randn(T, H, device=DEV, generator=g), *(torch.rand(H, device=DEV, generator=g) + 0.5 for _ in range(2))
    a, b = torch.randn(T, H, device=DEV, generator=g).bfloat16(), torch.randn(T, H, device=DEV, generator=g)
    unit = lambda v: (v.unflatten(1, (groups, -1)) / (v.unflatten(1, (groups, -1)).pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()).flatten(1)
    new = (x + a.float()) + b
    r = x.clone()
    one, two = ops.add_group_rmsnorm(r, ops.PendingSum([a, b]), [w1, w2], groups, 1e-5, torch.float32)
    exact = unit(new.double())
    assert torch.equal(r, new) and rel(one, exact * w1.double()) < 2e-6 and rel(two, exact * w2.double()) < 2e-6
    rows = torch.tensor([T - 1], dtype=torch.int32, device=DEV)
    r = x.clone()
    got, = ops.add_group_rmsnorm(r, ops.PendingSum([a, b]), [w1], groups, 1e-5, torch.float32, rows=rows)
    assert torch.equal(r, x) and rel(got, (exact * w1.double())[-1:]) < 2e-6


@pytest.mark.parametrize("H", [4, 2048, 4096, 4100, 8192, 8196])
@pytest.mark.parametrize("normed", [True, False])
def test_stream_rows_and_the_shift(H, normed):
    """A block per row up to 8,192 numbers, above the general form: portions, single tokens, a request without a slot."""
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(H)
    lengths, starts, slots = [3, 1, 2, 1, 1], [5, 0, 0, 7, 2], [2, 4, 0, 1, -1]
    T = sum(lengths)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    at = [sum(lengths[:i]) for i in range(len(lengths) + 1)]
    batch = SimpleNamespace(cu_seqlens=i32(at), req_of_token=i32([r for r, n in enumerate(lengths) for _ in range(n)]),
                            start_pos=i32(starts), state_slots=i32(slots))
    x, y = torch.randn(T, H, device=DEV, generator=g), torch.randn(T, H, device=DEV, generator=g)
    w, share = torch.rand(H, device=DEV, generator=g) + 0.5, torch.rand(H, device=DEV, generator=g)
    state = torch.randn(5, 1, H, device=DEV, generator=g)
    unit = y.double() / (y.double().pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() if normed else y.double()
    new = x.double() + unit
    before, after = torch.zeros_like(new), state.double().clone()
    for r, n in enumerate(lengths):
        before[at[r] + 1:at[r + 1]] = new[at[r]:at[r + 1] - 1]
        if slots[r] >= 0:
            if starts[r]:
                before[at[r]] = state[slots[r], 0].double()
            after[slots[r], 0] = new[at[r + 1] - 1]
    pending = ops.PendingNormed(y, w, 1e-5) if normed else y
    rows, h = ops.postnorm_shift(x, pending, share, state, batch, torch.float32)
    assert rel(rows, new) < 2e-6 and rel(h, new + (before - new) * share.double()) < 2e-6 and rel(state, after) < 2e-6
    rows, h = ops.postnorm_shift(x, pending, None, None, None, torch.float32)
    assert rows is x and rel(x, new) < 2e-6 and torch.equal(h, x)


@pytest.mark.parametrize("nh,nkv,d", [(32, 8, 64), (24, 8, 128), (4, 2, 48)])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("portions", [1, 9])
def test_single_tokens_beside_portions(nh, nkv, d, splits, portions):
    """Single tokens' attention that starts beside the portions' of the same step: the bits of both in turn, many times over."""
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(nh * d + portions)
    page, tokens, singles, ctx = 16, 130, 11, 700
    R, width = portions + singles, -(-ctx // page)
    T = portions * tokens + singles
    kv = torch.randn(R * width, 2, nkv, page, d, device=DEV, generator=g).bfloat16()
    table = torch.randperm(R * width, device=DEV, generator=g).to(torch.int32).view(R, width)
    q = torch.randn(T, (nh + 2 * nkv) * d, device=DEV, generator=g).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pos = i32([j for _ in range(portions) for j in range(ctx - tokens, ctx)] + [ctx - 1 - 60 * j for j in range(singles)])
    req = i32([r for r in range(portions) for _ in range(tokens)] + list(range(portions, R)))
    rows = i32(list(range(portions * tokens, T)))

    def tiles(size):
        return i32([[r * tokens + a, min(size, tokens - a), r] for r in range(portions) for a in range(0, tokens, size)])

    t128, t64 = tiles(128), tiles(64)

    def step(beside):
        out = torch.zeros(T, nh * d, dtype=torch.bfloat16, device=DEV)
        if d == 64:
            ops.prefill_attention_tc(q, out, kv, table, t128, pos, nh, nkv, d, 0, d ** -0.5)
        elif d == 128:
            ops.prefill_attention_wide(q, out, kv, table, t128, pos, nh, nkv, d, 0, d ** -0.5)
        else:
            ops.prefill_attention(q, q.shape[1], out, kv, table, t64, pos, nh, nkv, d, 0, d ** -0.5)
        ops.decode_attention(q, q.shape[1], out, kv, table, rows, singles, req, pos, nh, nkv, d, 0, d ** -0.5, splits, beside=beside)
        return out.clone()                                                  # behind both

    want = step(False)
    for _ in range(20):
        assert torch.equal(step(True), want)
    ops.tc_gemm_check()


@pytest.mark.parametrize("nh,nkv,d", [(32, 8, 64), (24, 8, 128), (4, 2, 48)])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("portions", [1, 9])
def test_single_tokens_beside_portions_between_a_steps_kernels(nh, nkv, d, splits, portions):
    """In the same buffers again and again, launched one by one and as a graph: a kernel that writes the queries and the step's own
    keys and values directly in front, and one that reads every row of the output directly behind."""
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(nh * d + portions + splits)
    page, tokens, singles, ctx, turns = 16, 130, 11, 700, 6
    R, width = portions + singles, -(-ctx // page)
    T = portions * tokens + singles
    first = torch.randn(R * width, 2, nkv, page, d, device=DEV, generator=g).bfloat16()
    table = torch.randperm(R * width, device=DEV, generator=g).to(torch.int32).view(R, width)
    news = [torch.randn(T, (nh + 2 * nkv) * d, device=DEV, generator=g).bfloat16() for _ in range(turns)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    pos = i32([j for _ in range(portions) for j in range(ctx - tokens, ctx)] + [ctx - 1 - 60 * j for j in range(singles)])
    req = i32([r for r in range(portions) for _ in range(tokens)] + list(range(portions, R)))
    slots = (table[req.long(), (pos // page).long()] * page + pos % page).to(torch.int32)
    rows = i32(list(range(portions * tokens, T)))
    tiles = lambda size: i32([[r * tokens + a, min(size, tokens - a), r] for r in range(portions) for a in range(0, tokens, size)])
    t128, t64 = tiles(128), tiles(64)
    angles = torch.randn(ctx, d, device=DEV, generator=g)
    weight = torch.rand(nh * d, device=DEV, generator=g) + 0.5
    kv, qkv, resid = first.clone(), news[0].clone(), torch.zeros(T, nh * d, device=DEV)

    def step(new, beside):
        out = torch.full((T, nh * d), float("nan"), dtype=torch.bfloat16, device=DEV)
        resid.zero_()
        qkv.copy_(new)
        ops.rope_cache_write(qkv, angles, pos, slots, kv, nh, nkv, d, page, None)
        if d == 64:
            ops.prefill_attention_tc(qkv, out, kv, table, t128, pos, nh, nkv, d, 0, d ** -0.5)
        elif d == 128:
            ops.prefill_attention_wide(qkv, out, kv, table, t128, pos, nh, nkv, d, 0, d ** -0.5)
        else:
            ops.prefill_attention(qkv, qkv.shape[1], out, kv, table, t64, pos, nh, nkv, d, 0, d ** -0.5)
        ops.decode_attention(qkv, qkv.shape[1], out, kv, table, rows, singles, req, pos, nh, nkv, d, 0, d ** -0.5, splits, beside=beside)
        return ops.add_rmsnorm(resid, out, weight, 1e-5, torch.float32)

    def all_of(run):
        kv.copy_(first)
        return [run(new).clone() for new in news * 2]

    want = all_of(lambda new: step(new, False))
    assert all(bool(t.isfinite().all()) for t in want)
    for got, one in zip(all_of(lambda new: step(new, True)), want):
        assert torch.equal(got, one)
    source, graph = news[0].clone(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        result = step(source, True)

    def replay(new):
        source.copy_(new)
        graph.replay()
        return result
    for got, one in zip(all_of(replay), want):
        assert torch.equal(got, one)
    ops.tc_gemm_check()


@pytest.mark.parametrize("nh,nkv,d", [(1, 1, 16), (32, 8, 64), (32, 8, 128), (64, 16, 128), (8, 8, 256)])
@pytest.mark.parametrize("paired", [False, True])
def test_rotation_and_cache_write(nh, nkv, d, paired):
    """Rows of less and of more pieces than a block has threads; tokens without a slot, a position outside the table."""
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(nh * d)
    T, page = 7, 4
    x = torch.randn(T, (nh + 2 * nkv) * d, device=DEV, generator=g).bfloat16()
    angle = torch.rand(50, d // 2, device=DEV, generator=g) * 6.0
    table = torch.cat([angle.cos(), angle.sin()], 1)
    pos = torch.tensor([0, 49, 3, 50, 7, 8, 9], dtype=torch.int32, device=DEV)
    slots = torch.tensor([3, 0, -1, 9, 4, 11, 6], dtype=torch.int32, device=DEV)
    cache = torch.full((3, 2, nkv, page, d), 7.0, dtype=torch.bfloat16, device=DEV)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    order = ops.rope_pair_order(d).to(DEV) if paired else torch.arange(d, device=DEV)      # storage index -> feature
    heads = x.view(T, -1, d)
    plain = torch.empty_like(heads)
    plain[..., order] = heads                                              # features in the model's order
    c, s = (table[pos.long().clamp(max=49) * (pos < 50)][:, None, i * d // 2:(i + 1) * d // 2].double() for i in (0, 1))
    u, v = plain[..., :d // 2].double(), plain[..., d // 2:].double()
    turned = torch.cat([u * c - v * s, v * c + u * s], -1)[..., order]
    want = torch.cat([turned[:, :nh + nkv], heads[:, nh + nkv:].double()], 1)
    got = x.clone()
    ops.rope_cache_write(got, table, pos, slots, cache, nh, nkv, d, page, err_flag=err, paired8=paired)
    close = lambda a, b: (a.double() - b).abs().max() <= 2.0 ** -8 * b.abs().max()
    assert close(got.view(T, -1, d)[:, :nh + nkv], want[:, :nh + nkv]) and err.item() == 1
    for t, slot in enumerate(slots.tolist()):
        if slot >= 0:
            k, v = cache[slot // page, 0, :, slot % page], cache[slot // page, 1, :, slot % page]
            assert close(k, want[t, nh:nh + nkv]) and torch.equal(v, heads[t, nh + nkv:])
    assert int((cache == 7.0).all(-1).sum()) >= 2 * nkv * (12 - 6)
