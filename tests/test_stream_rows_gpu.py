"""The streaming tcgen05 product at 65 to 256 rows (a step that holds short prompts), with the neighbouring operations in its
epilogues, where it can go wrong: token tiles of 64, 128 and 256, chunks of 64 of them, splits of K, ragged rows of W."""
import pytest
import torch

from test_kernels_gpu import DEV, rel_err

pytestmark = pytest.mark.gpu
F32 = 2e-5                  # 32-bit accumulation over all of K (as the tests of up to 64 rows)
BF16 = 1e-2                 # one rounding to bfloat16, 2^-9, on values of any size


def rows_of(M, H, K, splits, seed, eps=1e-3):
    from railgun_b200 import ops
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(H, K, generator=g) / K ** 0.5).to(torch.bfloat16).to(DEV)
    resid0 = (torch.randn(M, H, generator=g) * 3).to(DEV)
    nw = (torch.rand(H, generator=g) + 0.5).to(DEV)
    resid = resid0.clone()
    rows = ops.tc_stream_gemm_residual(x, w, resid, nw, eps, splits=splits)
    ops.tc_gemm_check()
    ref = resid0.double() + x.double() @ w.double().T
    return g, x, w, resid0, nw, resid, rows, ref, ref * torch.rsqrt((ref ** 2).mean(1, keepdim=True) + eps) * nw.double()


@pytest.mark.parametrize("splits", [0, 1, 2, 8])
@pytest.mark.parametrize("M,H,K", [(65, 200, 520), (128, 2048, 2048), (129, 1000, 1096), (191, 2048, 8192), (256, 3080, 520)])
def test_residual_then_scaled(M, H, K, splits):
    from railgun_b200 import ops
    g, x, w, resid0, nw, resid, rows, ref, normed = rows_of(M, H, K, splits, M + H + K)
    assert rel_err(resid, ref) < F32
    assert torch.equal(rows.scaled, (resid * nw).to(torch.bfloat16))           # one rounding, of the 32-bit product
    assert rel_err(rows.partials[:rows.blocks, :M].double().sum(0), (resid.double() ** 2).sum(1)) < 1e-6
    # a row does not depend on its batch: alone, or (where the launcher picks the splits) last of any other batch above 64 rows
    first = M - 1 if splits else M - 65
    again = resid0[first:].clone()
    ops.tc_stream_gemm_residual(x[first:].contiguous(), w, again, nw, 1e-3, splits=splits)
    assert torch.equal(again[-1], resid[M - 1])
    for N2, silu in ((136, False), (1008, True), (3072, False)):
        w2 = (torch.randn(N2, H, generator=g) / H ** 0.5).to(torch.bfloat16).to(DEV)
        assert ops.tc_stream_scaled_ok(rows, w2) == (M < 256)
        y = ops.tc_stream_gemm(rows, w2, silu_mul=silu, splits=splits if -(-H // 64) >= splits else 0, max_rows=256)
        ops.tc_gemm_check()
        z = normed @ w2.double().T
        if silu:
            z = z.view(M, N2 // 16, 2, 8)
            z = (z[:, :, 0] / (1 + torch.exp(-z[:, :, 0])) * z[:, :, 1]).reshape(M, N2 // 2)
        assert rel_err(y, z) < BF16
        if not silu and M < 256:
            assert rel_err(ops.linear(rows, w2), z) < BF16


@pytest.mark.parametrize("splits", [2, 4, 8])
@pytest.mark.parametrize("M,boxes,rest", [(17, 3, 0), (33, 16, 0), (64, 32, 0), (63, 32, 8), (19, 40, 24)])
def test_up_to_64_rows_in_splits(M, boxes, rest, splits):
    """Shares of K up to, at and above 32 boxes of 64 a split, where the number of stages changes; M tokens in `splits` shares."""
    from railgun_b200 import ops
    H, K = 200, 64 * boxes * splits + rest
    _, x, w, resid0, nw, resid, rows, ref, _ = rows_of(M, H, K, splits, M + K)
    assert rel_err(resid, ref) < F32
    assert torch.equal(rows.scaled, (resid * nw).to(torch.bfloat16))
    for first, n in ((M - 1, splits), (M - 2, 0)):
        again, whole = resid0[first:].clone(), resid
        if n == 0:
            whole = resid0.clone()
            ops.tc_stream_gemm_residual(x, w, whole, nw, 1e-3)
        ops.tc_stream_gemm_residual(x[first:].contiguous(), w, again, nw, 1e-3, splits=n)
        assert torch.equal(again[-1], whole[M - 1])


@pytest.mark.parametrize("M", [17, 65, 130, 256])
@pytest.mark.parametrize("nh,nkv,d,K,page", [(4, 2, 64, 256, 16), (6, 3, 48, 136, 8), (24, 8, 128, 1024, 32)])
def test_rotation_and_cache_write(M, nh, nkv, d, K, page):
    """Positions may repeat (portions of several requests); a token without a slot is not stored."""
    from railgun_b200 import ops
    from railgun_b200.parts.rope import rope_table
    g, *_, rows, _, _ = rows_of(M, K, 64, 0, M + d)
    N, NP, max_pos = (nh + 2 * nkv) * d, 40, 300
    table = rope_table(d, 500000.0, None, max_pos).to(DEV)
    w = (torch.randn(N, K, generator=g) / K ** 0.5).to(torch.bfloat16).to(DEV)
    positions = torch.randint(0, max_pos, (M,), generator=g, dtype=torch.int32).to(DEV)
    slots = torch.randperm(NP * page, generator=g)[:M].to(torch.int32)
    slots[1] = -1
    slots = slots.to(DEV)
    for x in (torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV), rows):
        assert ops.tc_stream_rope_ok(x, w, d, 256) == (x is not rows or M < 256)
        kv_f = torch.zeros(NP, 2, nkv, page, d, dtype=torch.bfloat16, device=DEV)
        kv_u = torch.zeros_like(kv_f)
        fused = ops.tc_stream_gemm_rope_cache(x, w, table, positions, slots, kv_f, nh, nkv, d)
        ops.tc_gemm_check()
        plain = ops.tc_stream_gemm(x, w, max_rows=256, check=True)
        ops.rope_cache_write(plain, table, positions, slots, kv_u, nh, nkv, d, page, paired8=True)
        # the unfused route rounds the projection to bfloat16 before it rotates: equal within that rounding
        assert rel_err(fused[:, :nh * d], plain[:, :nh * d].double()) < BF16 and rel_err(kv_f, kv_u.double()) < BF16
        assert torch.equal(kv_f != 0, kv_u != 0)


def test_a_position_outside_the_table_is_flagged_and_too_many_rows_are_refused():
    from railgun_b200 import ops
    from railgun_b200.parts.rope import rope_table
    table = rope_table(64, 1e4, None, 8).to(DEV)
    x, w = torch.ones(70, 64, dtype=torch.bfloat16, device=DEV), torch.ones(192, 64, dtype=torch.bfloat16, device=DEV)
    positions = torch.full((70,), 3, dtype=torch.int32, device=DEV)
    flag = torch.zeros(1, dtype=torch.int32, device=DEV)
    ops.tc_stream_gemm_rope_cache(x, w, table, positions, None, None, 1, 1, 64, flag)
    assert int(flag) == 0
    positions[69] = 8
    ops.tc_stream_gemm_rope_cache(x, w, table, positions, None, None, 1, 1, 64, flag)
    assert int(flag) == 1
    with pytest.raises(ops.KernelError):
        ops.tc_stream_gemm(torch.zeros(257, 64, dtype=torch.bfloat16, device=DEV), w, max_rows=1000)


def test_which_steps_take_it():
    """Decode batches up to 64 rows (they are replayed from graphs); steps with prompts up to 255 of a small width."""
    from types import SimpleNamespace as Batch
    from railgun_b200 import ops
    assert ops.tc_stream_rows(Batch(decode_only=True), 2048) == ops.tc_stream_rows(None, 2048) == 64
    assert [ops.tc_stream_rows(Batch(decode_only=False), w) for w in (64, 2048, 3072, 4096, 16384)] == [255, 255, 170, 128, 64]


@pytest.mark.parametrize("rows", [40, 41, 64, 65])
@pytest.mark.parametrize("N,K", [(37888, 64), (37889, 64), (50000, 264)])
def test_logits_of_decode_batches(rows, N, K):
    """Both sides of the rule's edges, against 64 bits."""
    from railgun_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(rows + N)
    x = torch.randn(rows, K, device="cuda", generator=g).bfloat16()
    w = torch.randn(N, K, device="cuda", generator=g).bfloat16()
    y = ops.linear(x, w, out_dtype=torch.float32)
    ops.tc_gemm_check()
    want = x.double() @ w.double().T
    assert y.dtype == torch.float32 and y.shape == (rows, N)
    assert float((y.double() - want).abs().max() / want.abs().max()) < K * 2.0 ** -24 + 1e-6


@pytest.mark.parametrize("M", [65, 96, 97, 128, 129, 176, 177, 255, 256])
def test_parts_of_the_tokens(M):
    """Few tiles of W above 64 rows: two parts of the tokens, of up to 64 and 128 each; a matrix of more tiles than half of the
    SMs takes them whole.  Residual, norm and partial sums against 64 bits."""
    from railgun_b200 import ops
    for N, K in ((256, 264), (2048, 256), (3072, 320)):
        g = torch.Generator(device="cuda").manual_seed(M + N)
        x = torch.randn(M, K, device="cuda", generator=g).bfloat16()
        w = torch.randn(N, K, device="cuda", generator=g).bfloat16()
        r, nw = torch.randn(M, N, device="cuda", generator=g), torch.rand(N, device="cuda", generator=g) + 0.5
        want = r.double() + x.double() @ w.double().T
        h = ops.tc_stream_gemm_residual(x, w, r, nw, 1e-5)
        ops.tc_gemm_check()
        err = lambda a, b: float((a.double() - b).abs().max() / b.abs().max())
        assert err(r, want) < K * 2.0 ** -24 + 1e-6 and err(h.scaled, want * nw.double()) < 2.0 ** -8
        assert err(h.partials[:h.blocks, :M].double().sum(0), want.pow(2).sum(1)) < 1e-5
