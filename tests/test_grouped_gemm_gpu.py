"""Products on CTA pairs with gated activations in their epilogues: the experts' products over a tile list, and a dense gate|up."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def act_of(g, u, kind, limit):
    if kind == "silu":
        return g * torch.sigmoid(g) * u
    if kind == "gelu_tanh":
        return torch.nn.functional.gelu(g, approximate="tanh") * u
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def close(got, want):
    # one rounding to bfloat16 behind 32-bit sums; products of a tile's few results of ordinary size
    return float((got.double() - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())


def close_after_two(got, g, u, kind, limit):
    """Gate and up each rounded to bfloat16 (2^-8 of the number) in front of the activation, its result rounded once more: every
    result lies between the least and the greatest of what the activation makes of such gates and ups, give or take a rounding
    and, for the 32-bit sums and what lies between the ends, 2^-12 of the largest."""
    ends = torch.stack([act_of(g * (1 + i * 2.0 ** -8), u * (1 + j * 2.0 ** -8), kind, limit) for i in (-1, 0, 1) for j in (-1, 0, 1)])
    lo, hi = ends.amin(0), ends.amax(0)
    slack = 2.0 ** -12 * float(ends.abs().max())
    got = got.double()
    return bool((got >= lo - 2.0 ** -8 * lo.abs() - slack).all() and (got <= hi + 2.0 ** -8 * hi.abs() + slack).all())


@pytest.mark.parametrize("tile_rows", [128, 256])
@pytest.mark.parametrize("F,K", [(8, 8), (136, 200), (20, 72), (512, 2048), (2048, 64)])
@pytest.mark.parametrize("kind", ["silu", "gelu_tanh", "clamped_swish", None])
def test_experts_products(F, K, tile_rows, kind):
    """Experts of no, one, a few, exactly a tile's and more places; rows of a matrix that end inside a tile; K that ends inside a
    box.  Places of no expert are not written."""
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(F + K)
    counts = [0, 1, 16, 17, 256, 270, 33, 0, 512, 100]
    E, P = len(counts), sum(counts)
    ids = torch.repeat_interleave(torch.arange(E), torch.tensor(counts)).to(torch.int32)
    ids = ids[torch.randperm(P, generator=torch.Generator().manual_seed(K))].view(-1, 1).to(DEV)
    x = torch.randn(P, K, device=DEV, generator=g).bfloat16()
    rows = 2 * F if kind else F
    w = (torch.randn(E, rows, K, device=DEV, generator=g) / K ** 0.5).bfloat16()
    pair, pos, tiles = ops.moe_align(ids, E, tile_rows)
    got = ops.moe_grouped_gemm(x, pair, 1, w, tiles, P, bool(kind), tile_rows, act=kind or "silu", limit=0.7)
    ops.tc_gemm_check()
    assert got.shape == (P, F)
    for e in range(E):
        at = (ids[:, 0] == e).nonzero()[:, 0]
        if not len(at):
            continue
        y = x[at].double() @ w[e].double().T
        rows_of = got[pos[at].long()]
        if kind and F % 8:                  # not in the product's kernel: the activation reads the rounded product
            assert close_after_two(rows_of, y[:, :F], y[:, F:], kind, 0.7), e
        else:
            assert close(rows_of, act_of(y[:, :F], y[:, F:], kind, 0.7) if kind else y), e


@pytest.mark.parametrize("M,I,K", [(1024, 200, 64), (1057, 1016, 136), (2048, 8192, 256), (1100, 8, 8)])
@pytest.mark.parametrize("kind", ["gelu_tanh", "clamped_swish", "silu"])
def test_gated_product(M, I, K, kind):
    from railgun_b200 import ops
    g = torch.Generator(device=DEV).manual_seed(M + I)
    x = torch.randn(M, K, device=DEV, generator=g).bfloat16()
    w = (torch.randn(2 * I, K, device=DEV, generator=g) / K ** 0.5).bfloat16()
    assert ops.tc_gemm_gated_ok(x, w)
    got = ops.tc_gemm_gated(x, w, kind, 0.7)
    ops.tc_gemm_check()
    y = x.double() @ w.double().T
    assert close(got, act_of(y[:, :I], y[:, I:], kind, 0.7))
    assert torch.equal(got, ops.tc_gemm_gated(x, w, kind, 0.7))
