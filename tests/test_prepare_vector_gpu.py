"""The per-token kernels in front of attention and retention that take several numbers at a time, against the forms that take
one: the same rows behind a pitch that rules the wide form out.  Sizes at the edges of the rule, rotations that end inside a
head, both layouts, biases, values of another size than keys, tokens without a slot."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def odd_pitch(x):
    """The same matrix as a view of rows an odd number of elements further apart."""
    wide = torch.zeros(x.shape[0], x.shape[1] + 1 + x.shape[1] % 2, dtype=x.dtype, device=x.device)
    wide = wide[:, :x.shape[1]]
    wide.copy_(x)
    assert wide.stride(0) % 2
    return wide


def same(a, b):
    # 32-bit: a root mean square added up in another order (1e-7 each); bfloat16: one unit where that tips a rounding
    tol = 2e-6 if a.dtype == torch.float32 else 2.0 ** -7
    return float((a.double() - b.double()).abs().max()) <= tol * float(b.double().abs().max())


@pytest.mark.parametrize("types", [("float32", "float32"), ("bfloat16", "bfloat16"), ("float32", "bfloat16")])
@pytest.mark.parametrize("H,G,d,dv,D,dims", [(16, 2, 128, 128, 128, 64), (3, 3, 24, 40, 48, 16), (2, 1, 4, 8, 16, 0),
                                             (8, 2, 64, 64, 64, 64), (20, 4, 96, 32, 96, 8), (1, 1, 128, 4, 128, 128)])
def test_attention_prepare(H, G, d, dv, D, dims, types):
    from railgun_b200 import ops
    from railgun_b200.parts.latent_attention import rotary_frequencies
    a, o = (getattr(torch, t) for t in types)
    g = torch.Generator(device=DEV).manual_seed(H * d + dims)
    T, page = 11, 4
    n = (H + G) * d + G * dv
    x = torch.randn(T, n, device=DEV, generator=g).to(a)
    freq = rotary_frequencies(dims, 1e4).to(DEV) if dims else torch.zeros(1, dtype=torch.float64, device=DEV)
    pos = torch.tensor([0, 1, 5, 6, 7, 13, 70000, 62, 63, 3, 2], dtype=torch.int32, device=DEV)
    slots = torch.tensor([5, 4, -1, 7, 0, 1, 2, 11, 3, 8, -1], dtype=torch.int32, device=DEV)
    norm = [0.5 + torch.rand(d, device=DEV, generator=g) for _ in range(2)]
    factor = torch.rand(H, device=DEV, generator=g)
    bias = torch.randn(n, device=DEV, generator=g)
    for interleaved, normed, more in ((True, True, dict(factor=factor)), (False, False, dict(factor=None, bias=bias)),
                                      (False, True, dict(factor=None, temp_coef=0.3, temp_every=7))):
        got = []
        for rows in (x, odd_pitch(x)):
            cache = torch.full((3, 2, G, page, D), 7.0, dtype=o, device=DEV)
            q = ops.attention_prepare(rows, cache, norm[0] if normed else None, norm[1] if normed else None, 1e-5, freq, dims,
                                      interleaved, pos, slots, more["factor"], H, G, d, dv, D, out_dtype=o,
                                      **{k: v for k, v in more.items() if k != "factor"})
            got.append((q, cache))
        assert same(got[0][0], got[1][0]) and same(got[0][1], got[1][1])
        assert torch.equal(got[0][1] == 7.0, got[1][1] == 7.0)                # the same places written
        q, _ = got[0]
        assert ops.attention_prepare(x, None, None, None, 1e-5, freq, dims, interleaved, pos, None, None, H, G, d, dv, D,
                                     out_dtype=o).shape == q.shape             # no cache: q alone


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,d,dims,dv", [(16, 128, 128, 128), (3, 24, 16, 8), (2, 8, 0, 16), (8, 64, 48, 64), (1, 32, 32, 40)])
@pytest.mark.parametrize("silu", [False, True])
def test_retention_prepare(H, d, dims, dv, dtype, silu):
    from railgun_b200 import ops
    from railgun_b200.parts.latent_attention import rotary_frequencies
    g = torch.Generator(device=DEV).manual_seed(H + d + dims)
    T = 7
    x = torch.randn(T, 2 * H * d + H * dv + 8, device=DEV, generator=g).to(dtype)
    freq = rotary_frequencies(dims, 1e4).to(DEV) if dims else torch.zeros(1, dtype=torch.float64, device=DEV)
    pos = torch.tensor([0, 1, 2, 500, 70000, 3, 8191], dtype=torch.int32, device=DEV)
    more = dict(silu=True, v_off=2 * H * d, dv=dv) if silu else {}
    wide, plain = (ops.retention_prepare(rows, 0, H * d, freq, dims, pos, H, d, d ** -0.5, **more) for rows in (x, odd_pitch(x)))
    for a, b in zip(wide, plain):
        assert same(a, b)
