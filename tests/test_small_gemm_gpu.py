"""The 32-bit product of a few rows by a small matrix, at the edges of its 32 x 32 tiles and 32-wide steps, along and across
16-byte boundaries, against 64 bits."""
import pytest
import torch

from test_kernels_gpu import DEV, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (1, 500, 96), (67, 160, 96), (32, 32, 32), (33, 33, 33), (31, 65, 511), (128, 1024, 512),
                                   (17, 96, 256), (2, 7, 4)])
def test_against_64_bits(M, N, K):
    from railgun_b200 import ops
    g = torch.Generator().manual_seed(M + N + K)
    x, w = torch.randn(M, K, generator=g).to(DEV), torch.randn(N, K, generator=g).to(DEV)
    ref = x.double() @ w.double().T
    y = ops.small_gemm_f32(x, w)
    # chains of eight products and of at most sixteen of their sums: some 25 x 2^-24 of the largest, 1.5e-6
    assert y.dtype == torch.float32 and rel_err(y, ref) < 2e-6
    assert torch.equal(ops.linear(x, w), y)
    if K <= 96:
        assert torch.equal(ops.small_gemm_f32(x[M // 2:M // 2 + 1], w)[0], y[M // 2])  # a row on its own
    wide = torch.full((M, K + 3), float("nan"), device=DEV)                            # rows off 16-byte boundaries
    wide[:, 1:K + 1] = x
    assert torch.equal(ops.small_gemm_f32(wide[:, 1:K + 1], w), y)


def test_what_it_refuses():
    from railgun_b200 import ops
    x, w = torch.zeros(4, 64, device=DEV), torch.zeros(8, 64, device=DEV)
    assert ops.small_gemm_f32_ok(x, w) and not ops.small_gemm_f32_ok(x.bfloat16(), w.bfloat16())
    assert not ops.small_gemm_f32_ok(x.t(), w) and not ops.small_gemm_f32_ok(x[:0], w)
    assert not ops.small_gemm_f32_ok(torch.zeros(8, 256, device=DEV), torch.zeros(64, 256, device=DEV))    # the library's is faster
    with pytest.raises(ops.KernelError):
        ops.small_gemm_f32(x, torch.zeros(8, 63, device=DEV))


@pytest.mark.parametrize("M,N,K,own", [(16, 64, 96, True), (16, 64, 97, False), (1, 8192, 128, False), (1, 8192, 96, True),
                                       (1, 8193, 96, False), (17, 64, 97, True),
                                       (17, 64, 448, True), (30, 64, 449, False), (31, 64, 512, True), (31, 64, 513, False),
                                       (32, 4736, 64, True), (32, 4737, 64, False), (33, 3000, 64, False), (256, 592, 64, False),
                                       (256, 576, 64, True), (257, 8, 64, False)])
def test_the_rules_edges(M, N, K, own):
    from railgun_b200 import ops
    assert ops.small_gemm_f32_ok(torch.zeros(M, K, device=DEV), torch.zeros(N, K, device=DEV)) == own


def test_what_stays_the_librarys():
    """A matrix elsewhere is refused as before; derivatives and maps go through the product as before."""
    from railgun_b200 import ops
    x, w = torch.randn(20, 64, device=DEV), torch.randn(8, 64, device=DEV)
    y = x @ w.t()
    with pytest.raises(RuntimeError):
        ops.linear(x, w.cpu())
    xg = x.clone().requires_grad_()
    ops.linear(xg, w).sum().backward()
    assert torch.allclose(xg.grad, w.sum(0).expand_as(x), atol=1e-5)
    wp = torch.nn.Parameter(w.clone())
    ops.linear(x, wp).sum().backward()
    assert torch.allclose(wp.grad, x.sum(0).expand_as(w), atol=1e-4)
    with torch.no_grad():
        assert ops.small_gemm_f32_ok(x, wp)
    value, moved = torch.func.jvp(lambda a: ops.linear(a, w), (x,), (torch.ones_like(x),))
    assert torch.allclose(value, y, atol=1e-4) and torch.allclose(moved, w.sum(1).expand(20, 8), atol=1e-4)
    maps = torch.vmap(lambda m: ops.linear(x, m))(torch.stack([w, 2 * w]))
    assert torch.allclose(maps, torch.stack([y, 2 * y]), atol=1e-4)


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (67, 160, 96), (33, 33, 33), (17, 96, 256), (31, 65, 255), (2, 7, 4), (256, 40, 130)])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows_that_the_kernel_makes(M, N, K, shift):
    """The norm of a residual with and without something pending in front of the product, SiLU-mul behind it; on and off 16-byte
    boundaries; the first row of blocks leaves the sum."""
    from railgun_b200 import ops
    g = torch.Generator().manual_seed(M + N + K)
    new = lambda *shape: torch.randn(shape[0] * shape[1] + shift, generator=g).to(DEV)[shift:].view(*shape)
    x, p, w = new(M, K), new(M, K), new(N, K)
    norm = (torch.rand(K, generator=g) + 0.5).to(DEV)
    for pending in (p, None):
        total = x if pending is None else x + pending
        unit = total.double() / (total.double().pow(2).mean(1, keepdim=True) + 1e-5).sqrt() * norm.double()
        h = ops.fresh_norm(x, pending, norm, 1e-5, w)
        if not ops.small_gemm_f32_ok(torch.empty(M, K, device=DEV), w):
            assert h is None                                             # the small product's rule
            continue
        y = ops.linear(h, w)
        # as above; the root mean square and its two products are four more roundings
        assert rel_err(y, unit @ w.double().T) < 3e-6 and torch.equal(h.new, total)
        assert (h.new is x) == (pending is None)
        if N % 2 == 0:
            # the same product, the same activation: silu's error is some 4 x 2^-24 of it
            gate, up = y[:, :N // 2].double(), y[:, N // 2:].double()
            assert rel_err(ops.gated_linear(h, w), torch.nn.functional.silu(gate) * up) < 5e-7
    if N % 2 == 0 and ops.gated_linear_ok(x, w):
        gate, up = (x.double() @ w.double().T).chunk(2, dim=1)
        # two products' errors (2e-6 each, above), the gate's by silu's slope of at most 1.1
        assert rel_err(ops.gated_linear(x, w), torch.nn.functional.silu(gate) * up) < 6e-6


def test_what_makes_no_rows():
    from railgun_b200 import ops
    x, w, n = torch.zeros(40, 64, device=DEV), torch.zeros(8, 64, device=DEV), torch.ones(64, device=DEV)
    assert ops.fresh_norm(x, None, n, 1e-5, w) is not None
    assert ops.fresh_norm(x, x.bfloat16(), n, 1e-5, w) is None and ops.fresh_norm(x, None, n, 1e-5, None) is None
    assert ops.fresh_norm(x, None, n, 1e-5, torch.zeros(8, 65, device=DEV)) is None
    wide = torch.zeros(40, 288, device=DEV)
    assert ops.fresh_norm(wide, None, torch.ones(288, device=DEV), 1e-5, torch.zeros(8, 288, device=DEV)) is None
    assert ops.gated_linear_ok(x, w) and not ops.gated_linear_ok(x, w[:7]) and not ops.gated_linear_ok(x[:, :63], w)
    assert not ops.gated_linear_ok(x.t(), w) and not ops.gated_linear_ok(wide, torch.zeros(8, 288, device=DEV))
    grown = torch.zeros(8, 64, device=DEV, requires_grad=True)
    assert ops.fresh_norm(x, None, n, 1e-5, grown) is None
