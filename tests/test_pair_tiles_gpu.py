"""Products on CTA pairs with tiles 224 and 192 columns wide, at the edges of the tiles, against 64 bits; and the choice
between them."""
import pytest
import torch

from test_kernels_gpu import DEV, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", ["256x224", "256x192"])
@pytest.mark.parametrize("M,N,K", [(1, 16, 8), (257, 448, 72), (256, 208, 512), (1056, 2048, 1024), (300, 4000, 136)])
def test_against_64_bits(tile, M, N, K):
    from railgun_b200 import ops
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(N, K, generator=g) / K ** 0.5).to(torch.bfloat16).to(DEV)
    ref = x.double() @ w.double().T
    assert rel_err(ops.tc_gemm(x, w, out_dtype=torch.float32, tile=tile, check=True), ref) < 2e-5     # 32-bit accumulation
    assert rel_err(ops.tc_gemm(x, w, tile=tile, check=True), ref) < 1e-2                              # one rounding
    gu = ref.view(M, N // 16, 2, 8)
    act = (gu[:, :, 0] / (1 + torch.exp(-gu[:, :, 0])) * gu[:, :, 1]).reshape(M, N // 2)
    assert rel_err(ops.tc_gemm(x, w, silu_mul=True, tile=tile, check=True), act) < 1e-2


def test_the_choice(monkeypatch):
    from railgun_b200 import ops
    monkeypatch.setattr(ops, "_sm_pairs", lambda i: 74)
    pick = lambda M, N: ops.tc_pair_tile(M, N, torch.device(DEV))  # noqa: E731
    assert pick(2048, 16384) == pick(2048, 28672) == pick(74 * 256, 256) == "256x256"     # full rounds, or nearly
    assert pick(1056, 16384) == pick(1701, 16384) == "256x224"                            # five rounds of four and a third
    assert all(pick(M, N) in ops.TC_TILES for M in (1, 255, 1024, 5000) for N in (16, 224, 3000, 28672))
