"""Which 32-bit products go to this package's kernel by address: only those whose operands a kernel can read."""
import torch

from railgun_b200 import ops


def test_an_operand_on_the_host_is_no_operand():
    x, w = torch.zeros(4, 64), torch.zeros(8, 64)
    assert not ops.small_gemm_f32_ok(x, w)
    assert not ops.small_gemm_f32_ok(x.to("meta"), w.to("meta"))
