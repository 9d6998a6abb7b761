"""Which products go to this package's kernels by address: only those whose operands a kernel can read."""
import pytest
import torch

from railgun_b200 import ops
from railgun_b200.parts.attention import PagedAttention
from railgun_b200.parts.mlp import SwiGLU
from railgun_b200.parts.norm import RMSNorm


def test_an_operand_on_the_host_is_no_operand():
    x, w = torch.zeros(4, 64), torch.zeros(8, 64)
    assert not ops.small_gemm_f32_ok(x, w)
    assert not ops.small_gemm_f32_ok(x.to("meta"), w.to("meta"))


@pytest.mark.parametrize("M,dtype", [(4, None), (48, torch.float32)])
def test_a_product_that_cannot_go_by_address_asks_for_no_address(M, dtype, monkeypatch):
    """With a bias, and logits of 41 to 64 rows: whether operands may go by address is asked before anything looks at one."""
    class Operand(torch.Tensor):
        is_cuda = True

        def data_ptr(self):
            raise AssertionError("an address")
    N = 24
    monkeypatch.setattr(ops, "_stream_head_pays", lambda N, sms: True)
    x, w, b = (torch.zeros(*s, dtype=torch.bfloat16).as_subclass(Operand) for s in ((M, 64), (N, 64), (N,)))
    monkeypatch.setattr(torch, "addmm", lambda *a: "library")
    monkeypatch.setattr(torch, "mm", lambda *a, **k: "library")
    monkeypatch.setattr(ops, "SKINNY_AUTO_ROWS", 16 if M == 4 else 0)
    assert ops.linear(x, w, dtype, bias=b if M == 4 else None) == "library"


def test_a_matrix_off_a_16_byte_boundary_is_not_for_16_byte_loads():
    x, flat = torch.zeros(4, 64).bfloat16(), torch.zeros(24 * 64 + 8).bfloat16()
    assert flat.data_ptr() % 16 == 0
    assert [ops.skinny_gemm_ok(x, flat[i:i + 24 * 64].view(24, 64)) for i in (0, 1, 4, 8)] == [True, False, False, True]


@pytest.mark.parametrize("what", ["plain", "norm", "gated"])
def test_32_bit_products_are_refused_while_tf32_is_on(what, monkeypatch):
    class Operand(torch.Tensor):
        is_cuda = True
    x, w = torch.zeros(4, 64).as_subclass(Operand), torch.zeros(8, 64)
    monkeypatch.setattr(ops, "gated_linear_ok", lambda x, w: True)
    monkeypatch.setattr(ops, "_small_rows", lambda *a: "launched")
    call = {"plain": lambda: ops.linear(x, w), "norm": lambda: ops.linear(ops.FreshNorm(torch.zeros(4, 64), None, torch.ones(64), 0.0), w),
            "gated": lambda: ops.gated_linear(x, w)}[what]
    monkeypatch.setattr(torch.backends.cuda.matmul, "allow_tf32", True)
    with pytest.raises(ops.KernelError, match="TF32"):
        call()


def test_a_norm_that_its_product_computes_takes_no_bias():
    fresh = ops.FreshNorm(torch.zeros(4, 64), None, torch.ones(64), 0.0)
    with pytest.raises(ops.KernelError, match="bias"):
        ops.linear(fresh, torch.zeros(8, 64), bias=torch.zeros(8))


@pytest.mark.parametrize("M,N,pays", [
    (1024, 16384, True), (1057, 16384, False), (1280, 16384, True), (2048, 16384, True), (1024, 28672, True), (1057, 28672, False),
    (1024, 4096, False), (1500, 4096, False), (2048, 4096, False), (3000, 4096, True), (4096, 4096, True), (1024, 2048, False),
    (4096, 2048, False), (1057, 8192, False), (1500, 8192, True), (2048, 8192, True)])
def test_which_gated_products_run_with_their_activation_inside(M, N, pays):
    """On both sides of the lines, on 74 pairs."""
    assert ops.tc_gemm_gated_pays(M, N, 74) == pays


@pytest.mark.parametrize("N,pays", [(128256, True), (94720, False), (94724, True), (50000, False), (37889, True), (37888, False), (32769, False)])
def test_which_logits_are_streamed(N, pays):
    assert ops._stream_head_pays(N, 148) == pays


@pytest.mark.parametrize("base,own,asked", [(RMSNorm, "add_norm", "plain_rms"), (PagedAttention, "forward", "first_matrix"),
                                            (SwiGLU, "forward", "first_matrix")])
def test_a_part_that_does_it_its_own_way_is_given_rows(base, own, asked):
    """A norm moves into the product that reads it only past the two classes' own code."""
    part = base.__new__(base)
    part.groups, part.w_qkv, part.w_gate_up = 1, "matrix", "matrix"
    assert getattr(part, asked)
    other = type("Other", (base,), {own: lambda self, *a, **k: None})
    part = other.__new__(other)
    part.groups, part.w_qkv, part.w_gate_up = 1, "matrix", "matrix"
    assert not getattr(part, asked)
