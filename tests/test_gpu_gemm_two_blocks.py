"""Stages of two k-blocks (csrc/gemm_tcgen05.cu, KB = 2: inner dimensions of whole k-blocks) against stages of one, which eight columns of zeros behind the
matrices bring: even and odd numbers of k-blocks, every tile width, edges of rows and columns.  The reference's order has no tolerance."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def product(f, a, b):
    out = torch.full((a.shape[0], b.shape[0]), 7.0, dtype=torch.bfloat16, device="cuda")
    f(a, b, out, a.shape[0], a.shape[1], b.shape[0])
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("inner", [128, 192, 448, 704, 832, 1536])
@pytest.mark.parametrize("rows,outer", [(1, 40), (9, 128), (16, 20000), (17, 1000), (33, 2304), (64, 4864), (65, 129), (200, 896)])
def test_same_bits_in_the_references_order(inner, rows, outer):
    from qwen_inference_engine_b200 import layers as L
    g = torch.Generator("cuda").manual_seed(inner + rows)
    a, b = (torch.randn(n, inner, generator=g, device="cuda").bfloat16() for n in (rows, outer))
    pad = torch.nn.functional.pad
    assert torch.equal(product(L.launch_matmul, a, b).view(torch.int16), product(L.launch_matmul, pad(a, (0, 8)), pad(b, (0, 8))).view(torch.int16))


@pytest.mark.parametrize("inner", [128, 960, 4864, 8960])
@pytest.mark.parametrize("rows,outer", [(1, 128), (8, 896), (40, 1536), (64, 896), (200, 256)])
def test_split_over_the_inner_dimension(inner, rows, outer):
    """splits of odd numbers of k-blocks; the sums' error in fp32 (a few 1e-6 of the values' scale) and one bf16 rounding (2^-9)"""
    from qwen_inference_engine_b200 import layers as L
    g = torch.Generator("cuda").manual_seed(inner + rows)
    a, b = (torch.randn(n, inner, generator=g, device="cuda").bfloat16() for n in (rows, outer))
    want = a.double() @ b.double().T
    assert ((product(L.launch_matmul_fast, a, b).double() - want).abs() <= want.abs() * 2.0 ** -8 + 1e-5 * inner ** 0.5).all()


@pytest.mark.parametrize("inner", [192, 320, 384, 448, 576])
@pytest.mark.parametrize("rows,outer", [(7, 130), (64, 896), (1000, 130), (16, 20001)])
def test_same_bits_around_the_rule_for_odd_numbers_of_k_blocks(inner, rows, outer):
    """3 and 5 k-blocks stay with stages of one, 6, 7 and 9 do not"""
    test_same_bits_in_the_references_order(inner, rows, outer)
