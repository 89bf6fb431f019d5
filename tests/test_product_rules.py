"""Which kernels take a product, and how attention is divided into blocks: rules on sizes."""
from ctypes import c_int

import pytest


@pytest.mark.parametrize("rows,width,k,one", [
    # measured on both sides (one kernel against the product with the activation kernel behind it)
    (257, 1024, 1024, True), (448, 2048, 1024, True), (384, 6144, 1024, True), (300, 2816, 2048, True), (320, 4096, 2048, True),
    (320, 1024, 4096, False), (257, 4096, 4096, False), (320, 4096, 8192, False), (448, 2048, 8192, False), (257, 6144, 8192, False),
    (320, 6912, 8192, True), (448, 5120, 8192, True), (384, 6144, 4096, True),
    (257, 8192, 1024, False), (448, 8192, 4096, False), (384, 10240, 1024, False), (257, 10240, 2048, False), (448, 12288, 4096, True),
    (448, 24576, 1024, False), (320, 16384, 2048, True), (300, 24576, 4096, True),
    # whole tiles, and few rows
    (256, 24576, 4096, True), (512, 4096, 8192, False), (511, 1024, 4096, False), (2048, 4096, 1024, True), (513, 4096, 8192, True), (128, 24576, 4096, False), (255, 24576, 4096, False),
    (1, 24576, 4096, False)])
def test_gate_up_products_with_their_activation_in_one_kernel(rows, width, k, one):
    from lumenllm_b200.ops.gemm import gate_up_in_one
    assert gate_up_in_one(rows, width, k) == one


@pytest.mark.parametrize("width,k", [(512, 4096), (4096, 8192), (5120, 8192), (10240, 2048), (24576, 4096), (16384, 1024)])
def test_a_captured_prompts_rows_take_the_way_of_the_eager_ones(width, k):
    """A captured step rounds its rows up to a multiple of 32 and must give the bits of the eager one."""
    from lumenllm_b200.ops.gemm import gate_up_in_one
    for rows in range(257, 700):
        assert gate_up_in_one(rows, width, k) == gate_up_in_one((rows + 31) // 32 * 32, width, k), rows


def test_heads_a_block_of_float32_prompt_attention():
    """Steps of few tokens keep the SMs busy with a head a block; long prompts share the staged keys among four, of one group."""
    from lumenllm_b200.ops.native import int_fn
    heads = lambda *a: int_fn("attn_generic", "lumen_attn_prompt_heads", [c_int] * 3)(*a)
    assert [heads(n, 16, 4) for n in (8, 16, 48, 64, 128, 192, 300, 2000)] == [1, 1, 1, 2, 2, 4, 4, 4]
    assert [heads(n, 8, 2) for n in (8, 100, 128, 200, 300)] == [1, 1, 2, 2, 4]
    for n in (8, 300, 5000):
        for nq, nkv in ((16, 16), (12, 6), (6, 2), (64, 8)):
            assert nq // nkv % heads(n, nq, nkv) == 0


def test_scratch_of_the_float32_product_is_bounded():
    """Cut activations are six bytes a number, and at most 256 MB at a time."""
    from ctypes import c_longlong
    from lumenllm_b200.ops.native import int_fn
    size = int_fn("gemm_f32_tc", "lumen_gemm_f32_tc_scratch", [c_int, c_int])
    size.restype = c_longlong
    assert size(1, 8192) == size(32, 8192) == 0
    for m, k in ((33, 1024), (300, 8192), (700, 5120), (2048, 5120), (1400, 16384), (2800, 16384), (8192, 25600), (100000, 2048), (161, 300000)):
        assert 0 < size(m, k) <= max(256 << 20, 160 * (k + 63) * 6)
        assert size(m, k) >= min(6 * m * k, (256 << 20) - 160 * (k + 63) * 6)
