"""Which gate/up products of fewer than 2,048 tokens leave the library, decided on the host: points on both sides of the line,
each as it was measured."""

import types

import pytest
import torch

from paged_llm_b200.kernels.ops import CudaOps


def taken(tokens, K, I, activation="silu", dtype=torch.bfloat16, kinds=("silu", "moe"), h_at=0, w_at=0):
    ops = types.SimpleNamespace(num_sms=148, gemm_tc_for=set(kinds), gemm_tc_min_tokens=2048)
    ops._gemm_tc_ok = lambda h, w, kind: CudaOps._gemm_tc_ok(ops, h, w, kind)
    h = torch.empty(tokens * K + 8, dtype=dtype)[h_at:h_at + tokens * K].view(tokens, K)
    w = types.SimpleNamespace(dtype=dtype, is_contiguous=lambda: True, shape=(2 * I, K), data_ptr=lambda: 4096 + 2 * w_at)
    return CudaOps._gate_up_tc_ok(ops, h, w, I, activation)


@pytest.mark.parametrize("K,I,tokens", [
    (2048, 8192, 256), (2048, 8192, 512), (2048, 8192, 768), (2048, 8192, 832), (2048, 8192, 960), (2048, 8192, 1024), (2048, 5632, 1024),
    (2048, 5632, 2047), (512, 8192, 832), (1024, 14336, 832), (4096, 8192, 1024), (4096, 14336, 768), (3072, 11008, 1024)])
def test_where_the_kernel_is_the_faster_one(K, I, tokens):
    assert taken(tokens, K, I)
    assert not taken(tokens, K, I, activation="gelu_tanh") and not taken(tokens, K, I, dtype=torch.float32)
    assert not taken(tokens, K, I, kinds=("moe",))
    for odd in (1, 2, 4, 7):
        assert not taken(tokens, K, I, h_at=odd) and not taken(tokens, K, I, w_at=odd)


@pytest.mark.parametrize("K,I,tokens", [
    # a tile's start and end weigh more than the library's
    (64, 8192, 1036), (64, 14336, 832), (128, 11008, 640), (256, 8192, 832), (256, 14336, 1036), (448, 8192, 1024),
    # the library's main loop is the faster one
    (4160, 8192, 1024), (8192, 5632, 1036), (8192, 8192, 512),
    # just above a multiple of 256 tokens
    (2048, 8192, 828), (2048, 8192, 1036), (3072, 8192, 1085), (4096, 8192, 1110), (4096, 11008, 1036), (4096, 14336, 1036), (2048, 6912, 828),
    # tiles that leave much of a wave
    (2048, 5632, 256), (2048, 5632, 832), (2048, 5632, 960), (2048, 8192, 576), (4096, 14336, 832), (512, 5632, 960), (2048, 8192, 65)])
def test_where_the_library_is(K, I, tokens):
    assert not taken(tokens, K, I)


def test_from_2048_tokens_on_all_of_them():
    for K, I in ((64, 1024), (2048, 5632), (8192, 8192)):
        assert taken(2048, K, I) and taken(2049, K, I, activation="gelu_tanh")
