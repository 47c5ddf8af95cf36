"""Which products of 17 to 64 tokens leave the library, decided on the host."""

import types

import torch

from paged_llm_b200.kernels.ops import CudaOps


def test_only_operands_that_start_on_16_bytes():
    ops = types.SimpleNamespace(mid_tokens=64, mid_widths=(0, 4096), mid_width_per_token=0)
    h, w = torch.zeros(24 * 128 + 8, dtype=torch.bfloat16), torch.zeros(256 * 128 + 8, dtype=torch.bfloat16)

    def taken(h_at, w_at):
        return CudaOps._mid_ok(ops, h[h_at:h_at + 24 * 128].view(24, 128), w[w_at:w_at + 256 * 128].view(256, 128), 4, 128)

    assert taken(0, 0) and taken(8, 8)
    for odd in (1, 2, 4, 7):
        assert not taken(odd, 0) and not taken(0, odd)


def test_only_where_the_kernel_is_the_faster_one():
    """Widths and numbers of tokens on both sides of the line between the library's product and this package's."""
    ops = types.SimpleNamespace(mid_tokens=64, mid_widths=(640, 4096), mid_width_per_token=20)

    def taken(tokens, width):
        return CudaOps._mid_ok(ops, torch.zeros(tokens, 64, dtype=torch.bfloat16), torch.zeros(128, 64, dtype=torch.bfloat16), 4, width)

    for width, most in ((64, 0), (256, 0), (512, 0), (576, 0), (640, 32), (768, 38), (1024, 51), (1280, 64), (2048, 64), (4032, 64), (4096, 0)):
        got = [m for m in range(1, 80) if taken(m, width)]
        assert got == list(range(17, most + 1)), width
