"""The products of 17 to 64 tokens (csrc/gemm_mid.cu) against float32: every epilogue, edges of the token range, widths that
do not fill the last tile, one to eight parts of k, and the norm that one product leaves to the next."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from paged_llm_b200.kernels.ops import CudaOps
    ops = CudaOps("cuda")
    ops.set_compute_dtype(torch.bfloat16)
    ops.mid_widths, ops.mid_width_per_token, ops.mid_features = (0, 1 << 30), 0, 1 << 30      # the kernel at any size
    return ops


def randn(*shape, seed, std=1.0, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * std).to(dtype)


def close(got, want, K, rounded=True):
    """Sums of K products of size `std` in float32 (error sqrt(K) 2^-24 of the sum's size, 64 times that allowed for the
    tensor core's coarser additions), rounded to bfloat16 where `rounded` (2^-9 of the value)."""
    torch.testing.assert_close(got.float(), want, atol=float(want.abs().mean()) * K ** 0.5 * 2 ** -18,
                               rtol=2 ** -8 if rounded else 1e-5)


@pytest.mark.parametrize("M", [17, 31, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(2560, 2048), (132, 64), (4, 192), (4100, 320), (508, 3520), (38400, 256)])
def test_plain(ops, M, N, K):
    h, w = randn(M, K, seed=1), randn(N, K, seed=2, std=0.02)
    want = h.float() @ w.float().T
    before = ops.launches
    close(ops.linear(h, w, out_float32=True), want, K, rounded=False)
    close(ops.linear(h, w), want, K)
    assert ops.launches == before + 2, "both are this package's kernel"
    one = ops.linear(h[:17].contiguous(), w, out_float32=True)
    assert torch.equal(one, ops.linear(h, w, out_float32=True)[:17]), "a token's result does not depend on the batch"


@pytest.mark.parametrize("M", [17, 48, 64])
@pytest.mark.parametrize("I,K", [(5632, 2048), (70, 128), (8192, 64), (2, 256)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_gated(ops, M, I, K, act):
    h, w = randn(M, K, seed=3), randn(2 * I, K, seed=4, std=0.05)
    gate, up = (h.float() @ w.float().T).to(torch.bfloat16).float().chunk(2, 1)
    a = torch.nn.functional.silu(gate) if act == "silu" else torch.nn.functional.gelu(gate, approximate="tanh")
    got = ops.gated_act_linear(h, w, act).float()
    # gate and up are rounded to bfloat16 (2^-9 each) before they are multiplied and the product is rounded again
    torch.testing.assert_close(got, a * up, atol=2 ** -7 * float((a * up).abs().mean()) + 1e-5, rtol=2 ** -6)


@pytest.mark.parametrize("wdtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("M", [17, 40, 64])
@pytest.mark.parametrize("N,K", [(2048, 5632), (128, 64), (384, 704)])
def test_add_and_the_norm_behind_it(ops, M, N, K, wdtype):
    from paged_llm_b200.kernels.ops import LazyNorm
    h, w, x = randn(M, K, seed=5), randn(N, K, seed=6, std=0.05), randn(M, N, seed=7, dtype=torch.float32)
    nw = randn(N, seed=8, std=0.1, dtype=torch.float32).add(1).to(wdtype)
    branch = h.float() @ w.float().T
    want = x + branch
    lazy = ops.linear_add_rms_norm(h, w, x, nw, 1e-5)
    assert isinstance(lazy, LazyNorm) and lazy.scaled is not None
    torch.testing.assert_close(x, want, atol=2 ** -8 * float(branch.abs().max()), rtol=1e-6)
    normed = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-5) * nw.float()
    torch.testing.assert_close(ops.materialize(lazy).float(), normed, atol=2 ** -8, rtol=2 ** -8)
    w2 = randn(260, N, seed=9, std=0.05)
    # the operand is rounded to bfloat16 (2^-9 of its size, N of them at random) before the product
    want2 = normed @ w2.float().T
    got2 = ops.linear(lazy, w2, out_float32=True)
    assert ((got2 - want2).norm() / want2.norm()).item() < 2 ** -8
    gate, up = want2.chunk(2, 1)
    got3 = ops.gated_act_linear(lazy, w2, "silu").float()
    want3 = torch.nn.functional.silu(gate) * up
    assert ((got3 - want3).norm() / want3.norm()).item() < 2 ** -6
    assert ops.kernel_timeouts() == 0


def shifted(t, by=1):
    """The same values at an address that is no multiple of 16 bytes."""
    buf = torch.empty(t.numel() + by, dtype=t.dtype, device=t.device)
    out = buf[by:].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 and out.is_contiguous()
    return out


@pytest.mark.parametrize("by", [1, 2])
@pytest.mark.parametrize("which", ["h", "w", "norm", "norm32", "stream"])
def test_operands_that_do_not_start_on_16_bytes(ops, which, by):
    """Views at odd offsets take the library's product, as they did before there was another."""
    M, N, K = 24, 256, 512
    h, w, x = randn(M, K, seed=5), randn(N, K, seed=6, std=0.05), randn(M, N, seed=7, dtype=torch.float32)
    nw = randn(N, seed=8, std=0.1, dtype=torch.float32).add(1)
    nw = nw if which == "norm32" else nw.to(torch.bfloat16)
    branch = (h.float() @ w.float().T)
    want = x + branch
    h, w, nw, x = (shifted(t, by) if which.startswith(name) else t for name, t in (("h", h), ("w", w), ("norm", nw), ("stream", x)))
    got = ops.materialize(ops.linear_add_rms_norm(h, w, x, nw, 1e-5)).float()
    torch.testing.assert_close(x, want, atol=2 ** -8 * float(branch.abs().max()), rtol=1e-6)
    normed = want * torch.rsqrt(want.square().mean(-1, keepdim=True) + 1e-5) * nw.float()
    torch.testing.assert_close(got, normed, atol=2 ** -6, rtol=2 ** -7)
    close(ops.linear(h, w), branch, K)
    gate, up = branch.to(torch.bfloat16).float().chunk(2, 1)
    act = torch.nn.functional.silu(gate) * up
    torch.testing.assert_close(ops.gated_act_linear(h, w).float(), act, atol=2 ** -7 * float(act.abs().mean()) + 1e-5, rtol=2 ** -6)
