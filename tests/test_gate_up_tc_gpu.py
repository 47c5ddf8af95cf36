"""The gate/up product on the tcgen05 kernel below 2,048 tokens (tests/test_gate_up_route.py has where it runs)."""

import pytest
import torch

from tests.test_kernels_gpu import randn

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from paged_llm_b200.kernels.ops import CudaOps
    ops = CudaOps("cuda")
    ops.set_compute_dtype(torch.bfloat16)
    return ops


# whole and ragged tiles of 256 tokens and of 128 features, one to eight waves of them
@pytest.mark.parametrize("M,I", [(256, 8192), (241, 8192), (455, 8192), (512, 9208), (700, 5632), (1000, 14336), (2047, 5632)])
def test_gate_up_below_2048_tokens(ops, monkeypatch, M, I):
    h, w = randn(M, 256, seed=61, dtype=torch.bfloat16), randn(2 * I, 256, seed=62, dtype=torch.bfloat16, std=1 / 16)
    monkeypatch.setattr(ops, "_gate_up_tc_ok", lambda *a: True)               # (the kernel is tested beyond the sizes it runs at)
    before = ops.launches
    got = ops.gated_silu_linear(h, w)
    assert ops.launches == before + 1, "one kernel"
    both = (h.float() @ w.float().T).to(torch.bfloat16).float()
    g, u = both[:, :I], both[:, I:]
    want = torch.nn.functional.silu(g) * u
    # Sums of 256 products of size 1/16 in float32 in another order (some 2^-20 apart); a gate or up value beside a tie may so
    # round to the neighbour, which is up to 2^-7 of it away, times the other factor (silu' is below 1.1); the result is
    # rounded once more (2^-8 of it).
    near = lambda v: 2.0 ** -7 * v.abs() + 2.0 ** -20
    bound = 1.1 * near(g) * u.abs() + torch.nn.functional.silu(g).abs() * near(u) + 1.1 * near(g) * near(u) + 2.0 ** -8 * want.abs() * 1.02
    assert bool(((got.float() - want).abs() <= bound).all())


# the shortest and the longest sums that the rule sends here: one number of tokens and features each side of a tile's edge
@pytest.mark.parametrize("K", [512, 4096])
@pytest.mark.parametrize("M,I", [(512, 8192), (511, 8200)])
def test_the_ends_of_the_rule(ops, M, I, K):
    h, w = randn(M, K, seed=63, dtype=torch.bfloat16), randn(2 * I, K, seed=64, dtype=torch.bfloat16, std=K ** -0.5)
    assert ops._gate_up_tc_ok(h, w, I, "silu") and not ops._gemm_tc_ok(h, w, "silu")
    before = ops.launches
    got = ops.gated_silu_linear(h, w)
    assert ops.launches == before + 1, "one kernel"
    exact = h.double() @ w.double().T
    g, u = exact[:, :I], exact[:, I:]
    silu = torch.nn.functional.silu
    # Gate and up are float32 sums (K products: off by K 2^-24 of the sum of their sizes at most) rounded to bfloat16 (2^-8 of the
    # value at most); the result is rounded once more (silu' is below 1.1).
    sizes = h.double().abs() @ w.double().abs().T
    off = 2.0 ** -8 * exact.abs() + 1.01 * K * 2.0 ** -24 * sizes
    og, ou = off[:, :I], off[:, I:]
    want = silu(g) * u
    bound = 1.1 * og * u.abs() + silu(g).abs() * ou + 1.1 * og * ou + 2.0 ** -8 * want.abs() * 1.02 + 1e-30
    assert bool(((got.double() - want).abs() <= bound).all())
