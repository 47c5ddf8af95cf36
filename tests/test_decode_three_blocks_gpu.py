"""Decode steps of so many requests that three blocks of the decode kernel share an SM (`CudaOps._three_blocks`), with the
rotation inside and without, against the plain formulation."""

import pytest
import torch

from tests import plain_llama
from tests.test_kernels_gpu import make_ctx, paged_case, randn, tol

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from paged_llm_b200.kernels.ops import CudaOps
    ops = CudaOps("cuda")
    ops.set_compute_dtype(torch.bfloat16)
    return ops


# the fewest requests that take this form and more; contexts of one key, around a tile (16) and a range (128), and long ones
# among short ones, which are cut into ranges; eight query heads per kv head and fewer
@pytest.mark.parametrize("nh,nkv,n", [(32, 4, 223), (16, 8, 112), (8, 8, 160)])
@pytest.mark.parametrize("lens", [(1, 15, 16, 17, 33), (127, 128, 129, 40, 300), (20, 31, 900, 7, 2000)])
@pytest.mark.parametrize("inside", [True, False])
def test_many_requests(ops, nh, nkv, n, lens, inside):
    from paged_llm_b200.parts.rope import RotaryEncoding
    d, ps, H, theta, dtype = 64, 16, 128, 10000.0, torch.bfloat16
    k_lens = [lens[i % 5] if i < 20 or lens[i % 5] < 500 else 64 for i in range(n)]
    q_lens = [1] * n
    rope = RotaryEncoding({}, head_dim=d, theta=theta)
    rope.prepare(2048, "cuda", ops)
    _, kv, bt, keys, vals = paged_case(q_lens, k_lens, nh, nkv, d, ps, dtype, seed=7)
    h, w = randn(n, H, seed=71, dtype=dtype), randn((nh + 2 * nkv) * d, H, seed=72, dtype=dtype, std=H ** -0.5)
    y = (h.float().cpu() @ w.float().cpu().T).to(dtype).float()
    cos, sin = plain_llama.rotary_cos_sin(torch.tensor(k_lens) - 1, plain_llama.inv_frequencies(d, theta, None))
    q_rot = plain_llama.apply_rotary(y[:, :nh * d].view(n, nh, d), cos, sin).to(dtype).float()
    k_rot = plain_llama.apply_rotary(y[:, nh * d:(nh + nkv) * d].view(n, nkv, d), cos, sin).to(dtype).float()
    kv = kv.clone()
    for s, L in enumerate(k_lens):
        kv[bt[s, (L - 1) // ps], :, :, (L - 1) % ps] = float("nan")        # the step's own slot, until it is written
        keys[s][L - 1], vals[s][L - 1] = k_rot[s], y[s, (nh + nkv) * d:].view(nkv, d)
    ctx = make_ctx(ops, q_lens, k_lens, nh, nkv, None, d, planned=True)
    assert ops._three_blocks(n, nkv, nh // nkv, d) and not ops._three_blocks(6 * ops.num_sms // nkv, nkv, nh // nkv, d)
    assert ctx.attention_plans[(nh // nkv, nkv, None, d)].even
    kv_dev, old = kv.cuda(), ops.rope_in_attention
    ops.rope_in_attention = inside
    try:
        out = ops.qkv_attention(h, w, nh, nkv, d, rope, ctx, kv_dev, bt.cuda(), d ** -0.5, None).float().cpu()
    finally:
        ops.rope_in_attention = old
    for s, L in enumerate(k_lens):
        qs = torch.zeros(L, nh, d)
        qs[L - 1] = q_rot[s]
        want = plain_llama.causal_attention(qs, keys[s], vals[s], d ** -0.5, window=None)[L - 1:].reshape(1, nh * d)
        torch.testing.assert_close(out[s:s + 1], want, atol=tol(dtype), rtol=tol(dtype), msg=f"request {s}")
