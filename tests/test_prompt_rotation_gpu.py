"""Steps with prompt portions whose queries are rotated by the kernel of the prompt tiles as it loads them
(`CudaOps.qkv_attention`), against the plain formulation."""

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


# 17 tokens and more in each step (up to 16 rotate in the projection); tiles of 128 rows, so of 128 / group tokens; portions of
# few tokens that are small items (rotated with their keys) beside tiles; behind nothing, inside a page and inside a tile of keys
@pytest.mark.parametrize("nh,nkv,d", [(32, 4, 64), (32, 8, 128), (6, 6, 64), (14, 2, 128)])
@pytest.mark.parametrize("ps", [8, 16, 64])
@pytest.mark.parametrize("q_lens,k_lens", [([61], [61]), ([17], [200]), ([130, 1, 2, 33], [130, 77, 300, 161]), ([300, 16, 129], [300, 16, 1000])])
def test_prompt_tiles_rotate_their_queries(ops, nh, nkv, d, ps, q_lens, k_lens):
    from paged_llm_b200.parts.rope import RotaryEncoding
    dtype, theta, H = torch.bfloat16, 10000.0, 128
    rope = RotaryEncoding({}, head_dim=d, theta=theta)
    rope.prepare(1024, "cuda", ops)
    _, kv, bt, keys, vals = paged_case(q_lens, k_lens, nh, nkv, d, ps, dtype, seed=5)
    T = sum(q_lens)
    h, w = randn(T, H, seed=51, dtype=dtype), randn((nh + 2 * nkv) * d, H, seed=52, dtype=dtype, std=H ** -0.5)
    y = (h.float().cpu() @ w.float().cpu().T).to(dtype).float()           # the projection rounds to bfloat16
    pos = torch.cat([torch.arange(k - q, k) for q, k in zip(q_lens, k_lens)])
    cos, sin = plain_llama.rotary_cos_sin(pos, plain_llama.inv_frequencies(d, theta, None))
    q_rot = plain_llama.apply_rotary(y[:, :nh * d].view(T, nh, d), cos, sin).to(dtype).float()
    k_rot = plain_llama.apply_rotary(y[:, nh * d:(nh + nkv) * d].view(T, nkv, d), cos, sin).to(dtype).float()
    v_new = y[:, (nh + nkv) * d:].view(T, nkv, d)
    kv, t = kv.clone(), 0
    for s, (nq, L) in enumerate(zip(q_lens, k_lens)):
        for n in range(L - nq, L):
            kv[bt[s, n // ps], :, :, n % ps] = float("nan")
            keys[s][n], vals[s][n] = k_rot[t], v_new[t]
            t += 1
    ctx = make_ctx(ops, q_lens, k_lens, nh, nkv, None, d, planned=True)
    kv_dev = kv.cuda()
    assert ops._prompt_tiles_rotate(nh, nkv, d, kv_dev, rope), "this test is about the kernel that rotates"
    out = ops.qkv_attention(h, w, nh, nkv, d, rope, ctx, kv_dev, bt.cuda(), d ** -0.5, None).float().cpu()
    cu = ctx.host.cu
    for s, (nq, L) in enumerate(zip(q_lens, k_lens)):
        qs = torch.zeros(L, nh, d)
        qs[L - nq:] = q_rot[cu[s]:cu[s + 1]]
        want = plain_llama.causal_attention(qs, keys[s], vals[s], d ** -0.5, window=None)[L - nq:].reshape(nq, nh * d)
        torch.testing.assert_close(out[cu[s]:cu[s + 1]], want, atol=tol(dtype), rtol=tol(dtype), msg=f"request {s}")
    # the cache holds the same keys and values as behind the separate kernels, bit for bit
    separate = kv.cuda()
    ops.qkv_rope_write(h, w, nh, nkv, d, rope, ctx, separate, bt.cuda())
    assert torch.equal(separate.view(torch.int16), kv_dev.view(torch.int16))
