"""Steps with prompt portions whose queries are rotated by the kernel of the prompt tiles as it loads them
(`CudaOps.qkv_attention`), against the plain formulation."""

import contextlib

import numpy as np
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


@contextlib.contextmanager
def tiles_that_rotate(ops):
    """Per call of the attention, whether it was left the rotation of the prompt tiles' queries."""
    seen, attention = [], ops.paged_attention
    ops.paged_attention = lambda *a, **kw: (seen.append(kw.get("tile_rope") is not None), attention(*a, **kw))[1]
    try:
        yield seen
    finally:
        del ops.paged_attention


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
    with tiles_that_rotate(ops) as seen:
        out = ops.qkv_attention(h, w, nh, nkv, d, rope, ctx, kv_dev, bt.cuda(), d ** -0.5, None).float().cpu()
    assert seen == [True], "this test is about the kernel that rotates"
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


# Under the masks of windows and of chunks too.  A query is the same bfloat16 number whichever kernel rotates it, so the outputs are
# the same bit for bit with the separate rotation; and against the plain formulation.
@pytest.mark.parametrize("nh,nkv,d", [(32, 4, 64), (8, 2, 128)])
@pytest.mark.parametrize("window,chunk", [(None, None), (40, None), (200, None), (None, 48), (None, 256)])
def test_windows_and_chunks(ops, nh, nkv, d, window, chunk):
    from paged_llm_b200.engine.context import AttentionPlan
    from paged_llm_b200.kernels.ops import attention_plan_key
    from paged_llm_b200.parts.rope import RotaryEncoding
    dtype, theta, H, ps = torch.bfloat16, 10000.0, 128, 16
    q_lens, k_lens = [150, 1, 2, 33], [150, 300, 97, 420]
    rope = RotaryEncoding({}, head_dim=d, theta=theta)
    rope.prepare(1024, "cuda", ops)
    _, kv, bt, keys, vals = paged_case(q_lens, k_lens, nh, nkv, d, ps, dtype, seed=6)
    T = sum(q_lens)
    h, w = randn(T, H, seed=61, dtype=dtype), randn((nh + 2 * nkv) * d, H, seed=62, dtype=dtype, std=H ** -0.5)
    ctx = make_ctx(ops, q_lens, k_lens, nh, nkv, window, d, planned=True)
    plan = ops.plan_attention(q_lens, k_lens, nh // nkv, nkv, window, d, chunk=chunk)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda()
    small, large = plan["small"].reshape(-1, 4), plan["large"].reshape(-1, 4)
    ctx.attention_plans = {attention_plan_key(nh, nkv, window, d, chunk): AttentionPlan(
        dev(small), dev(large), dev(plan["splits"]), len(small), len(large), plan["max_splits"], plan["num_small_tokens"],
        plan["long_context"], plan["even"])}
    outs, pools, old = [], [], ops.rope_in_attention
    for inside in (True, False):
        ops.rope_in_attention, kv_dev = inside, kv.cuda()
        try:
            with tiles_that_rotate(ops) as seen:
                outs.append(ops.qkv_attention(h, w, nh, nkv, d, rope, ctx, kv_dev, bt.cuda(), d ** -0.5, window, chunk=chunk))
        finally:
            ops.rope_in_attention = old
        assert seen == [inside]
        pools.append(kv_dev)
    assert torch.equal(pools[0].view(torch.int16), pools[1].view(torch.int16))
    assert torch.equal(outs[0], outs[1])
    y = (h.float().cpu() @ w.float().cpu().T).to(dtype).float()
    pos = torch.cat([torch.arange(k - q, k) for q, k in zip(q_lens, k_lens)])
    cos, sin = plain_llama.rotary_cos_sin(pos, plain_llama.inv_frequencies(d, theta, None))
    q_rot = plain_llama.apply_rotary(y[:, :nh * d].view(T, nh, d), cos, sin).to(dtype).float()
    k_rot = plain_llama.apply_rotary(y[:, nh * d:(nh + nkv) * d].view(T, nkv, d), cos, sin).to(dtype).float()
    v_new, out, cu = y[:, (nh + nkv) * d:].view(T, nkv, d), outs[0].float().cpu(), ctx.host.cu
    for s, (nq, L) in enumerate(zip(q_lens, k_lens)):
        keys[s][L - nq:], vals[s][L - nq:] = k_rot[cu[s]:cu[s + 1]], v_new[cu[s]:cu[s + 1]]
        qs = torch.zeros(L, nh, d)
        qs[L - nq:] = q_rot[cu[s]:cu[s + 1]]
        step = chunk or L                                             # (a chunk's queries see its own keys alone)
        want = torch.cat([plain_llama.causal_attention(qs[c:c + step], keys[s][c:c + step], vals[s][c:c + step], d ** -0.5, window=window)
                          for c in range(0, L, step)])[L - nq:].reshape(nq, nh * d)
        torch.testing.assert_close(out[cu[s]:cu[s + 1]], want, atol=tol(dtype), rtol=tol(dtype), msg=f"request {s}")


def test_one_graph_while_requests_pass_between_the_forms(tmp_path):
    """Four query heads per kv head: up to four tokens of a request are a small item, more are tiles.  Steps of one 64-token
    bucket in which requests pass from one to the other and back replay one captured graph, whose lists hold places for tiles
    that are not there."""
    from paged_llm_b200.engine.replay import TraceReplayer
    from tests import schedules
    from tests.helpers import assert_bf16_close_to_f32, requests_for
    from tests.tiny import make_folder
    hf = {"architectures": ["LlamaForCausalLM"], "vocab_size": 256, "hidden_size": 128, "intermediate_size": 256, "num_hidden_layers": 2,
          "num_attention_heads": 8, "num_key_value_heads": 2, "head_dim": 64, "rms_norm_eps": 1e-5, "rope_theta": 10000.0,
          "max_position_embeddings": 512, "tie_word_embeddings": False, "hidden_act": "silu", "torch_dtype": "float32"}
    folder = make_folder(tmp_path, hf, dict(seed=3, std=0.05, norm_std=0.1))
    cuts = {"r0": (20, 3, 40, 4, 30, 5), "r1": (4, 40, 2, 41, 3, 4), "r2": (16, 1, 5, 2, 17, 40)}
    reqs = {rid: toks for rid, toks in zip(cuts, requests_for(256, [sum(c) for c in cuts.values()], seed=8).values())}
    steps, at = [], dict.fromkeys(cuts, 0)
    for i in range(6):
        entries = []
        for rid, toks in reqs.items():
            n = cuts[rid][i]
            entries.append({"id": rid, "tokens": toks[at[rid]:at[rid] + n], "want": [n - 1]})
            at[rid] += n
        steps.append({"step": i, "entries": entries, "end": list(cuts) if i == 5 else []})

    def logits(dtype, **kw):
        rp = TraceReplayer(folder, dtype, 512, poison=float("nan"), **kw)
        with tiles_that_rotate(rp.ops) as seen:
            outputs = {rec["step"]: rp.step(rec) for rec in steps}
        return schedules.collect(steps, outputs), rp, seen

    want, _, seen = logits("float32")
    assert not any(seen)
    launched, rp, seen = logits("bfloat16", enforce_eager=True)
    assert all(seen) and len(seen) == 12 and rp.runner.num_graph_steps == 0
    replayed, rp, seen = logits("bfloat16")
    assert seen and all(seen) and rp.runner.num_graph_steps >= 4 and [k[0] for k in rp.runner._graphs] == ["mixed"]
    for rid in cuts:
        assert_bf16_close_to_f32(launched[rid], want[rid], f"launched {rid}")
        assert_bf16_close_to_f32(replayed[rid], want[rid], f"replayed {rid}")
