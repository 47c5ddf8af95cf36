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
    lib, attention = ops._attention_bf16(d)
    asked = []

    def noting(p, stream):
        asked.append((p._obj.three_blocks, p._obj.small_rows, bool(p._obj.rope_table)))
        return attention(p, stream)

    ops._attention_bf16 = lambda _: (lib, noting)
    try:
        out = ops.qkv_attention(h, w, nh, nkv, d, rope, ctx, kv_dev, bt.cuda(), d ** -0.5, None).float().cpu()
    finally:
        ops.rope_in_attention = old
        del ops._attention_bf16
    assert asked == [(1, nh // nkv, inside)]                                  # what dec::launch takes that form by
    for s, L in enumerate(k_lens):
        qs = torch.zeros(L, nh, d)
        qs[L - 1] = q_rot[s]
        want = plain_llama.causal_attention(qs, keys[s], vals[s], d ** -0.5, window=None)[L - 1:].reshape(1, nh * d)
        torch.testing.assert_close(out[s:s + 1], want, atol=tol(dtype), rtol=tol(dtype), msg=f"request {s}")


def test_contexts_that_grow_past_the_form(tmp_path):
    """64 requests of 16 kv heads: short contexts take the form, and a graph of their own takes over once the longest context is
    past the limit (lowered here).  Logits on both sides, replayed and launched one by one, against the float32 engine's."""
    from paged_llm_b200.engine.replay import TraceReplayer
    from tests import schedules
    from tests.helpers import assert_bf16_close_to_f32, requests_for
    from tests.tiny import make_folder
    hf = {"architectures": ["LlamaForCausalLM"], "vocab_size": 256, "hidden_size": 128, "intermediate_size": 256, "num_hidden_layers": 2,
          "num_attention_heads": 16, "num_key_value_heads": 16, "head_dim": 64, "rms_norm_eps": 1e-5, "rope_theta": 10000.0,
          "max_position_embeddings": 512, "tie_word_embeddings": False, "hidden_act": "silu", "torch_dtype": "float32"}
    folder = make_folder(tmp_path, hf, dict(seed=4, std=0.05, norm_std=0.1))
    reqs = requests_for(256, [21 + i % 5 for i in range(60)] + [45] * 4, seed=9)
    steps = [{"step": 0, "entries": [{"id": r, "tokens": t[:-6], "want": []} for r, t in reqs.items()], "end": []}]
    for i in range(6):
        steps.append({"step": i + 1, "entries": [{"id": r, "tokens": [t[len(t) - 6 + i]], "want": [0]} for r, t in reqs.items()],
                      "end": list(reqs) if i == 5 else []})

    def logits(dtype, **kw):
        rp = TraceReplayer(folder, dtype, 64 * 64, **kw)
        rp.ops.THREE_BLOCKS_KEYS = 42                              # the longest context is 40 to 45 keys
        return schedules.collect(steps, {rec["step"]: rp.step(rec) for rec in steps}), rp

    want, _ = logits("float32")
    launched, rp = logits("bfloat16", enforce_eager=True)
    assert rp.runner.num_graph_steps == 0
    replayed, rp = logits("bfloat16")
    assert {("decode", 64), ("decode", 64, (True,))} <= set(rp.runner._graphs) and rp.runner.num_graph_steps == 6
    for rid in reqs:
        assert_bf16_close_to_f32(launched[rid], want[rid], f"launched {rid}")
        assert_bf16_close_to_f32(replayed[rid], want[rid], f"replayed {rid}")
