"""Decode attention whose ranges are cut evenly (work list), with the rotation and the cache write inside, against the plain
rotation and softmax in float32: ragged contexts on the edges of tiles, pages and ranges, one to sixteen query heads per
kv head, and a step padded to the size of its graph."""

import types

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from paged_llm_b200.kernels.ops import CudaOps
    ops = CudaOps("cuda")
    ops.set_compute_dtype(torch.bfloat16)
    return ops


def rotated(x, table):
    """x [..., d] bfloat16 rotated by (cos, sin) [d / 2, 2] in float32, rounded back as the kernels store it."""
    d = x.shape[-1]
    a, b = x[..., :d // 2].float(), x[..., d // 2:].float()
    c, s = table[:, 0], table[:, 1]
    return torch.cat([a * c - b * s, b * c + a * s], -1).to(torch.bfloat16)


EDGES = [1, 2, 15, 16, 17, 31, 32, 33, 127, 128, 129, 144, 513, 1000, 2049, 3500]


@pytest.mark.parametrize("nh,nkv,d,ps,S,pad", [(32, 4, 64, 16, 40, 48), (32, 8, 64, 32, 24, 32), (32, 8, 128, 16, 21, 24),
                                               (32, 2, 64, 48, 80, 96), (8, 8, 128, 64, 19, 19), (16, 1, 64, 16, 150, 192)])
def test_even_ranges_against_plain_attention(ops, nh, nkv, d, ps, S, pad):
    from paged_llm_b200.engine.context import AttentionPlan, HostBatch
    G, W = nh // nkv, (nh + 2 * nkv) * d
    k_lens = [EDGES[(i * 5) % len(EDGES)] for i in range(S)]
    g = torch.Generator(device="cuda").manual_seed(S)
    pages = [-(-n // ps) for n in k_lens]
    order = torch.randperm(sum(pages) + 3, generator=torch.Generator().manual_seed(1)).int()
    bt = torch.full((pad, max(pages) + 1), 10 ** 6, dtype=torch.int32)
    kv = torch.full((sum(pages) + 3, 2, nkv, ps, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    qkv = torch.randn(pad, W, device="cuda", generator=g).to(torch.bfloat16)
    table = torch.randn(4096, d // 2, 2, device="cuda", generator=g)
    old, o = [], 0
    for s, n in enumerate(k_lens):                        # all keys but the step's own are in the cache, the rest is NaN
        mine = order[o:o + pages[s]]
        bt[s, :pages[s]] = mine
        o += pages[s]
        both = torch.randn(2, n - 1, nkv, d, device="cuda", generator=g).to(torch.bfloat16)
        flat = torch.full((2, pages[s] * ps, nkv, d), float("nan"), dtype=torch.bfloat16, device="cuda")
        flat[:, :n - 1] = both
        kv[mine.long().cuda()] = flat.view(2, pages[s], ps, nkv, d).permute(1, 0, 3, 2, 4)
        old.append(both)
    plan = ops.plan_attention([1] * S, k_lens, G, nkv, None, d, pad_requests=pad, fixed_capacity=True)
    assert plan["even"] and plan["small"].reshape(-1, 4)[:, 3].max() > 1, "some request is meant to be split"
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda()
    small = plan["small"].reshape(-1, 4)
    ap = AttentionPlan(dev(small), None, dev(plan["splits"]), len(small), 0, plan["max_splits"], plan["num_small_tokens"],
                       plan["long_context"], plan["even"])
    host = HostBatch([1] * S, [n - 1 for n in k_lens], [-1] * S)
    ctx = types.SimpleNamespace(num_tokens=pad, num_seqs=pad, host=host, cu_seqlens_q=dev(list(range(S + 1)) + [S] * (pad - S)),
                                seq_lens_k=dev(k_lens + [0] * (pad - S)), attention_plans={(G, nkv, None, d): ap}, padded=pad > S)
    rope = types.SimpleNamespace(table=table, rotary_dim=d)
    for _ in range(2):                                    # the second time finds the counters as the first left them
        out = ops.paged_attention(qkv, nh, nkv, d, kv, bt.cuda(), ctx, d ** -0.5, None, rope=rope).float()
    assert (out[S:] == 0).all()
    for s, n in enumerate(k_lens):
        q, k, v = (t.view(-1, d) for t in qkv[s].split([nh * d, nkv * d, nkv * d]))
        q, k = rotated(q, table[n - 1]), rotated(k, table[n - 1])
        slot = kv[bt[s, (n - 1) // ps], :, :, (n - 1) % ps]
        # (the kernel may round one product of a rotated pair less than torch does: a neighbouring bfloat16)
        torch.testing.assert_close(slot[0].float(), k.float(), atol=2 ** -20, rtol=2 ** -7, msg=f"request {s}: the cached key")
        assert torch.equal(slot[1], v), f"request {s}: the cached value"
        keys, vals = torch.cat([old[s][0], slot[0][None]]).float(), torch.cat([old[s][1], v[None]]).float()
        score = torch.einsum("jgd,njd->jgn", q.float().view(nkv, G, d), keys) * d ** -0.5
        want = torch.einsum("jgn,njd->jgd", score.softmax(-1), vals).reshape(-1)
        # probabilities and the result are rounded to bfloat16 (2^-9 each), relative to values of up to 4.5
        torch.testing.assert_close(out[s], want, atol=2 * 4.5 * 2 ** -9, rtol=2 ** -8, msg=f"request {s} of {n} keys")
    assert ops.kernel_timeouts() == 0


@pytest.mark.parametrize("nq", [1, 2])
@pytest.mark.parametrize("nh,nkv,d,ps,window", [(32, 8, 64, 16, None), (32, 8, 128, 16, None),             # attention_decode.cuh
                                                (4, 4, 16, 16, None), (8, 4, 32, 16, None), (6, 2, 48, 16, None), (8, 2, 80, 16, None),
                                                (4, 2, 256, 16, None), (16, 2, 64, 8, None), (8, 2, 128, 20, None),
                                                (16, 2, 64, 16, 50), (4, 4, 16, 8, 300), (4, 2, 256, 16, 200)])
def test_rotation_inside_the_list_form(ops, nh, nkv, d, ps, window, nq):
    """The list form that rotates and writes the cache itself, for every kernel behind it (head sizes, page sizes, windows),
    one and two new tokens per request.  At 385 and 897 keys the last range begins with the second of the two."""
    from paged_llm_b200.engine.context import AttentionPlan, HostBatch
    G, W = nh // nkv, (nh + 2 * nkv) * d
    k_lens = [n for n in [2, 3, 16, 17, 31, 32, 33, 34, 127, 128, 129, 144, 385, 513, 897, 1000, 2049] if n >= nq] * 2
    S, T = len(k_lens), len(k_lens) * nq
    g = torch.Generator(device="cuda").manual_seed(d + nq)
    pages = [-(-n // ps) for n in k_lens]
    order = torch.randperm(sum(pages) + 3, generator=torch.Generator().manual_seed(1)).int()
    bt = torch.full((S, max(pages) + 1), 10 ** 6, dtype=torch.int32)
    kv = torch.full((sum(pages) + 3, 2, nkv, ps, d), float("nan"), dtype=torch.bfloat16, device="cuda")
    qkv = torch.randn(T, W, device="cuda", generator=g).to(torch.bfloat16)
    table = torch.randn(4096, d // 2, 2, device="cuda", generator=g)
    old, o = [], 0
    for s, n in enumerate(k_lens):                        # all keys but the step's own are in the cache, the rest is NaN
        mine = order[o:o + pages[s]]
        bt[s, :pages[s]] = mine
        o += pages[s]
        both = torch.randn(2, n - nq, nkv, d, device="cuda", generator=g).to(torch.bfloat16)
        flat = torch.full((2, pages[s] * ps, nkv, d), float("nan"), dtype=torch.bfloat16, device="cuda")
        flat[:, :n - nq] = both
        kv[mine.long().cuda()] = flat.view(2, pages[s], ps, nkv, d).permute(1, 0, 3, 2, 4)
        old.append(both)
    before = kv.clone()
    splits = [min(8, -(-n // 128)) for n in k_lens]
    small = np.array([(s, s * nq, j, m) for s, m in enumerate(splits) for j in range(m)], np.int32)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda()
    ap = AttentionPlan(dev(small), None, dev([(m, s * nq) for s, m in enumerate(splits)]), len(small), 0, 8, T, False, True)
    host = HostBatch([nq] * S, [n - nq for n in k_lens], [-1] * S)
    key = (G, nkv, window, d)
    ctx = types.SimpleNamespace(num_tokens=T, num_seqs=S, host=host, cu_seqlens_q=dev(host.cu), seq_lens_k=dev(k_lens),
                                attention_plans={key: ap}, padded=False)
    rope = types.SimpleNamespace(table=table, rotary_dim=d)
    for _ in range(2):                                    # the second time finds the counters as the first left them
        launches = ops.launches
        out = ops.paged_attention(qkv, nh, nkv, d, kv, bt.cuda(), ctx, d ** -0.5, window, rope=rope).float()
        assert ops.launches == launches + 1
    for s, n in enumerate(k_lens):
        keys, vals = old[s][0], old[s][1]
        for i in range(nq):
            q, k, v = (t.view(-1, d) for t in qkv[s * nq + i].split([nh * d, nkv * d, nkv * d]))
            pos = n - nq + i
            q, k = rotated(q, table[pos]), rotated(k, table[pos])
            slot = kv[bt[s, pos // ps], :, :, pos % ps]
            before[bt[s, pos // ps], :, :, pos % ps] = slot
            # (the kernel may round one product of a rotated pair less than torch does: a neighbouring bfloat16)
            torch.testing.assert_close(slot[0].float(), k.float(), atol=2 ** -20, rtol=2 ** -7, msg=f"request {s}: the cached key")
            assert torch.equal(slot[1], v), f"request {s}: the cached value"
            keys, vals = torch.cat([keys, slot[0][None]]), torch.cat([vals, v[None]])
            lo = max(0, pos - window + 1) if window else 0
            score = torch.einsum("jgd,njd->jgn", q.float().view(nkv, G, d), keys[lo:].float()) * d ** -0.5
            want = torch.einsum("jgn,njd->jgd", score.softmax(-1), vals[lo:].float()).reshape(-1)
            # probabilities and the result are rounded to bfloat16 (2^-9 each), relative to values of up to 4.5
            torch.testing.assert_close(out[s * nq + i], want, atol=2 * 4.5 * 2 ** -9, rtol=2 ** -8, msg=f"request {s} of {n} keys")
    assert ((kv == before) | (torch.isnan(kv) & torch.isnan(before))).all(), "only the slots of the step's own tokens may change"
    assert ops.kernel_timeouts() == 0


@pytest.mark.parametrize("nh,nkv,d,H", [(32, 8, 64, 1280), (32, 8, 128, 96), (8, 8, 16, 96), (8, 8, 48, 1280), (8, 4, 256, 64), (32, 4, 64, 2048)])
@pytest.mark.parametrize("q_lens", [[1] * 40, [1] * 64, [2, 1, 2] * 14])
def test_front_of_a_decode_step_as_it_is_planned(ops, nh, nkv, d, H, q_lens):
    """`qkv_attention` of a step whose ranges the plan cuts evenly, as the engine runs it: the product (this package's or the
    library's, by width), then one kernel that rotates, writes the cache and attends.  Held to the same pieces in float32."""
    from paged_llm_b200.parts.rope import RotaryEncoding
    from tests import plain_llama
    from tests.test_kernels_gpu import make_ctx, paged_case, tol
    dtype, ps, G = torch.bfloat16, 16, nh // nkv
    S, T = len(q_lens), sum(q_lens)
    k_lens = [EDGES[(i * 5) % len(EDGES)] + 2 for i in range(S)]
    rope = RotaryEncoding({}, head_dim=d, theta=10000.0)
    rope.prepare(4096, "cuda", ops)
    _, kv, bt, keys, vals = paged_case(q_lens, k_lens, nh, nkv, d, ps, dtype, seed=3)
    g = torch.Generator().manual_seed(d)
    h = torch.randn(T, H, generator=g).to(dtype)
    w = (torch.randn((nh + 2 * nkv) * d, H, generator=g) * H ** -0.5).to(dtype)
    y = (h.float() @ w.float().T).to(dtype).float()                       # the projection rounds to bfloat16
    pos = torch.cat([torch.arange(k - q, k) for q, k in zip(q_lens, k_lens)])
    cos, sin = plain_llama.rotary_cos_sin(pos, plain_llama.inv_frequencies(d, 10000.0, None))
    q_rot = plain_llama.apply_rotary(y[:, :nh * d].view(T, nh, d), cos, sin).to(dtype).float()
    k_rot = plain_llama.apply_rotary(y[:, nh * d:(nh + nkv) * d].view(T, nkv, d), cos, sin).to(dtype).float()
    v_new = y[:, (nh + nkv) * d:].view(T, nkv, d)
    ctx = make_ctx(ops, q_lens, k_lens, nh, nkv, None, d, planned=True)
    plan = ctx.attention_plans[(G, nkv, None, d)]
    inside = max(q_lens) * G <= 16
    if nkv * S >= 148:
        assert plan.even and not ops._runs_as_clusters(plan, ctx, nh, nkv, True) and ops._rotates_inside(plan, ctx, nh, nkv) == inside
    kv_dev = kv.cuda()
    at = ctx.host.cu
    for s in range(S):
        for n in range(k_lens[s] - q_lens[s], k_lens[s]):                 # poison until the step writes them
            kv_dev[bt[s, n // ps], :, :, n % ps] = float("nan")
            t = at[s] + n - (k_lens[s] - q_lens[s])
            keys[s][n], vals[s][n] = k_rot[t], v_new[t]
    before = ops.launches
    out = ops.qkv_attention(h.cuda(), w.cuda(), nh, nkv, d, rope, ctx, kv_dev, bt.cuda(), d ** -0.5, None).float().cpu()
    if inside:
        assert ops.launches - before == 1 + (H >= 1280 and T <= 64)
    for s, (nq, n) in enumerate(zip(q_lens, k_lens)):
        for j in range(n - nq, n):
            t = at[s] + j - (n - nq)
            score = torch.einsum("jgd,njd->jgn", q_rot[t].view(nkv, G, d), keys[s][:j + 1]) * d ** -0.5
            want = torch.einsum("jgn,njd->jgd", score.softmax(-1), vals[s][:j + 1]).reshape(-1)
            torch.testing.assert_close(out[t], want, atol=tol(dtype), rtol=tol(dtype), msg=f"request {s} of {n} keys")
            got = kv_dev[bt[s, j // ps], :, :, j % ps].float().cpu()
            torch.testing.assert_close(got[0], keys[s][j], atol=tol(dtype), rtol=tol(dtype))
            torch.testing.assert_close(got[1], vals[s][j], atol=tol(dtype), rtol=tol(dtype))
    assert ops.kernel_timeouts() == 0
