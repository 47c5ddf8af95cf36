"""Host-side attention work lists: every query row and every key is covered
exactly once, and the array form for decode steps equals the general form."""

import numpy as np
import pytest

from paged_llm_b200.kernels import plan as planning


def general(q_lens, k_lens, G, nkv, window, **kw):
    args = dict(small_rows=16, large_rows=64, min_split_keys=128, num_sms=148, max_splits=32)
    args.update(kw)
    return planning.plan_attention(q_lens, k_lens, G, nkv, window, **args)


@pytest.mark.parametrize("q_lens,k_lens,G", [([1, 1, 1], [5, 700, 2048], 8), ([33, 1, 2, 200], [33, 64, 300, 500], 8),
                                              ([5, 17], [5, 17], 1), ([1], [1], 2)])
def test_items_cover_rows_and_keys(q_lens, k_lens, G):
    plan = general(q_lens, k_lens, G, 4, None)
    small, large = plan["small"].reshape(-1, 4), plan["large"].reshape(-1, 4)
    splits = plan["splits"].reshape(-1, 2)
    for s, (nq, lk) in enumerate(zip(q_lens, k_lens)):
        rows = nq * G
        if rows <= 16:
            mine = small[small[:, 0] == s]
            assert sorted(mine[:, 2].tolist()) == list(range(splits[s, 0])) and (mine[:, 3] == splits[s, 0]).all()
            assert splits[s, 0] <= max(1, -(-lk // 128)) and not (large[:, 0] == s).any()
        else:
            mine = large[large[:, 0] == s]
            assert sorted(mine[:, 1].tolist()) == list(range(-(-rows // 64))) and not (small[:, 0] == s).any()
    bases = [splits[s, 1] for s in range(len(q_lens)) if q_lens[s] * G <= 16]
    sizes = [q_lens[s] for s in range(len(q_lens)) if q_lens[s] * G <= 16]
    assert bases == list(np.cumsum([0] + sizes[:-1])) and plan["num_small_tokens"] == sum(sizes)


@pytest.mark.parametrize("fixed", [False, True])
@pytest.mark.parametrize("k_lens", [[5], [513, 640, 90, 2048, 129], list(range(100, 164))])
def test_decode_fast_path_equals_the_general_plan(k_lens, fixed):
    S = len(k_lens)
    pad = {1: 1, 5: 8, 64: 64}[S] if fixed else None
    fast = general([1] * S, k_lens, 8, 4, None, pad_requests=pad, fixed_capacity=fixed)
    slow = general([1] * S, k_lens, 8, 4, 10 ** 9, pad_requests=pad, fixed_capacity=fixed)   # a window switches it off
    for key in ("small", "large", "splits"):
        assert np.array_equal(fast[key], slow[key]), key
    assert fast["max_splits"] == slow["max_splits"] and fast["num_small_tokens"] == slow["num_small_tokens"]


def test_longest_tiles_first():
    plan = general([300, 40], [300, 900], 8, 4, None)
    large = plan["large"].reshape(-1, 4)
    assert large[0, 0] == 1                     # the request with the longest context leads


def test_long_context_decode_steps_are_split_further():
    """Few long requests: a block of a cluster of at most 8 would walk thousands of keys alone, so
    the plan turns to about three blocks per SM through the work list; short contexts and steps
    with prompt portions stay as they are."""
    from paged_llm_b200.kernels.plan import is_long_context, long_context_splits, plan_attention

    kw = dict(small_rows=16, large_rows=128, min_split_keys=128, num_sms=148, max_splits=32, cluster_max=8, long_keys=600)
    short = plan_attention([1] * 8, [700] * 8, 8, 4, None, **kw)
    assert not short["long_context"] and short["max_splits"] == 5
    long = plan_attention([1] * 8, [16000] * 8, 8, 4, None, **kw)
    assert long["long_context"] and long["max_splits"] == 13 == long_context_splits(8, 4, 148, 32)
    assert len(long["small"]) // 4 == 8 * 13
    one = plan_attention([1], [16000], 8, 4, None, **kw)
    assert one["long_context"] and one["max_splits"] == 32
    assert not plan_attention([1], [4000], 8, 4, None, **kw)["long_context"]           # 8 blocks x 500 keys
    assert not plan_attention([1, 40], [16000, 16000], 8, 4, None, **kw)["long_context"]   # a prompt portion in the step
    assert not plan_attention([1] * 8, [16000] * 8, 8, 4, None, **{**kw, "cluster_max": 0})["long_context"]
    # the class of a padded graph bucket is that of the bucket, whatever the live requests
    assert is_long_context(8, 4, 148, 32, 8, 600, 3001) and not is_long_context(8, 4, 148, 32, 8, 600, 3000)
    # 64 requests x 4 kv heads: one block each either way, so there is no second class (and no second graph)
    assert not is_long_context(64, 4, 148, 32, 8, 600, 100000)


@pytest.mark.parametrize("k_lens,nkv,pad", [([641] * 64, 4, 64), (list(range(131, 3501, 130)), 8, 32), ([1] * 40, 4, 48),
                                             ([1, 4000] * 20, 8, 48), (list(range(70, 778, 5)), 4, 192), ([3000] * 16, 8, 16),
                                             ([17] * 255 + [4000], 1, 256)])
def test_even_ranges_cover_every_key_and_fit_the_graph(k_lens, nkv, pad):
    """Steps that are cut into even ranges: every request has all its ranges, the list fits the capacity that a captured
    graph has, whatever the lengths, and its shape does not depend on them; a request has no more ranges than its keys have
    started multiples of 128 (129 keys may be cut into 96 and 33, since ranges begin at multiples of 32)."""
    kw = dict(cluster_max=8, long_keys=600, slots=296)
    S = len(k_lens)
    plan = general([1] * S, k_lens, 8, nkv, None, pad_requests=pad, fixed_capacity=True, **kw)
    assert plan["even"]
    small, splits = plan["small"].reshape(-1, 4), plan["splits"].reshape(-1, 2)
    real = small[small[:, 0] >= 0]
    assert (small[len(real):] == -1).all() and len(small) == pad + 296 // nkv
    for s, n in enumerate(k_lens):
        mine = real[real[:, 0] == s]
        assert sorted(mine[:, 2].tolist()) == list(range(splits[s, 0])) and (mine[:, 3] == splits[s, 0]).all()
        assert splits[s, 0] <= min(plan["max_splits"], max(1, -(-n // 128)))
    same = general([1] * S, [5] * (S - 1) + [max(k_lens)], 8, nkv, None, pad_requests=pad, fixed_capacity=True, **kw)
    assert same["small"].size == plan["small"].size and same["max_splits"] == plan["max_splits"]
    ends = [-(-k_lens[int(s)] // int(m)) for s, _, _, m in real]
    assert ends[0] <= max(max(k_lens), 128) and (len(set(k_lens)) > 1 or len(set(ends)) == 1)


def test_even_ranges_beside_prompt_portions():
    """A step of mixed items that replays a graph: the same capacity with and without decoding requests."""
    kw = dict(cluster_max=8, long_keys=600, slots=296, pad_requests=64, fixed_capacity=True, pad_tokens=448)
    busy = general([1] * 33 + [200, 100], [128 + 40 * i for i in range(33)] + [1200, 1100], 4, 8, None, **kw)
    alone = general([400], [400], 4, 8, None, **kw)
    for key in ("small", "large", "splits"):
        assert busy[key].size == alone[key].size
    assert busy["max_splits"] == alone["max_splits"] and busy["num_small_tokens"] == alone["num_small_tokens"]
    small = busy["small"].reshape(-1, 4)
    assert set(small[small[:, 0] >= 0][:, 0].tolist()) == set(range(33)) and (alone["small"] == -1).all()


@pytest.mark.parametrize("k_lens,nkv,pad", [(list(range(131, 3501, 130)), 8, 32), (list(range(70, 778, 5)), 4, 192), ([3000] * 16, 8, 16)])
def test_even_ranges_do_not_depend_on_the_step_they_were_planned_for(k_lens, nkv, pad):
    """A replayed decode step keeps its plan until a context grows past another multiple of 128 keys.  So that it gives what
    the same step gives with a plan of its own, bit for bit, all lengths between two multiples have one plan."""
    kw = dict(cluster_max=8, long_keys=600, slots=296, pad_requests=pad, fixed_capacity=True)
    from paged_llm_b200.kernels.ops import CudaOps
    assert CudaOps.MIN_SPLIT_KEYS % planning.GRAIN == 0, "what a replayed step goes by"
    S = len(k_lens)
    first, last = [-(-k // 128) * 128 - 127 for k in k_lens], [-(-k // 128) * 128 for k in k_lens]
    plans = [general([1] * S, lens, 8, nkv, None, **kw) for lens in (k_lens, first, last)]
    assert plans[0]["even"]
    for key in ("small", "splits"):
        assert np.array_equal(plans[0][key], plans[1][key]) and np.array_equal(plans[0][key], plans[2][key]), key


def plain_split(keys, extra, max_splits):
    """`split_evenly` one length at a time, block by block."""
    keys = [-(-int(k) // 128) * 128 for k in keys]
    share = max(128, -(-sum(keys) // extra))
    best = None
    for length in [max(keys)] + [int(share * f) for f in (1.0, 1.15, 1.35, 1.6, 2.0, 2.7, 4.0)]:
        ns = [min(-(-k // length), max_splits) for k in keys]
        cost = [-(-k // n) + planning.BLOCK_KEYS + planning.MERGE_KEYS * (n > 1) for k, n in zip(keys, ns)]
        blocks = sorted((c for c, n in zip(cost, ns) for _ in range(n)), reverse=True)
        end = max(sum(blocks) / extra, max(c * (i + 1) for i, c in enumerate(blocks[::extra])))
        if best is None or end < best[0]:
            best = (end, ns)
    return best[1]


def test_even_ranges_equal_the_plain_search():
    rng = np.random.default_rng(7)
    for _ in range(300):
        keys = rng.integers(1, int(2 ** rng.uniform(1, 15)) + 1, int(rng.integers(1, 200)))
        extra, most = int(rng.integers(1, 300)), int(rng.integers(1, 33))
        assert planning.split_evenly(keys, extra, most).tolist() == plain_split(keys, extra, most)


@pytest.mark.parametrize("S,pad", [(27, 32), (64, 64), (131, 192)])
def test_even_ranges_cost_the_host_little_more_than_equal_ones(S, pad):
    """Planning stands in front of every step whose contexts grew past a multiple of 128 keys (two of three steps at 131
    requests).  Without even ranges it takes some 25 us here, with them three times that; a search that goes through the
    blocks of every length takes seven."""
    import time
    k_lens = np.random.default_rng(S).integers(70, 3500, S).tolist()

    def best(slots):
        kw = dict(cluster_max=8, long_keys=600, slots=slots, pad_requests=pad, fixed_capacity=True)
        least = 1.0
        for _ in range(200):
            start = time.perf_counter()
            plan = general([1] * S, k_lens, 8, 8, None, **kw)
            least = min(least, time.perf_counter() - start)
        assert plan.get("even", False) == bool(slots)
        return least

    assert best(296) < 5 * best(0)


@pytest.mark.parametrize("nh,nkv,d", [(32, 4, 64), (32, 8, 128), (32, 32, 128), (64, 64, 256), (128, 8, 128), (16, 16, 16)])
def test_even_ranges_keep_the_scratch_within_its_bound(nh, nkv, d):
    """What the partial results of any even step take, replayed or not, decoding alone or mixed: the declared bound, or what
    one range per request takes where that is more."""
    G, kw = nh // nkv, dict(cluster_max=8, long_keys=600, slots=296)
    for pad in (8, 64, 160, 256):
        steps = [([1] * pad, dict(pad_requests=pad, fixed_capacity=True)), ([1] * pad, {}),
                 ([1] * (pad - 1) + [256], dict(pad_requests=pad, fixed_capacity=True, pad_tokens=512)),
                 ([1] * (pad - 1) + [max(1, 16 // G)], {})]
        for q_lens, more in steps:
            plan = general(q_lens, [4000] * pad, G, nkv, None, head_dim=d, **kw, **more)
            rows = max(plan["num_small_tokens"], 1)
            splits = plan["splits"].reshape(-1, 2)
            assert plan["max_splits"] >= splits[:, 0].max()
            if plan["even"] and plan["max_splits"] > 1:
                assert rows * nh * plan["max_splits"] * (d + 2) * 4 <= planning.EVEN_SCRATCH_BYTES
