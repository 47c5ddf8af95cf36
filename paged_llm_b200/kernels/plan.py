"""Work lists for the attention kernels, made on the host once per step.

A request with nq new tokens and G query heads per kv head has nq*G query rows
per kv head (row r = token r // G, head r % G).  Requests with at most
`small_rows` rows (decoding, or a portion of a very few tokens) go to the
split-context kernel: their keys are cut into `splits` ranges that run in
separate thread blocks and are merged afterwards, so that a few long requests
still fill the machine (the reference runs one program per query tile and never
splits the context: pagedllm/attention/triton_kernel.py:10-12, :120).  The
others are cut into tiles of `large_rows` rows.

An item is four int32: (request, tile or scratch base, split, splits).  For a
fixed request count and fixed lengths the plan is deterministic, so replaying a
step reproduces its logits bit for bit.
"""

from __future__ import annotations

import numpy as np


def wanted_splits(num_small: int, num_kv_heads: int, num_sms: int, max_splits: int) -> int:
    """Splits per request so that requests x kv heads x splits is about one
    thread block per SM (measured: more splits cost more in merging than they win)."""
    if num_small <= 0:
        return 1
    target_items = -(-num_sms // max(num_kv_heads, 1))
    return int(min(max_splits, max(1, -(-target_items // num_small))))


def long_context_splits(num_requests: int, num_kv_heads: int, num_sms: int, max_splits: int) -> int:
    return int(max(1, min(max_splits, (3 * num_sms) // max(1, num_requests * max(num_kv_heads, 1)))))


def is_long_context(num_requests: int, num_kv_heads: int, num_sms: int, max_splits: int, cluster_max: int,
                    long_keys: int, max_context: int) -> bool:
    """Whether a decode step of this shape is in the long-context class: the blocks of a cluster
    (at most `cluster_max` per request and kv head) would each walk more than `long_keys` keys.
    Such a step is split further, through the work list: about three blocks per SM, which is
    what is resident at a time and what it takes to keep memory busy with one block's latencies
    (measured on `attn_bf16_kernel`: 16 k context at batch 8, 2.05 ms per step as clusters of 5, 1.50 ms as 13 splits; the
    line has not been measured again for the kernel that head sizes 64 and 128 run now)."""
    if cluster_max <= 0:
        return False
    cluster = min(wanted_splits(num_requests, num_kv_heads, num_sms, max_splits), cluster_max)
    if long_context_splits(num_requests, num_kv_heads, num_sms, max_splits) <= cluster:
        return False                 # so many requests that the work list would not split further either
    return max_context > long_keys * cluster


# What a block costs beside its keys (its start, its query, the merge of its warps), and what the merge of the ranges of a
# request adds, in keys: 4 and 1.2 us where a block reads some 85 keys per us.  (Head size 64.  Other head sizes are planned
# with the same figures and two blocks per SM, whatever kernel they run; against a cluster or one range per request, us per
# layer: 20 requests of 300 to 3,500 keys, 8 kv heads of 16 30.1 -> 19.7, 8 of 32 35.7 -> 24.7, 8 of 96 73 -> 55, 8 of 256
# 182 -> 158; 64 of 100 to 700, 8 of 96 53.9 -> 39.9.  A window of 512 gains from 40 requests on: 15.6 -> 16.2 at 20.)
BLOCK_KEYS, MERGE_KEYS = 350, 100


def even_ranges(num_requests: int, num_kv_heads: int, num_sms: int, slots: int, max_splits: int) -> int:
    """For a step whose small items are cut into ranges of about equal length (`split_evenly`): how many ranges per kv head
    are resident at a time.  0: the step is not cut that way, since a block per request and kv head would leave SMs idle
    and every request is split alike (the cluster form, which merges without global memory)."""
    if slots <= 0 or wanted_splits(num_requests, num_kv_heads, num_sms, max_splits) > 1:
        return 0
    return max(1, slots // max(num_kv_heads, 1))


# Scratch for the partial results of such a step: bytes, and (row, range) pairs.
EVEN_SCRATCH_BYTES, EVEN_SCRATCH_ROWS = 36 << 20, 2048


def even_max_splits(scratch_rows: int, num_heads: int, head_dim: int, max_splits: int) -> int:
    """Ranges a request may have in such a step: as many as EVEN_SCRATCH_ROWS and EVEN_SCRATCH_BYTES have room for (a row and
    range takes a maximum, a sum and `head_dim` values of 4 bytes per query head), one if they have room for less."""
    rows = max(scratch_rows, 1)
    return int(max(1, min(max_splits, EVEN_SCRATCH_ROWS // rows, EVEN_SCRATCH_BYTES // (rows * num_heads * (head_dim + 2) * 4))))


# Contexts are rounded up to multiples of this many keys before they are cut: a plan then changes only when a context grows
# past another multiple, which is when a replayed step makes its plan anew, and never depends on the step it was made for.
GRAIN = 128
# Lengths of a range that `split_evenly` weighs, in even shares; the first stands for the longest context.
RANGE_LENGTHS = np.array([[1.0], [1.0], [1.15], [1.35], [1.6], [2.0], [2.7], [4.0]])


def split_evenly(keys: np.ndarray, extra: int, max_splits: int) -> np.ndarray:
    """Ranges per request so that the blocks of a step end at about the same time although the requests' contexts differ
    (131 to 3,500 keys in one batch: a block per request and kv head walks 3,500 keys alone while most others have long
    ended).  `extra` ranges per kv head are resident at a time, and fit the lists beside one per request; of a few lengths
    of a range, none below an even share, the one after which the last block should end first."""
    keys = (keys + (GRAIN - 1)) // GRAIN * GRAIN
    longest = int(keys.max())
    if longest <= GRAIN:
        return np.ones(len(keys), np.int32)
    share = max(GRAIN, -(-int(keys.sum()) // extra))
    # all lengths at once, a row each
    length = (share * RANGE_LENGTHS).astype(np.int64)
    length[0, 0] = longest
    ns = np.minimum((keys + (length - 1)) // length, max_splits)
    cost = (keys + (ns - 1)) // ns + BLOCK_KEYS + MERGE_KEYS * (ns > 1)
    # the blocks by falling cost (cost and number of a request's ranges in one word, so that one sort does), and how many
    # come up to each: the last block ends no earlier than an even share, nor than k blocks of which a place must take that many
    order = np.sort((-cost << 16) + ns, axis=1)
    cost, many = -(order >> 16), order & 0xFFFF
    upto = np.cumsum(many, axis=1)
    end = np.maximum((cost * many).sum(1) / extra, ((upto + (extra - 1)) // extra * cost).max(1))
    return ns[int(end.argmin())].astype(np.int32)


def even_items(ids: np.ndarray, base: np.ndarray, keys: np.ndarray, ns: np.ndarray, capacity: int | None) -> np.ndarray:
    """The list of such a step: the ranges of a request side by side, requests with long ranges first, filled up with
    items of no request to `capacity`."""
    order = np.argsort(-((keys + (GRAIN - 1)) // GRAIN * GRAIN // ns), kind="stable")
    total = int(ns.sum())
    if capacity is not None and total > capacity:
        raise PlanCapacityError(f"{total} small items for a capacity of {capacity}")
    heads = np.empty((len(ns), 4), np.int32)
    many = ns[order]
    heads[:, 0], heads[:, 1], heads[:, 3] = ids[order], base[order], many
    heads[:, 2] = many - np.cumsum(many)                  # minus the place of the request's first range
    small = np.empty((capacity if capacity is not None else total, 4), np.int32)
    small[:total] = np.repeat(heads, many, axis=0)
    small[:total, 2] += np.arange(total, dtype=np.int32)
    small[total:] = -1
    return small


def _plan_decode(S, S_pad, k_lens, num_kv_heads, min_split_keys, num_sms, max_splits, fixed_capacity,
                 cluster_max=0, long_keys=0, slots=0, num_heads=32, head_dim=64) -> dict:
    """The same plan for the common step in which every request brings one token, in array form."""
    n_req = S_pad if fixed_capacity else S
    long_context = is_long_context(n_req, num_kv_heads, num_sms, max_splits, cluster_max, long_keys,
                                   int(max(k_lens)) if len(k_lens) else 0)
    extra = max(1, slots // max(num_kv_heads, 1)) if long_context and slots > 0 \
        else even_ranges(n_req, num_kv_heads, num_sms, slots, max_splits)
    if extra:
        lk = np.asarray(k_lens, np.int64)
        most = even_max_splits(n_req, num_heads, head_dim, max_splits)
        ns = split_evenly(lk, extra, most)
        ids = np.arange(S, dtype=np.int32)                                       # (the scratch base too: one token each)
        small = even_items(ids, ids, lk, ns, S_pad + extra if fixed_capacity else None)
        splits = np.ones((S_pad, 2), np.int32)
        splits[:, 1] = 0
        splits[:S, 0] = ns
        splits[:S, 1] = ids
        return {"small": small.reshape(-1), "large": np.zeros(0, np.int32), "splits": splits.reshape(-1),
                "max_splits": int(most if fixed_capacity else ns.max()),
                "num_small_tokens": int(S_pad if fixed_capacity else S), "long_context": long_context, "even": True}
    want = long_context_splits(n_req, num_kv_heads, num_sms, max_splits) if long_context \
        else wanted_splits(n_req, num_kv_heads, num_sms, max_splits)
    lk = np.asarray(k_lens, np.int64)
    ns = np.maximum(1, np.minimum(want, -(-lk // min_split_keys))).astype(np.int32)
    splits = np.ones((S_pad, 2), np.int32)
    splits[:, 1] = 0
    splits[:S, 0] = ns
    splits[:S, 1] = np.arange(S, dtype=np.int32)
    total = int(ns.sum())
    seq = np.repeat(np.arange(S, dtype=np.int32), ns)
    first = np.cumsum(ns) - ns
    small = np.empty((total, 4), np.int32)
    small[:, 0] = seq
    small[:, 1] = seq                                   # scratch base: one token per request
    small[:, 2] = np.arange(total, dtype=np.int32) - np.repeat(first, ns).astype(np.int32)
    small[:, 3] = np.repeat(ns, ns)
    if fixed_capacity:
        cap = S_pad * want
        if cap > total:
            small = np.concatenate([small, np.full((cap - total, 4), -1, np.int32)])
    return {"small": small.reshape(-1), "large": np.zeros(0, np.int32), "splits": splits.reshape(-1),
            "max_splits": int(want), "num_small_tokens": int(S_pad if fixed_capacity else S),
            "long_context": long_context}


class PlanCapacityError(ValueError):
    """A step does not fit the fixed capacity its plan was asked for."""


def large_capacity(num_tokens: int, group_size: int, small_rows: int, large_rows: int) -> int:
    """An upper bound of the row tiles of the large items of any step of `num_tokens` tokens: every tile but a
    request's last is full, and a request with a large item has more than `small_rows` rows."""
    rows = num_tokens * group_size
    return rows // large_rows + rows // (small_rows + 1) + 1


def first_visible_key(pos: int, window: int | None, chunk: int | None) -> int:
    """The lowest key position the query at `pos` sees: the last `window` keys, and none before its chunk."""
    lo = max(0, pos - window + 1) if window else 0
    if chunk:
        lo = max(lo, pos - pos % chunk)
    return lo


def visible_keys(first_pos: int, context: int, window: int | None, chunk: int | None, keep_first: int | None = None) -> int:
    """How many keys the queries from `first_pos` on walk together: from the first one's lowest key to the end of the
    context, and the first `keep_first` keys of the request that lie in front of the window."""
    lo = first_visible_key(first_pos, window, chunk)
    return context - lo + (min(lo, keep_first) if window and keep_first else 0)


def plan_attention(q_lens, k_lens, group_size: int, num_kv_heads: int, window: int | None, *, small_rows: int,
                   large_rows: int, min_split_keys: int, num_sms: int, max_splits: int = 32,
                   pad_requests: int | None = None, fixed_capacity: bool = False, cluster_max: int = 0,
                   long_keys: int = 0, pad_tokens: int | None = None, chunk: int | None = None,
                   keep_first: int | None = None, slots: int = 0, head_dim: int = 64) -> dict:
    """`slots` > 0 (blocks that are resident at a time): steps of so many requests that none would be split, and
    long-context steps, are cut into ranges of about equal length instead (see `split_evenly`; `head_dim` says what the
    scratch for their partial results takes).

    `pad_tokens` (with `fixed_capacity`, for a step of mixed items that replays a captured graph): both lists
    get the capacity of any step of that many tokens and `pad_requests` requests, filled up with items of
    request -1 that the kernels skip."""
    S = len(q_lens)
    S_pad = pad_requests or S
    if pad_tokens is None and S and max(q_lens) == 1 and group_size <= small_rows and not window and not chunk:
        return _plan_decode(S, S_pad, k_lens, num_kv_heads, min_split_keys, num_sms, max_splits, fixed_capacity,
                            cluster_max, long_keys, slots, group_size * num_kv_heads, head_dim)
    small_ids = [s for s in range(S) if q_lens[s] * group_size <= small_rows]
    n_small = S_pad if fixed_capacity else len(small_ids)
    want = wanted_splits(n_small, num_kv_heads, num_sms, max_splits)
    cap = S_pad * want
    # (what a captured graph has baked in depends on its capacity alone, also where no request is small this time)
    extra = even_ranges(n_small, num_kv_heads, num_sms, slots, max_splits) if n_small else 0
    if extra:
        want = even_max_splits(S_pad * max(1, small_rows // group_size) if fixed_capacity else sum(q_lens[s] for s in small_ids),
                               group_size * num_kv_heads, head_dim, max_splits)
        cap = S_pad + extra
    n_keys = [visible_keys(k_lens[s] - q_lens[s], k_lens[s], window, chunk, keep_first) for s in small_ids]
    splits = np.ones((S_pad, 2), np.int32)
    splits[:, 1] = 0
    small = []
    small_arr = None
    scratch_base = 0
    if extra and small_ids:
        ids, keys, new = np.array(small_ids), np.array(n_keys, np.int64), np.array([q_lens[s] for s in small_ids])
        ns, upto = split_evenly(keys, extra, want), np.cumsum(new)
        splits[ids, 0], splits[ids, 1] = ns, upto - new
        scratch_base = int(upto[-1])
        small_arr = even_items(ids, upto - new, keys, ns, cap if fixed_capacity else None)
    else:
        for s, n in zip(small_ids, n_keys):
            ns = max(1, min(want, -(-n // min_split_keys)))
            splits[s] = (ns, scratch_base)
            for j in range(ns):
                small.append((s, scratch_base, j, ns))
            scratch_base += q_lens[s]
    large = []
    for s in range(S):
        rows = q_lens[s] * group_size
        if rows <= small_rows:
            continue
        tiles = -(-rows // large_rows)
        for t in range(tiles):
            last_tok = min(rows - 1, (t + 1) * large_rows - 1) // group_size
            large.append((k_lens[s] - q_lens[s] + last_tok, s, t))
    large.sort(key=lambda x: -x[0])                       # longest first
    if small_arr is None:
        small_arr = np.array(small, np.int32).reshape(-1, 4)
    if fixed_capacity:
        if len(small_arr) > cap:
            raise PlanCapacityError(f"{len(small_arr)} small items for a capacity of {cap}")
        pad = np.full((cap - len(small_arr), 4), -1, np.int32)
        small_arr = np.concatenate([small_arr, pad]) if len(pad) else small_arr
    large_arr = np.array([(s, t, 0, 1) for _, s, t in large], np.int32).reshape(-1, 4)
    small_tokens = int(scratch_base) if not fixed_capacity else int(S_pad)
    if pad_tokens is not None and fixed_capacity:
        cap = large_capacity(pad_tokens, group_size, small_rows, large_rows)
        if len(large_arr) > cap or sum(q_lens) > pad_tokens:
            raise PlanCapacityError(f"{len(large_arr)} large items for a capacity of {cap}")
        large_arr = np.concatenate([large_arr, np.full((cap - len(large_arr), 4), -1, np.int32)])
        small_tokens = int(S_pad) * max(1, small_rows // group_size)       # a small item may bring several tokens
        if scratch_base > small_tokens:
            raise PlanCapacityError(f"{scratch_base} tokens of small items for {small_tokens} scratch rows")
    return {
        "small": small_arr.reshape(-1),
        "large": large_arr.reshape(-1),
        "splits": splits.reshape(-1),
        "max_splits": int(want),
        "num_small_tokens": small_tokens,
        "long_context": False,
        "even": bool(extra),
    }
