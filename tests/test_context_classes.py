"""Decode steps of very many requests: which form of the decode attention a step takes, and that every step that replays a graph
has the plan that the graph was captured with."""

import types

import pytest
import torch

from paged_llm_b200.engine.runner import ModelRunner
from paged_llm_b200.kernels.ops import CudaOps


class HostOps(CudaOps):
    """The planning side of the kernel library, without a device."""

    def __init__(self):
        self.num_sms, self.compute_dtype, self.cluster_attention = 148, torch.bfloat16, True

    def _large_rows(self, head_dim):
        return 128


def graph_key(ops, plan_key, lens):
    runner = types.SimpleNamespace(ops=ops, plan_keys=[plan_key], GRAPH_BUCKETS=ModelRunner.GRAPH_BUCKETS)
    items = [types.SimpleNamespace(num_new_tokens=1, want=(0,), seq=types.SimpleNamespace(num_computed_tokens=n - 1)) for n in lens]
    return ModelRunner._graph_key_of(runner, items)


def test_three_blocks_up_to_4096_keys():
    ops = HostOps()
    for longest in (1, 4096):
        assert ops._three_blocks(112, 8, 4, 64, longest) and not ops._three_blocks(111, 8, 4, 64, longest)
        assert not ops.beyond_three_blocks(112, 8, 4, 64, longest)
    assert not ops._three_blocks(112, 8, 4, 64, 4097) and ops.beyond_three_blocks(112, 8, 4, 64, 4097)
    for n, nkv, group, d in ((111, 8, 4, 64), (112, 8, 16, 64), (112, 8, 4, 128)):
        assert not ops.beyond_three_blocks(n, nkv, group, d, 10 ** 6)
    ops.compute_dtype = torch.float32
    assert not ops.beyond_three_blocks(112, 8, 4, 64, 4097)


@pytest.mark.parametrize("plan_key", [(4, 8, None, 64), (8, 4, None, 64), (1, 32, None, 64), (4, 8, 512, 64), (4, 8, None, 128), (16, 4, None, 64)])
def test_a_key_has_one_plan(plan_key):
    """Sizes of the lists, splits and classes of the plan: the same for all steps with one key."""
    ops, seen = HostOps(), {}
    for n in (1, 8, 28, 63, 97, 112, 128, 193, 256):
        for lens in ([1] * n, [700] * n, [4095] * n, [4096] * n, [4097] * n, [30] * (n - 1) + [4096], [30] * (n - 1) + [4097], [9000] * n):
            key = graph_key(ops, plan_key, lens)
            group, nkv, window, d = plan_key
            plan = ops.plan_attention([1] * n, lens, group, nkv, window, d, pad_requests=key[1], fixed_capacity=True)
            shape = ModelRunner._plan_shapes({plan_key: plan})
            assert seen.setdefault(key, shape) == shape, (n, lens[-1])
    three = [k for k in seen if ops._three_blocks(k[1], plan_key[1], plan_key[0], plan_key[3])] if not plan_key[2] else []
    assert {k[1] for k in three} == {k[1] for k in three if len(k) == 3}, "both forms have been seen where there are two"
