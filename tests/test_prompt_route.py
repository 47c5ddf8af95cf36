"""Which steps leave the rotation of their queries to the kernel of the prompt tiles, decided on the host."""

import types

import pytest
import torch

from paged_llm_b200.kernels.ops import CudaOps

NH, NKV, D, T = 8, 2, 64, 40


class Recorder(CudaOps):
    """The route of `qkv_attention` alone: every kernel behind it is noted, none is launched."""

    def __init__(self):
        self.compute_dtype, self.use_skinny, self.cluster_attention, self.rope_in_attention = torch.bfloat16, True, True, True
        self.calls = []

    def _prompt_tiles_rotate(self, nh, nkv, d, kv, position):
        return True

    def linear(self, h, w):
        return torch.zeros(h.shape[0], w.shape[0])

    def rope_kv_write(self, qkv, nh, nkv, d, position, ctx, kv, block_table, write=True, value_from_key=False, rotated_later=0,
                      early=False):
        self.calls.append(("rope_kv_write", rotated_later, early))

    def qkv_rope_write(self, h, w_qkv, nh, nkv, d, position, ctx, kv, block_table, write=True, value_from_key=False, early=False):
        self.calls.append(("qkv_rope_write", 0, early))
        return self.linear(h, w_qkv)

    def paged_attention(self, qkv, nh, nkv, d, kv, block_table, ctx, scale, window, softcap=None, slopes=None, rope=None, chunk=None,
                        tile_rope=None):
        self.calls.append(("paged_attention", rope is not None, tile_rope is not None, window, chunk))


def route(ops, tokens=T, n_large=3, window=None, chunk=None, pairing="half", rotary_dim=D, page=16, **how):
    plan = types.SimpleNamespace(n_small=0 if n_large else 1, n_large=n_large, long_context=False, even=False, max_splits=1)
    key = (NH // NKV, NKV, window, D) if not chunk else (NH // NKV, NKV, window, D, chunk)
    ctx = types.SimpleNamespace(num_tokens=tokens, num_seqs=1, attention_plans={key: plan}, host=types.SimpleNamespace(q_lens=[tokens if n_large else 1]))
    position = types.SimpleNamespace(pairing=pairing, rotary_dim=rotary_dim)
    kv = torch.zeros(1, 2, NKV, page, D, dtype=torch.bfloat16)
    ops.calls.clear()
    ops.qkv_attention(torch.zeros(tokens, 128, dtype=torch.bfloat16), torch.zeros((NH + 2 * NKV) * D, 128, dtype=torch.bfloat16), NH, NKV, D,
                      position, ctx, kv, None, D ** -0.5, window, chunk=chunk, **how)
    return list(ops.calls)


@pytest.mark.parametrize("window,chunk,page", [(None, None, 16), (None, None, 64), (None, None, 8), (32, None, 16), (None, 64, 16)])
def test_prompt_tiles_rotate(window, chunk, page):
    """... and the rotation overlaps its neighbours where all items run kernels that gain by it."""
    early = window is None and chunk is None and page % 16 == 0
    assert route(Recorder(), window=window, chunk=chunk, page=page) == [("rope_kv_write", CudaOps.SMALL_ROWS, early),
                                                                        ("paged_attention", False, True, window, chunk)]


@pytest.mark.parametrize("how,early", [(dict(write=False), True), (dict(softcap=30.0), False), (dict(slopes=torch.ones(NH)), False),
                                       (dict(value_from_key=True), True), (dict(pairing="interleaved"), True),
                                       (dict(rotary_dim=D // 2), True), (dict(tokens=16), False)])
def test_steps_that_do_not(how, early):
    assert route(Recorder(), **how) == [("qkv_rope_write", 0, early), ("paged_attention", False, False, None, None)]


def test_other_kernels_behind_the_rotation():
    """Where the prompt tiles run a kernel that does not rotate (float32, other head sizes, other pages), nothing starts early."""
    ops = Recorder()
    ops._prompt_tiles_rotate = lambda *a: False
    assert route(ops) == [("qkv_rope_write", 0, False), ("paged_attention", False, False, None, None)]


@pytest.mark.parametrize("n_large", [0, 3])
def test_the_switch_turns_both_forms_off(n_large):
    ops = Recorder()
    assert any(c[0] == "paged_attention" and (c[1] or c[2]) for c in route(ops, n_large=n_large))
    ops.rope_in_attention = False
    assert route(ops, n_large=n_large) == [("qkv_rope_write", 0, True), ("paged_attention", False, False, None, None)]
