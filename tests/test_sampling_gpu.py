"""The filtered draw against an oracle that keeps what the filter keeps, token for token: rows whose candidates just fit, just
fill and just overflow the kernel's list, ties with the threshold (also where they straddle the edge of a bin of the
histogram that finds the candidates), masked tokens and flat rows."""

import math

import numpy as np
import pytest
import torch

from tests.plain_sampling import uniforms

pytestmark = pytest.mark.gpu
LIST = 2048                                    # candidates of a row that the kernel gathers at most


@pytest.fixture(scope="module")
def ops():
    from paged_llm_b200.kernels.ops import CudaOps
    return CudaOps("cuda")


def draws(row, temperature, top_k, top_p, seeds, counter):
    """Per seed the tokens that a correct draw may return.  logit / T is one float32 product; everything else is 64 bits.
    More than one token: scores within 1e-4 of the best (the kernel's logarithms are float32: errors of some 1e-6 on scores
    of up to 30), or a top-p threshold within 1e-6 of the mass (float32 exponentials)."""
    x = row * (np.float32(1) / np.float32(temperature))
    keep = np.ones(row.size, bool)
    if 0 < top_k < row.size:
        keep &= x >= np.sort(x)[-top_k]
    limits = [keep]
    if top_p < 1.0:
        p = np.exp(x.astype(np.float64) - float(x.max()))
        values, inverse, counts = np.unique(-x, return_inverse=True, return_counts=True)
        mass = np.bincount(inverse, weights=p)
        above = (np.cumsum(mass) - mass)[inverse] / p.sum()                 # mass of the larger tokens
        limits = [keep & (above <= np.float32(top_p) + e) for e in (-1e-6, 1e-6)]
    out = []
    for seed in seeds:
        score = x - np.log(-np.log(uniforms(int(seed), counter, row.size).astype(np.float64)))
        may = set()
        for kept in limits:
            s = np.where(kept, score, -np.inf)
            may |= set(np.flatnonzero(s >= s.max() - 1e-4).tolist())
        out.append(may)
    return out


def check(ops, row, temperature, top_k, top_p, rows=64):
    seeds = np.arange(1000, 1000 + rows, dtype=np.uint64)
    logits = torch.from_numpy(row).cuda().expand(rows, row.size).contiguous()
    got = ops.sample(logits, np.full(rows, temperature, np.float32), np.full(rows, top_k, np.int32), np.full(rows, top_p, np.float32),
                     seeds, np.full(rows, 9, np.uint64)).tolist()
    for r, (token, may) in enumerate(zip(got, draws(row, temperature, top_k, top_p, seeds, 9))):
        assert token in may, f"row {r}: {token} instead of one of {sorted(may)}"
    return got


@pytest.mark.parametrize("rows", [16, 64, 160])                # eight blocks, two and one per row
def test_ties_on_the_edge_of_a_bin(ops, rows):
    """Tokens of two adjacent logits whose products with 1 / T round to the same value, eight bins (of 1/8) below the largest
    token: they tie, so both kinds stay, although the exact products lie on the two sides of the bin's edge."""
    T = 1.1
    inv = np.float32(1) / np.float32(T)
    top, lower, upper = np.float32(8.0), np.float32(6.487499713897705), np.float32(6.487500190734863)
    assert lower * inv == upper * inv == top * inv - np.float32(11 / 8)
    assert float(lower) * float(inv) < float(lower * inv) < float(upper) * float(inv)
    row = np.full(20000, -50.0, np.float32)
    row[5::300] = lower                                        # 67 of each, in both halves of the row
    row[7::300] = upper
    row[11] = top
    got = check(ops, row, T, 20, 1.0, rows)
    assert any(row[t] == lower for t in got) and any(row[t] == upper for t in got)


@pytest.mark.parametrize("count", [LIST - 1, LIST, LIST + 1, 3 * LIST])
@pytest.mark.parametrize("top_k,top_p", [(LIST - 1, 1.0), (LIST, 1.0), (LIST + 1, 1.0), (0, 0.95), (40, 0.7)])
@pytest.mark.parametrize("same", [True, False])
def test_candidates_around_the_size_of_the_list(ops, count, top_k, top_p, same):
    rng = np.random.default_rng(count)
    row = np.full(30000, -math.inf, np.float32)
    at = rng.permutation(row.size)[:count]
    row[at] = 3.0 if same else rng.uniform(-9, 9, count).astype(np.float32)
    check(ops, row, 0.7, top_k, top_p)


@pytest.mark.parametrize("rows", [16, 64, 160])
@pytest.mark.parametrize("kind", ["flat", "peaked", "ties", "masked"])
@pytest.mark.parametrize("top_k,top_p", [(50, 0.9), (0, 0.9), (3000, 1.0), (1, 1.0), (0, 0.999)])
def test_draws_are_those_of_the_filter(ops, rows, kind, top_k, top_p):
    rng = np.random.default_rng(3)
    row = (rng.standard_normal(40001) * {"flat": 1e-4, "peaked": 6.0}.get(kind, 2.0)).astype(np.float32)
    if kind == "ties":
        row = np.round(row * 2) / np.float32(2)
    if kind == "masked":
        row[1000:] = -math.inf
    check(ops, row, 0.7, top_k, top_p, rows)


def test_more_rows_while_copies_are_in_flight():
    """A draw whose parameters are still to be copied, behind a long kernel, when a draw of more rows takes larger buffers: what
    the pool of pinned memory hands out next must not be the buffer that the copy reads."""
    from paged_llm_b200.kernels.ops import CudaOps
    ops, rows, V = CudaOps("cuda"), 8, 1000
    g = torch.Generator(device="cuda").manual_seed(5)
    logits = torch.empty(400, V, device="cuda").normal_(0.0, 0.3, generator=g)
    args = lambda n: (np.full(n, 1.0, np.float32), np.zeros(n, np.int32), np.full(n, 1.0, np.float32),
                      np.arange(n, dtype=np.uint64) + np.uint64(77), np.full(n, 9, np.uint64))
    want = CudaOps("cuda").sample(logits[:rows], *args(rows)).tolist()
    # (what is allocated behind the long kernel comes from the pools: an allocation by the driver might wait for it)
    spare = [torch.empty(n, dtype=torch.int64, pin_memory=True) for n in [1024] * 16 + [2800] * 4]
    spare.append(torch.empty(1 << 18, device="cuda"))
    del spare
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)                                  # some 0.1 s
    got = ops.sample(logits[:rows], *args(rows))
    many = ops.sample(logits, *args(400))
    taken = [torch.zeros(1024, dtype=torch.int64, pin_memory=True) for _ in range(32)]
    for t in taken:                                                 # (parameters of eight rows too, with another seed)
        t[:2 * rows] = 123456789
        t.view(torch.float32)[4 * rows:6 * rows] = 1.0
    torch.cuda.synchronize()
    assert got.tolist() == want and many[:rows].tolist() == want and len(taken) == 32
