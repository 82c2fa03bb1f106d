"""The sampling kernel's search by buckets and the descent behind it, where one takes over from the other: rows in which so many
tokens share all of the mass, exactly, that the walk can be done in whole numbers here."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from spissa_b200.csrc import lib
    return lib


@pytest.mark.parametrize("V", [1030, 32000, 128256, 140001])
@pytest.mark.parametrize("equal", [1, 2, 1023, 1024, 1025])
@pytest.mark.parametrize("top_k,top_p", [(0, 1.0), (0, 0.5), (700, 1.0), (700, 0.9)])
def test_equal_tokens_are_walked_in_whole_numbers(K, V, equal, top_k, top_p):
    rows = 5
    g = torch.Generator().manual_seed(V + equal)
    at = torch.stack([torch.randperm(V, generator=g)[:equal].sort().values for _ in range(rows)])
    logits = torch.full((rows, V), -200.0)                     # exp(-200 - 0) is zero in 32 bits
    logits.scatter_(1, at, 0.0)
    p = float(np.float32(1.0) / np.float32(equal))             # exp(0) over the sum of so many ones
    weight = math.floor(p * 2 ** 44)
    count = min(equal, top_k) if top_k and top_k < V else equal
    reach = int(np.float32(top_p) * np.float32(2 ** 44))
    if weight * equal >= reach:
        count = min(count, max(1, -(-reach // weight)))
    us = [0.0, 1.0 / 2 ** 24, 0.25, 0.7310585618019104, (2 ** 24 - 1) / 2 ** 24]
    want = []
    for r, u in enumerate(us):
        target = (weight * count * int(u * 2 ** 24)) >> 24
        want.append(int(at[r, max(1, -(-target // weight)) - 1]))
    scratch = torch.empty(K.sample_scratch_keys(rows, V), dtype=torch.int64, device=DEV)
    for draws in (us, torch.tensor(us, device=DEV)):           # with the launch, and from the device
        out = torch.empty(rows, dtype=torch.int32, device=DEV)
        K.sample_rows(logits.to(DEV), 1.0, top_k, top_p, draws, scratch, out)
        assert out.tolist() == want


def test_draws_that_do_not_fit(K):
    logits = torch.zeros(65, 100, device=DEV)
    scratch, out = torch.empty(K.sample_scratch_keys(65, 100), dtype=torch.int64, device=DEV), torch.empty(65, dtype=torch.int32, device=DEV)
    with pytest.raises(K.KernelError, match="do not go with a launch"):
        K.sample_rows(logits, 1.0, 0, 1.0, [0.5] * 65, scratch, out)
    with pytest.raises(K.KernelError):
        K.sample_rows(logits, 1.0, 0, 1.0, [0.5] * 3, scratch, out)
    K.sample_rows(logits, 1.0, 0, 1.0, torch.full((65,), 0.5, device=DEV), scratch, out)
    assert out.tolist() == [49] * 65


@pytest.mark.parametrize("V,equal", [(270001, 266310), (32000, 31999), (128256, 128256), (2000, 2000)])
@pytest.mark.parametrize("top_k,top_p", [(0, 1.0), (0, 0.5), (50, 0.9), (1500, 0.3), (1500, 1.0)])
def test_many_equal_tokens(K, V, equal, top_k, top_p):
    """All of the mass in one bucket: its sums pass 32 bits in every slice (266,310 tokens), and the search goes on from it."""
    if equal == 266310:
        low = int(np.float32(1.0 / 266310).view(np.uint32)) & ((1 << 18) - 1)
        assert low * (equal // 8) > 2 * 2 ** 32
    test_equal_tokens_are_walked_in_whole_numbers(K, V, equal, top_k, top_p)


@pytest.mark.parametrize("rows", [3, 20])
@pytest.mark.parametrize("std", [0.02, 0.5])
@pytest.mark.parametrize("top_k,top_p", [(0, 0.95), (50, 0.9), (9000, 0.4), (9000, 1.0)])
def test_nearly_equal_tokens(K, rows, std, top_k, top_p):
    """More than 1,024 tokens in the bucket of an answer. The walk in 64 bits says between which tokens it lies: a float32
    probability is off by some 2^-22, which moves a running total by as much of itself."""
    V = 32000
    g = torch.Generator().manual_seed(rows)
    logits = torch.randn(rows, V, generator=g) * std
    us = [(i + 0.5) / rows for i in range(rows)]
    us = [int(u * 2 ** 24) / 2 ** 24 for u in us]
    scratch = torch.empty(K.sample_scratch_keys(rows, V), dtype=torch.int64, device=DEV)
    out = torch.empty(rows, dtype=torch.int32, device=DEV)
    K.sample_rows(logits.to(DEV), 1.0, top_k, top_p, us, scratch, out)
    p, order = torch.softmax(logits.double(), dim=-1).sort(dim=-1, descending=True, stable=True)
    run = p.cumsum(dim=-1)
    for r, (u, token) in enumerate(zip(us, out.tolist())):
        at = int((order[r] == token).nonzero())
        kept = min(float(run[r, top_k - 1]) if top_k else 1.0, max(top_p, float(run[r, 0])))
        slack = 2.0 ** -19 + 2 * float(p[r, 0])                        # the kept mass ends behind the token that reaches top_p
        assert float(run[r, at]) >= u * kept - slack and float(run[r, at] - p[r, at]) <= u * kept + slack


@pytest.mark.parametrize("rows", [6, 18])
@pytest.mark.parametrize("head", [40, 900])
def test_answers_of_few_and_of_many_tokens_in_one_row(K, rows, head):
    """The top_k boundary lies among 2,000 equal tokens (the descent), the draw among tokens of their own probabilities (by bins)
    or among the equal ones. Every draw is aimed at the middle of a token's mass: 1e-4 of the total, a thousand times what the
    32-bit probabilities are off by."""
    V, top_k = 5003, 1500
    g = torch.Generator().manual_seed(head)
    at = torch.randperm(V, generator=g)
    logits = torch.full((V,), -200.0)
    logits[at[:head]] = 1.0 + torch.arange(head, 0, -1) * (0.5 / head)
    logits[at[head:head + 2000]] = 0.0
    p, order = torch.softmax(logits.double(), dim=-1).sort(descending=True, stable=True)
    run = p.cumsum(dim=-1)
    kept = float(run[top_k - 1])
    want = [0, 5, head - 1, head, (head + top_k) // 2, top_k - 1] * (rows // 6)
    us = [int((float(run[j]) - float(p[j]) / 2) / kept * 2 ** 24) / 2 ** 24 for j in want]
    scratch = torch.empty(K.sample_scratch_keys(rows, V), dtype=torch.int64, device=DEV)
    out = torch.empty(rows, dtype=torch.int32, device=DEV)
    K.sample_rows(logits.repeat(rows, 1).to(DEV), 1.0, top_k, 1.0, us, scratch, out)
    assert out.tolist() == [int(order[j]) for j in want]
