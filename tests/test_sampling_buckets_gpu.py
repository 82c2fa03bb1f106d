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
