"""Units of the scatter that change hands as often as they can: 2^24 keys that
fall into a few partitions, so that every warp of a CTA fills and frees the same
units, for each unit size; every tuple arrives whole and once."""
import numpy as np
import pytest
import torch

from partitioned_join_b200 import DIGIT_RAW, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("bits", [3, 8, 12])
@pytest.mark.parametrize("used", [1, 2, 5])
def test_units_change_hands_whole(dtype, bits, used):
    n, words, P = (1 << 24) + 77, 2 if dtype == np.int32 else 4, 1 << bits
    g = torch.Generator(device="cuda")
    g.manual_seed(bits * 10 + used)
    # row r's key names the row in the bits above the digit, so a torn tuple shows
    digit = torch.randint(0, used, (n,), generator=g, device="cuda", dtype=torch.int64) * (P // 8 or 1) % P
    keys = (torch.arange(n, device="cuda") * P + digit).to(torch.int32 if dtype == np.int32 else torch.int64)
    plan = api.plan_default(n, n, np.dtype(dtype).itemsize)
    plan.bits1, plan.wc_tuples, plan.digit_mode = bits, 8 // words, DIGIT_RAW
    tuples, offsets = api.partition(keys, plan)
    rec = tuples[: int(offsets[-1]) * words].view(-1, words)
    rows = rec[:, -1].long()
    real = rows >= 0
    assert torch.equal(torch.sort(rows[real])[0], torch.arange(n, device="cuda"))
    got = rec[real]
    if words == 4:
        lo = got[:, 0].long() & 0xffffffff
        assert torch.equal(lo | (got[:, 1].long() << 32), keys[rows[real]])
    hashes = api.hash_keys(keys)
    assert torch.equal(got[:, 0 if words == 2 else 2], hashes.view(torch.int32)[rows[real]])
    part = torch.repeat_interleave(torch.arange(P, device="cuda"), torch.diff(offsets))
    assert torch.equal(part[real], (keys[rows[real]].long() & (P - 1)))


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_second_pass_item_of_more_tuples_than_a_count_holds(dtype):
    # one first-pass partition holds every key, so one second-pass item places
    # more tuples than the 24 bits of a unit's count could number
    n, words = (1 << 25) + 5, 2 if dtype == np.int32 else 4
    keys = torch.full((n,), 12345, dtype=torch.int32 if dtype == np.int32 else torch.int64, device="cuda")
    plan = api.plan_default(n, n, np.dtype(dtype).itemsize)
    plan.passes, plan.bits1, plan.bits2, plan.wc_tuples = 2, 10, 2, 8 // words
    plan.table_mode, plan.table_capacity = 0, 4096
    tuples, offsets = api.partition(keys, plan)
    assert int((torch.diff(offsets) > 0).sum()) == 1
    rows = tuples[: int(offsets[-1]) * words].view(-1, words)[:, -1]
    real = rows[rows >= 0].long()
    assert real.numel() == n and torch.equal(torch.sort(real)[0], torch.arange(n, device="cuda"))
