"""The scatter over 4096 partitions on both sides of the line between units and
rounds (16 tuples a partition and item), and under skew that fills one unit again
and again: every row lands once, in its partition."""
import numpy as np
import pytest
import torch

from oracle import oracle
from partitioned_join_b200 import DIGIT_HASH, TABLE_BUCKET, api

pytestmark = pytest.mark.gpu

LINE = 148 * 16 * 4096  # rows from which an item has 16 tuples a partition


def hashes(keys):
    return torch.from_numpy(oracle.hash_keys(keys.cpu().numpy()).astype(np.int64)).cuda()


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("kind", ["uniform", "half_one_key"])
@pytest.mark.parametrize("n", [1, 148 * 16, 100003, LINE - 2368, LINE + 4, LINE + 1000003])
@pytest.mark.parametrize("bits", [11, 12])
def test_every_row_lands_once(dtype, kind, n, bits):
    g = torch.Generator(device="cuda").manual_seed(n + bits)
    keys = torch.randint(-(1 << 31), (1 << 31) - 1, (n,), device="cuda", generator=g).to(dtype)
    if kind == "half_one_key":
        keys[torch.rand(n, device="cuda", generator=g) < 0.5] = 12345
    words = keys.element_size() // 2
    plan = api.plan_default(n, n, keys.element_size())
    plan.passes, plan.bits1, plan.bits2, plan.digit_mode = 1, bits, 0, DIGIT_HASH
    plan.table_mode, plan.table_capacity, plan.wc_tuples = TABLE_BUCKET, 8192, 8 // words
    tuples, off = api.partition(keys, plan)
    total = int(off[-1])
    rec = tuples[: total * words].view(-1, words)
    rows = rec[:, -1].long()
    real = rows >= 0
    assert bool((rows[~real] == -1).all())
    assert int(real.sum()) == n and bool((torch.sort(rows[real])[0] == torch.arange(n, device="cuda")).all())
    h = hashes(keys)
    assert bool((rec[real][:, 0 if words == 2 else 2].long() & 0xFFFFFFFF == h[rows[real]]).all())
    part = torch.repeat_interleave(torch.arange(1 << bits, device="cuda"), off[1:] - off[:-1])
    assert bool((part[real] == h[rows[real]] >> (32 - bits)).all())
    assert bool(((off[1:] - off[:-1]) % plan.wc_tuples == 0).all())


@pytest.mark.parametrize("heavy", [False, True])
@pytest.mark.parametrize("n_probe", [5000, LINE // 16, LINE + 100])
def test_joins_over_4096_partitions(heavy, n_probe):
    nb = 1 << 21
    b, p, _ = api.generate_tables(nb, n_probe, torch.int64, 1 << 40, 0.8, True, 1.25, 7)
    plan = api.plan_default(nb, n_probe, 8)
    plan.passes, plan.bits1, plan.bits2, plan.digit_mode = 1, 12, 0, DIGIT_HASH
    plan.table_mode, plan.table_capacity, plan.wc_tuples = TABLE_BUCKET, 8192, 2
    if heavy:
        k, c = torch.unique(p, return_counts=True)
        plan.set_heavy(k[torch.argsort(-c)[:40]].tolist())
    br, pr = api.partitioned_join(b, p, plan=plan)
    assert bool((b[br.long()] == p[pr.long()]).all())
    assert torch.equal(torch.sort(pr.long())[0], torch.nonzero(torch.isin(p, b)).flatten())
