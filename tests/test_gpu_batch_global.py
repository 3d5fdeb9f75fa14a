"""Batches whose joins take tables in L2 (unique build keys): several groups of
tables, small and large items, misaligned columns, joins without capacity, and
the same pairs as the partitioned and direct kernels (large_batched = 0)."""
import numpy as np
import pytest
import torch

from oracle import oracle
from partitioned_join_b200 import api

pytestmark = pytest.mark.gpu


def batch(seed, sizes, dtype):
    rng = np.random.default_rng(seed)
    pairs, host = [], []
    for nb, np_, shift in sizes:
        b = (rng.permutation(2 * nb + 1)[:nb].astype(np.int64) * 0x100000001B3).astype(dtype)
        p = np.where(rng.random(np_) < 0.7, rng.choice(b, np_), -1 - rng.integers(0, 1 << 30, np_)).astype(dtype)
        # a column that starts `shift` elements into its allocation
        cols = [torch.from_numpy(np.concatenate([np.zeros(shift, dtype), c])).cuda()[shift:] for c in (b, p)]
        pairs.append(tuple(cols))
        host.append((b, p))
    return pairs, host


def check(bj, host):
    for (br, pr), (b, p) in zip(bj.results(), host):
        got = oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy())
        assert np.array_equal(got, oracle.sorted_pairs(*oracle.inner_join(b, p, True)))


SMALL = [(1, 1, 0), (255, 511, 1), (256, 512, 0), (257, 513, 3), (1023, 2047, 0), (4096, 30000, 1)]
LARGE = [(1 << 20, 2049, 0), (700001, 2000003, 1), (1 << 20, 4097, 0), (900001, 1 << 20, 0), (3, 2047, 1),
         (1 << 20, 70001, 3), (1 << 20, 5, 0)]   # int32 tables of 16 MB: two groups


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("sizes", [SMALL, LARGE], ids=["small_items", "two_groups"])
def test_batch_of_global_tables(dtype, sizes):
    pairs, host = batch(len(sizes), sizes, dtype)
    bj = api.BatchJoiner(pairs)
    for _ in range(2):
        bj.launch()
    check(bj, host)
    bj.config.large_batched = 0
    bj.config.direct_max_build = 4096
    if all(s == 0 for _, _, s in sizes):   # (the partitioned joins take 16-byte aligned columns)
        bj.prepare()
        bj.launch()
        check(bj, host)


def test_batch_capacity_of_one_join_is_reported():
    pairs, host = batch(9, SMALL, np.int32)
    bj = api.BatchJoiner(pairs)
    bj.launch()
    torch.cuda.synchronize()
    full = bj.count.clone()
    bj.outs[4].capacity = 10
    bj.prepare()
    bj.launch()
    with pytest.raises(Exception) as e:
        bj.results()
    assert "capacity" in str(e.value)
    assert torch.equal(bj.count, full)
