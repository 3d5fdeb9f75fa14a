"""Batches of unique joins with few probe rows for their build sides: those go to
the direct kernel or are partitioned together, not to tables in L2, beside joins
that do take tables -- any alignment, any mix, the oracle's pairs."""
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
        b = ((np.arange(nb, dtype=np.int64) * 2 + 1) * 0x100000001B3).astype(dtype)
        rng.shuffle(b)
        p = np.where(rng.random(np_) < 0.7, rng.choice(b, np_), (2 * rng.integers(0, 1 << 30, np_)).astype(dtype))
        cols = [torch.from_numpy(np.concatenate([np.zeros(shift, dtype), c])).cuda()[shift:] for c in (b, p.astype(dtype))]
        pairs.append(tuple(cols))
        host.append((b, p.astype(dtype)))
    return pairs, host


def check(bj, host):
    for (br, pr), (b, p) in zip(bj.results(), host):
        got = oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy())
        assert np.array_equal(got, oracle.sorted_pairs(*oracle.inner_join(b, p, True)))


SMALL = [(4096, 500, 0), (8000, 8000, 1), (300, 1, 0), (20001, 3, 3)]               # all direct
MIXED = SMALL + [(4096, 60000, 1), (70001, 300000, 0)]                              # few direct rows: all tables
MANY = [(16000, 100, i % 4) for i in range(64)] + [(4096, 60000, 1)]                # direct, and a table
LARGE = [(1 << 21, 5000, 1), (1 << 21, 70001, 0), (3000001, 1, 3), (1000, 9000, 0), (900000, 4000000, 0)]
WIDE = [((1 << 22) - i, 3000 + i, i % 2) for i in range(6)] + [(50000, 400000, 0)]  # 8-byte keys: only this many rows


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("sizes", [SMALL, MIXED, MANY, LARGE, WIDE], ids=["small", "mixed", "many", "large", "wide"])
def test_few_probe_rows(dtype, sizes):
    pairs, host = batch(len(sizes), sizes, dtype)
    bj = api.BatchJoiner(pairs)
    for _ in range(2):
        bj.launch()
    check(bj, host)
    g = bj.graph()
    bj.count.zero_()
    g.replay()
    torch.cuda.synchronize()
    check(bj, host)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_a_workspace_for_no_direct_joins_holds_every_limit(dtype):
    pairs, host = batch(3, MIXED + LARGE, dtype)
    bj = api.BatchJoiner(pairs)
    sizes = {}
    for limit in (0, 300, 4096, 16384, 20480, 40960):
        bj.config.direct_max_build = limit
        sizes[limit] = bj._ws_size(bj.config)
    assert max(sizes.values()) == sizes[0], sizes
    for limit in sizes:
        bj.config.direct_max_build = limit
        bj.prepare()
        bj.launch()
        check(bj, host)


def test_few_probe_rows_cost_no_table():
    # eight joins of 2^21 x 2^15 4-byte rows: 412 us by tables, 234 partitioned together
    pairs, host = batch(4, [(1 << 21, 1 << 15, 0)] * 8, np.int32)
    bj = api.BatchJoiner(pairs)
    g = bj.graph()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t = []
    for _ in range(10):
        e0.record()
        g.replay()
        e1.record()
        torch.cuda.synchronize()
        t.append(e0.elapsed_time(e1))
    assert min(t) < 0.32, t
    check(bj, host)


def test_capacity_of_a_join_off_the_tables_is_reported():
    pairs, host = batch(5, LARGE, np.int32)
    bj = api.BatchJoiner(pairs)
    bj.launch()
    torch.cuda.synchronize()
    full = bj.count.clone()
    bj.outs[1].capacity = 10
    bj.prepare()
    bj.launch()
    with pytest.raises(Exception) as e:
        bj.results()
    assert "capacity" in str(e.value)
    assert torch.equal(bj.count, full)
