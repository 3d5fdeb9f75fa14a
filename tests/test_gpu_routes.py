"""Routes that default calls of ordinary sizes no longer reach, checked pair by
pair: batches of unique joins partitioned together (build sides above 2^22 rows)
and by the direct kernel, planned heavy keys on a small build side, and joins
whose columns are partitioned in several item groups."""
import numpy as np
import pytest
import torch

from oracle import oracle
from partitioned_join_b200 import (DIGIT_HASH, SPLIT_HASH, SPLIT_POSITION, TABLE_BUCKET, TABLE_COMPACT, TABLE_EXACT, api,
                                   datagen)

pytestmark = pytest.mark.gpu


def expect(b, p, unique=True):
    return oracle.sorted_pairs(*oracle.inner_join(b, p, unique))


def batch(seed, sizes, dtype, unique=True):
    rng = np.random.default_rng(seed)
    pairs, host = [], []
    for nb, np_ in sizes:
        k = rng.permutation(2 * nb + 1)[:nb] if unique else rng.integers(0, nb // 2 + 1, nb)
        b = (k.astype(np.int64) * 0x100000001B3).astype(dtype)
        p = np.where(rng.random(np_) < 0.7, rng.choice(b, np_), -1 - rng.integers(0, 1 << 30, np_)).astype(dtype)
        pairs.append((torch.from_numpy(b).cuda(), torch.from_numpy(p).cuda()))
        host.append((b, p))
    return pairs, host


def check(bj, host, unique=True):
    for (br, pr), (b, p) in zip(bj.results(), host):
        assert np.array_equal(oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy()), expect(b, p, unique))


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_batch_of_unique_joins_partitioned_together(dtype):
    # two joins above the tables' 2^22 build rows share the partitioned launches; one takes a table
    pairs, host = batch(1, [((1 << 22) + 1, 300001), (70001, 200000), (5000003, 1 << 20)], dtype)
    bj = api.BatchJoiner(pairs)
    assert bj.config.large_batched == 1
    for delta in (0, 1):
        bj.config.large_bits_delta = delta
        bj.prepare()
        bj.launch()
        check(bj, host)
    g = bj.graph()
    bj.count.zero_()
    g.replay()
    torch.cuda.synchronize()
    check(bj, host)


@pytest.mark.parametrize("threads", [256, 512, 1024])
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_batch_of_unique_joins_by_the_direct_kernel(dtype, threads):
    # large_batched = 0: builds that fit a shared-memory table go direct, the others one after another
    pairs, host = batch(2, [(1, 1), (255, 70001), (4096, 513), (20000, 100003), (30001, 50000)], dtype)
    bj = api.BatchJoiner(pairs)
    bj.launch()
    check(bj, host)  # (tables in L2)
    bj.config.large_batched = 0
    bj.config.direct_max_build = 20480
    bj.config.direct_threads = threads
    bj.prepare()
    bj.count.zero_()
    bj.launch()
    check(bj, host)


def test_batch_tables_agree_with_the_other_kernels():
    # aligned columns of every size class, by tables, by direct and single joins
    sizes = [(1 << 20, 2049), (700001, 2000003), (3, 2047), (4096, 30000), (900001, 1 << 20)]
    for dtype in (np.int32, np.int64):
        pairs, host = batch(3, sizes, dtype)
        bj = api.BatchJoiner(pairs)
        bj.launch()
        check(bj, host)
        for delta in (0, 1):  # (with one radix bit more a single join is partitioned, not a default plan)
            bj.config.large_batched = 0
            bj.config.direct_max_build = 4096
            bj.config.large_bits_delta = delta
            bj.prepare()
            bj.count.zero_()
            bj.launch()
            check(bj, host)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_planned_heavy_keys_on_a_small_build_side(dtype):
    b, p = datagen.config3(seed=51, theta=1.5, n_build=1 << 18, n_probe=1 << 21)
    b, p = (b % (1 << 31)).astype(dtype), (p % (1 << 31)).astype(dtype)
    b, first = np.unique(b, return_index=True)
    bt, pt = torch.from_numpy(b).cuda(), torch.from_numpy(p).cuda()
    plan = api.plan_exact(bt, pt, True)
    assert plan.n_heavy > 0
    plan.flags = 0  # the partitions and the heavy keys, not the table in L2
    br, pr = api.partitioned_join(bt, pt, plan=plan)
    assert np.array_equal(oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy()), expect(b, p))
    assert api.join_count(bt, pt, plan=plan) == br.numel()


# Tuples beyond 512 MB over 4096 partitions are scattered in groups of items of
# at most 256 MB: three groups here, the last one smaller.
GROUPED = {torch.int32: (1 << 26) + 100003, torch.int64: (1 << 25) + 50021}
ODD = {torch.int32: 0x9E3779B1, torch.int64: 0x9E3779B97F4A7C15}  # an odd multiplier: distinct keys for distinct rows


def signed(dtype):
    bits = 32 if dtype == torch.int32 else 64
    return ODD[dtype] - (1 << bits) if ODD[dtype] >= 1 << (bits - 1) else ODD[dtype]


def columns(dtype, n_build, n_probe, copies):
    """Build row r has key number r // copies; two thirds of the probe rows have the number of some build row."""
    def keys(number):
        return (number * signed(dtype)).to(dtype)

    g = torch.Generator(device="cuda").manual_seed(n_build + copies)
    order = torch.randperm(n_build, device="cuda", generator=g)
    number = order // copies
    numbers = n_build // copies  # (complete runs)
    want = torch.randint(0, numbers + numbers // 2, (n_probe,), device="cuda", generator=g)
    want[want >= numbers] += n_build  # not in the build side
    return keys(number), keys(want), number, want, numbers


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64], ids=["int32", "int64"])
@pytest.mark.parametrize("name,table,copies,capacity,big_build", [
    ("exact", TABLE_EXACT, 1, 0, True),
    ("bucket_split_by_hash", TABLE_BUCKET, 1, 3200, True),       # several pieces a partition, each over all groups
    ("bucket_split_by_position", TABLE_BUCKET, 2, 3200, True),   # pieces that end inside a group
    ("compact_probe_groups", TABLE_COMPACT, 1, 0, False),        # build side in one group
    ("compact_repeated_keys", TABLE_COMPACT, 3, 0, True),
    ("bucket_probe_groups", TABLE_BUCKET, 2, 0, False),
    ("bucket_heavy_keys", TABLE_BUCKET, 1, 0, False)])
def test_joins_over_several_item_groups(dtype, name, table, copies, capacity, big_build):
    n_probe = GROUPED[dtype]
    n_build = n_probe + 4099 if big_build else 5000003
    b, p, number, want, numbers = columns(dtype, n_build, n_probe, copies)
    plan = api.plan_default(n_build, n_probe, b.element_size(), copies == 1)
    plan.passes, plan.bits1, plan.bits2, plan.digit_mode = 1, 12, 0, DIGIT_HASH
    plan.wc_tuples = 16 // b.element_size()
    plan.split_mode = SPLIT_HASH if copies == 1 else SPLIT_POSITION
    if table != TABLE_EXACT or plan.table_mode != TABLE_EXACT:
        plan.table_mode = table
        plan.table_capacity = capacity or {TABLE_BUCKET: 8192, TABLE_COMPACT: 16384, TABLE_EXACT: 16384}[table]
    if name == "bucket_heavy_keys":  # every seventh probe row, and one in 21 without a build row
        want[::7], want[::21] = 5, numbers + n_build + 1
        p = (want * signed(dtype)).to(dtype)
        plan.set_heavy([int(p[7]), int(p[0]), 123456789])
    j = api.Joiner(b, p, copies == 1, plan, capacity=copies * n_probe)
    j.launch()
    br, pr = j.result()
    # the pairs: right, distinct, and as many as there are
    found = want < numbers
    left = n_build - numbers * copies  # build rows of the last, incomplete run
    last = int((want == numbers).sum()) if left else 0
    assert last == 0
    assert br.numel() == copies * int(found.sum())
    assert bool((number[br.long()] == want[pr.long()]).all())
    code = torch.sort(pr.long() * n_build + br.long())[0]
    assert not bool((code[1:] == code[:-1]).any())
    del code
    # as many again in a count
    assert api.join_count(b, p, copies == 1, plan) == br.numel()
