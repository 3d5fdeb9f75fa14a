"""Repeated build keys by one table in L2 where few keys hold many rows: their
ranges are cut into slices over the GPU.  The pairs are the oracle's around the
length from which a range is cut, the ends of slices and rounds, with other keys
in a long range, and past the capacity -- and one hot key costs no more than it
does the partitioned path."""
import numpy as np
import pytest
import torch

from oracle import oracle
from partitioned_join_b200 import _lib, api

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def pairs(br, pr):
    return oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy())


def expect(b, p):
    return oracle.sorted_pairs(*oracle.inner_join(b, p, False))


def run_keys(rng, copies, runs, others, dtype):
    """`runs` keys of `copies` rows each among `others` rows of single ones."""
    k = (rng.permutation(4 * (runs + others))[: runs + others].astype(np.int64) * 0x100000001B3).astype(dtype)
    b = np.concatenate([np.repeat(k[:runs], copies), k[runs:]])
    rng.shuffle(b)
    return b, k


# up to 32 entries are walked by a lane, four at a time; a range is cut from 33 entries on, into slices of 64, 32 of
# them a round
@pytest.mark.parametrize("copies", [1, 3, 4, 5, 31, 32, 33, 63, 64, 65, 255, 2048, 2049])
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("n_probe", [1, 65, 5000])
def test_ranges_around_the_slices(copies, dtype, n_probe):
    rng = np.random.default_rng(copies + n_probe)
    b, k = run_keys(rng, copies, 3, 9000, dtype)
    # rows of the runs, of single keys, and misses of which some fall into the long ranges
    p = np.where(rng.random(n_probe) < 0.1, rng.choice(k[:3], n_probe),
                 np.where(rng.random(n_probe) < 0.5, rng.choice(k[3:], n_probe), rng.integers(-(1 << 30), -1, n_probe))).astype(dtype)
    p[0] = k[0]
    br, pr = api.partitioned_join(dev(b), dev(p), False)
    assert np.array_equal(pairs(br, pr), expect(b, p))
    assert api.join_count(dev(b), dev(p), False) == br.numel()


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_many_words_of_long_ranges(dtype):
    # every warp's probe rows meet long ranges of all lengths: more rounds than CTAs, and fewer
    rng = np.random.default_rng(3)
    lengths = rng.integers(1, 400, 300)
    b = np.repeat(np.arange(300), lengths).astype(dtype)
    rng.shuffle(b)
    for n_probe in (300, 20001):
        p = rng.integers(0, 310, n_probe).astype(dtype)
        br, pr = api.partitioned_join(dev(b), dev(p), False)
        assert np.array_equal(pairs(br, pr), expect(b, p))


# from 2^19 probe rows on, ranges of up to 256 (8-byte keys) or 1024 entries are walked, longer ones cut
@pytest.mark.parametrize("dtype,copies", [(np.int32, 1024), (np.int32, 1025), (np.int64, 256), (np.int64, 257)])
def test_many_probe_rows_around_the_walked_length(dtype, copies):
    rng = np.random.default_rng(copies)
    b, k = run_keys(rng, copies, 2, 20000, dtype)
    p = rng.integers(-(1 << 30), -1, (1 << 19) + 5).astype(dtype)
    p[rng.integers(0, p.shape[0], 700)] = k[0]
    p[rng.integers(0, p.shape[0], 3000)] = k[5]
    br, pr = api.partitioned_join(dev(b), dev(p), False)
    assert np.array_equal(pairs(br, pr), expect(b, p))


# one CTA groups up to 4096 build rows
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("nb", [7, 1023, 4095, 4096, 4097])
def test_builds_grouped_by_one_cta(dtype, nb):
    rng = np.random.default_rng(nb)
    b = rng.integers(0, max(1, nb // 3), nb).astype(dtype)
    p = rng.integers(0, nb, 9001).astype(dtype)
    j = api.Joiner(dev(b), dev(p), False)
    for _ in range(2):  # (the second on a used workspace)
        j.launch()
        assert np.array_equal(pairs(*j.result()), expect(b, p))


@pytest.mark.parametrize("nb", [3000, 30000])
def test_captured_and_timed_calls(nb):
    rng = np.random.default_rng(nb)
    b = np.concatenate([np.full(nb // 2, 9), rng.integers(0, nb, nb // 2)]).astype(np.int64)
    p = np.concatenate([np.full(5, 9), rng.integers(0, nb, 10000)]).astype(np.int64)
    j = api.Joiner(dev(b), dev(p), False)
    j.launch()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        j.launch()
    for _ in range(3):
        j.build_row.zero_()
        g.replay()
        assert np.array_equal(pairs(*j.result()), expect(b, p))
    j.build_row.zero_()
    assert j.launch_timed()["total"] > 0
    assert np.array_equal(pairs(*j.result()), expect(b, p))


def test_capacity_inside_a_long_range():
    b = np.full(5000, 7, dtype=np.int64)
    p = np.full(3, 7, dtype=np.int64)
    j = api.Joiner(dev(b), dev(p), False, capacity=6000)
    j.launch()
    st, n = j.status_count()
    assert st == _lib.ERR_CAPACITY and n == 15000
    # what was written is pairs of the join, none twice
    x = j.probe_row.long() * 5000 + j.build_row.long()
    assert torch.unique(x).numel() == 6000 and int(x.min()) >= 0 and int(x.max()) < 15000


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_a_hot_build_key_uses_the_whole_gpu(dtype):
    nb, hits = 1 << 20, 64
    rng = np.random.default_rng(11)
    b = rng.integers(1, nb, nb).astype(dtype)
    b[: nb // 2] = -7
    rng.shuffle(b)
    p = np.concatenate([np.full(hits, -7), rng.integers(nb, 2 * nb, (1 << 21) - hits)]).astype(dtype)
    bt, pt = dev(b), dev(p)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = []
    for written in (False, True):
        plan = api.plan_default(nb, p.shape[0], b.itemsize, False)
        if written:
            plan.hist_split = 1 if plan.hist_split != 1 else 2  # the caller's own schedule: partitioned
        j = api.Joiner(bt, pt, False, plan, capacity=hits * (nb // 2))
        j.launch()
        st, n = j.status_count()
        assert st == _lib.OK and n == hits * (nb // 2)
        t = []
        for _ in range(3):
            e0.record()
            j.launch()
            e1.record()
            torch.cuda.synchronize()
            t.append(e0.elapsed_time(e1))
        best.append(min(t))
        # every hot build row with every hot probe row once
        x = torch.unique(j.probe_row.long() * nb + j.build_row.long())
        assert x.numel() == n and int(x.max()) < hits * nb and bool((bt[(x % nb)] == -7).all())
    assert best[0] < best[1], best


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_few_rows_a_key_gain_from_the_table(dtype):
    # 16 probe rows a build row, four build rows a key: the table is the faster route for both key widths
    nb, n_probe = 1 << 20, 1 << 24
    rng = np.random.default_rng(12)
    b = (rng.permutation(nb) // 4 * 0x1003F).astype(dtype)
    p = (rng.integers(0, 3 * nb // 8, n_probe) * 0x1003F).astype(dtype)
    bt, pt = dev(b), dev(p)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = []
    for written in (False, True):
        plan = api.plan_default(nb, n_probe, b.itemsize, False)
        if written:
            plan.hist_split = 1 if plan.hist_split != 1 else 2
        j = api.Joiner(bt, pt, False, plan)
        t = []
        for _ in range(5):
            e0.record()
            j.launch()
            e1.record()
            torch.cuda.synchronize()
            t.append(e0.elapsed_time(e1))
        best.append(min(t))
        br, pr = j.result()
        assert br.numel() == 4 * int((p < nb // 4 * 0x1003F).sum()) if dtype == np.int64 else br.numel() > 0
        assert bool((bt[br.long()] == pt[pr.long()]).all())
    assert best[0] < best[1], best
