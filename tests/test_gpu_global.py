"""Joins by one table in L2 (default plans of up to 2^22 build rows): the pairs
are the oracle's at the edges of tiles, of the table's densities, with full
buckets, repeated keys and outputs past the capacity -- and the partitioned
path's, which the same plan with any field changed takes."""
import numpy as np
import pytest
import torch

from oracle import oracle
from partitioned_join_b200 import PJError, api

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def pairs(br, pr):
    return oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy())


def expect(b, p, unique):
    return oracle.sorted_pairs(*oracle.inner_join(b, p, unique))


def tables(rng, nb, np_, dtype, unique, spread=2):
    info = np.iinfo(dtype)
    k = rng.permutation(nb * spread + 3)[:nb].astype(np.int64)
    if dtype == np.int64:
        k = k * 0x100000001B3 - (1 << 40)
    if not unique:
        k = rng.choice(k[: max(1, nb // 3)], nb)
    b = k.astype(dtype)
    p = np.where(rng.random(np_) < 0.7, rng.choice(b, np_), rng.integers(info.min, info.max, np_, dtype=dtype))
    return b, p.astype(dtype)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("unique", [True, False])
@pytest.mark.parametrize("nb,np_", [(1, 1), (2, 513), (255, 511), (257, 512), (2047, 2049), (20011, 30007),
                                    ((1 << 20) - 1, 1 << 20), ((1 << 20) + 1, (1 << 22) + 5), (1 << 22, 70001),
                                    ((1 << 22) + 1, 1000)])
def test_global_table_matches_oracle(dtype, unique, nb, np_):
    rng = np.random.default_rng(nb + np_)
    b, p = tables(rng, nb, np_, dtype, unique)
    br, pr = api.partitioned_join(dev(b), dev(p), unique)
    assert np.array_equal(pairs(br, pr), expect(b, p, unique))
    assert api.join_count(dev(b), dev(p), unique) == br.numel()


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_global_and_partitioned_routes_agree(dtype):
    rng = np.random.default_rng(5)
    b, p = tables(rng, 150001, 400003, dtype, True)
    plan = api.plan_default(b.shape[0], p.shape[0], np.dtype(dtype).itemsize)
    written = api.plan_default(b.shape[0], p.shape[0], np.dtype(dtype).itemsize)
    written.hist_split = 1  # the caller's own schedule: partitioned
    got = [pairs(*api.partitioned_join(dev(b), dev(p), plan=q)) for q in (plan, written, api.plan_exact(dev(b), dev(p)))]
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_repeated_keys_under_the_unique_flag_match_one_row(dtype):
    rng = np.random.default_rng(6)
    b = rng.integers(0, 500, size=300000).astype(dtype)   # 600 rows a key
    p = rng.integers(0, 1000, size=100000).astype(dtype)
    br, pr = api.partitioned_join(dev(b), dev(p), True)
    br, pr = br.cpu().numpy(), pr.cpu().numpy()
    assert np.array_equal(b[br], p[pr])
    assert np.array_equal(np.sort(pr), np.nonzero(p < 500)[0])


@pytest.mark.parametrize("copies", [31, 33, 700, 40000])
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_long_runs_of_one_key(copies, dtype):
    # around the length from which a warp walks a bucket together, and past
    # the pairs a CTA stages
    rng = np.random.default_rng(copies)
    b = np.concatenate([np.full(copies, -7), rng.integers(0, 5000, size=9000)]).astype(dtype)
    p = np.concatenate([np.full(9, -7), rng.integers(0, 6000, size=2000)]).astype(dtype)
    rng.shuffle(b)
    rng.shuffle(p)
    br, pr = api.partitioned_join(dev(b), dev(p), False)
    assert np.array_equal(pairs(br, pr), expect(b, p, False))


@pytest.mark.parametrize("unique", [True, False])
def test_outputs_past_the_capacity_report_the_count(unique):
    b = np.arange(3000, dtype=np.int32)
    p = np.tile(b, 3)
    j = api.Joiner(dev(b), dev(p), unique, capacity=100)
    j.launch()
    with pytest.raises(PJError):
        j.result()
    assert int(j.count.item()) == 9000
    j.launch()  # the workspace is clean again
    assert j.status() == 2


def test_twin_fingerprints_of_eight_byte_keys():
    # build keys whose hashes agree on the home bucket's bits and the
    # fingerprint: only the key tells them apart
    keys = (np.arange(1, 1 << 22, dtype=np.int64) * 2654435761 + 12345) * 0x10001
    h = oracle.hash_keys(keys).astype(np.uint64)
    n = 4096
    home = (h * np.uint64(n)) >> np.uint64(32)
    group = (home << np.uint64(10)) | (h & np.uint64(1023))
    order = np.argsort(group, kind="stable")
    g = group[order]
    twin = np.nonzero(g[1:] == g[:-1])[0]
    a, c = keys[order[twin]], keys[order[twin + 1]]
    build = np.unique(a)[:n]
    assert build.shape[0] == n
    probe = np.concatenate([c[:5000], a[:5000], build])
    br, pr = api.partitioned_join(dev(build), dev(probe))
    assert np.array_equal(pairs(br, pr), expect(build, probe, True))
