"""Repeated build keys by one table in L2: the pairs of a warp's 64 probe rows
pass through a stage of 256, what does not fit is walked again; entries of
8-byte keys hold the key where the probe side is no smaller than the build
side.  The pairs are the oracle's around each limit."""
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


def check(b, p):
    br, pr = api.partitioned_join(dev(b), dev(p), False)
    assert np.array_equal(pairs(br, pr), expect(b, p))
    assert api.join_count(dev(b), dev(p), False) == br.numel()


# 64 rows of `copies` pairs and `extra` more pairs in one warp: below, at and above 256, all lanes or one
@pytest.mark.parametrize("copies,extra", [(1, 0), (3, 63), (4, 0), (4, 1), (5, 0), (8, 31), (16, 0), (31, 32), (32, 32)])
@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("n_build", [4000, 9000])  # grouped by one CTA, by three launches
def test_pairs_of_a_warp_around_the_stage(copies, extra, dtype, n_build):
    rng = np.random.default_rng(copies + extra)
    key = (rng.permutation(1 << 20)[:n_build].astype(np.int64) * 0x100000001B3).astype(dtype)
    runs = 90
    b = np.concatenate([np.repeat(key[:runs], copies), np.full(extra, key[runs]), key[runs + 1:]])[:n_build]
    rng.shuffle(b)
    for n_probe in (64, 63, 512 + 65, 20000):  # (8-byte entries hold the key in the last only)
        p = rng.choice(key[:runs], n_probe)
        p[:: 64] = key[runs]
        check(b, p)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("copies", [33, 40, 200])
def test_walked_ranges_behind_a_full_stage(dtype, copies):
    # from 2^19 probe rows on a warp walks ranges of 33 and more entries itself, after the rows with short ones
    rng = np.random.default_rng(copies)
    k = (rng.permutation(1 << 20)[:30000].astype(np.int64) * 0x100000001B3).astype(dtype)
    b = np.concatenate([np.repeat(k[:20], copies), np.repeat(k[20:120], 9), k[120:]])
    rng.shuffle(b)
    p = rng.integers(-(1 << 30), -1, (1 << 19) + 3).astype(dtype)
    p[:6400] = rng.choice(k[20:120], 6400)
    p[rng.integers(0, 9000, 500)] = rng.choice(k[:20], 500)
    check(b, p)


@pytest.mark.parametrize("n_probe", [2000, 8191, 8192, 8193, 30000])
def test_8_byte_keys_that_differ_in_one_word(n_probe):
    # equal low words, equal high words, and complements, on both sides of the entries that hold the key
    rng = np.random.default_rng(n_probe)
    word = rng.integers(0, 1 << 31, 8).astype(np.int64)
    grid = (word[:, None] << 32 | word[None, :]).ravel()
    b = rng.choice(np.concatenate([grid, ~grid]), 8192)
    b[100:] = np.where(rng.random(8092) < 0.05, b[100:], rng.integers(-(1 << 62), 1 << 62, 8092))
    p = np.where(rng.random(n_probe) < 0.02, rng.choice(np.concatenate([grid, ~grid]), n_probe), rng.choice(b, n_probe))
    check(b, p)


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_capacity_inside_a_stage(dtype):
    b = np.repeat(np.arange(500), 12).astype(dtype)
    p = np.arange(480).repeat(20).astype(dtype)
    for capacity in (100, 768 + 5):
        j = api.Joiner(dev(b), dev(p), False, capacity=capacity)
        j.launch()
        st, n = j.status_count()
        assert st == _lib.ERR_CAPACITY and n == 12 * 9600
        x = j.probe_row.long() * 6000 + j.build_row.long()
        assert torch.unique(x).numel() == capacity and bool((dev(b)[j.build_row.long()] == dev(p)[j.probe_row.long()]).all())
