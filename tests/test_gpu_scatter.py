"""The barrier-free write-combining scatter: every row lands once, in its
partition, with less than W padding tuples a segment -- over fan-outs from one
partition to the most (units of 2 to 128 tuples), sizes around a warp's and a
round's, and skew that keeps one unit full while others idle."""
import numpy as np
import pytest
import torch

from oracle import oracle
from partitioned_join_b200 import DIGIT_HASH, DIGIT_RAW, api

pytestmark = pytest.mark.gpu

SMS = 148


def keys_of(kind, n, dtype, rng):
    info = np.iinfo(dtype)
    if kind == "uniform":
        return rng.integers(info.min, info.max, size=n, dtype=dtype)
    if kind == "one":
        return np.full(n, 12345, dtype=dtype)
    k = rng.integers(0, 1 << 20, size=n).astype(dtype)   # half of the rows in three partitions
    hot = rng.random(n) < 0.5
    k[hot] = rng.choice(np.array([7, 8, 1000003], dtype=dtype), int(hot.sum()))
    return k


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
@pytest.mark.parametrize("mode", [DIGIT_RAW, DIGIT_HASH])
@pytest.mark.parametrize("kind", ["uniform", "one", "hot"])
@pytest.mark.parametrize("bits,w", [(0, 0), (1, 32), (4, 8), (7, 0), (9, 16), (11, 0), (12, 0), (13, 2)])
def test_every_row_lands_once(dtype, mode, kind, bits, w):
    if bits == 13 and dtype == np.int64:
        pytest.skip("8192 partitions of 16-byte tuples do not fit shared memory")
    rng = np.random.default_rng(bits * 10 + mode)
    words = 2 if dtype == np.int32 else 4
    W = w or 8 // words
    P = 1 << bits
    for n in (1, 33, 4099, 700001):
        keys = keys_of(kind, n, dtype, rng)
        plan = api.plan_default(n, n, np.dtype(dtype).itemsize)
        plan.bits1, plan.wc_tuples, plan.digit_mode = bits, W, mode
        tuples, offsets = api.partition(torch.from_numpy(keys).cuda(), plan)
        off = offsets.cpu().numpy()
        rec = tuples.cpu().numpy()[: off[-1] * words].reshape(-1, words)
        rows = rec[:, -1]
        real = rows >= 0
        assert np.all(rows[~real] == -1)
        assert np.array_equal(np.sort(rows[real]), np.arange(n)), (n, kind)
        h = oracle.hash_keys(keys)
        got = rec[real, 0 if words == 2 else 2].astype(np.uint32)
        assert np.array_equal(got, h[rows[real]])
        part = np.repeat(np.arange(P), np.diff(off))
        assert np.array_equal(part[real], oracle.digits(keys, mode, bits, 0, 0)[rows[real]])
        # one segment per partition and chunk, each padded to a multiple of W
        assert np.all(np.diff(off) % W == 0)
        pad = np.bincount(part[~real], minlength=P)
        assert pad.max() <= SMS * (W - 1)
