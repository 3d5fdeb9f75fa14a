"""The batch autotuner compares whole batches: it keeps the shared tables where
they are the faster route, leaves alone what reaches no join of the batch, and
never ends slower than the defaults."""
import numpy as np
import pytest
import torch

from oracle import oracle
from partitioned_join_b200 import api

pytestmark = pytest.mark.gpu


def small_batch(seed, n, dtype):
    rng = np.random.default_rng(seed)
    pairs, host = [], []
    for _ in range(n):
        nb = int(2 ** rng.uniform(8, 13))
        b = (rng.permutation(3 * nb)[:nb].astype(np.int64) * 0x100000001B3).astype(dtype)
        p = rng.choice(b, 7 * nb)
        pairs.append((torch.from_numpy(b).cuda(), torch.from_numpy(p).cuda()))
        host.append((b, p))
    return pairs, host


def best_ms(g, reps=20):
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t = float("inf")
    for _ in range(reps):
        e0.record()
        g.replay()
        e1.record()
        torch.cuda.synchronize()
        t = min(t, e0.elapsed_time(e1))
    return t


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_small_joins_stay_together(dtype):
    pairs, host = small_batch(71, 64, dtype)
    bj = api.BatchJoiner(pairs)
    before = bj.config.as_dict()
    t0 = best_ms(bj.graph())
    ms = bj.autotune()
    # one group of tables takes a sixth of the direct kernel's time here
    assert bj.config.large_batched == 1
    # (no join is direct or partitioned: the other knobs keep their defaults)
    assert bj.config.as_dict() == before
    assert best_ms(bj.graph()) < 1.5 * t0 and ms > 0
    for (br, pr), (b, p) in zip(bj.results(), host):
        got = oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy())
        assert np.array_equal(got, oracle.sorted_pairs(*oracle.inner_join(b, p, True)))


def test_repeated_keys_are_still_tuned():
    rng = np.random.default_rng(72)
    pairs, host = [], []
    for _ in range(12):
        nb = int(2 ** rng.uniform(10, 16))
        b, p = rng.integers(0, nb, nb).astype(np.int32), rng.integers(0, nb, 3 * nb).astype(np.int32)
        pairs.append((torch.from_numpy(b).cuda(), torch.from_numpy(p).cuda()))
        host.append((b, p))
    bj = api.BatchJoiner(pairs, unique_build_keys=False)
    t0 = best_ms(bj.graph())
    bj.autotune()
    assert best_ms(bj.graph()) < 1.2 * t0
    for (br, pr), (b, p) in zip(bj.results(), host):
        got = oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy())
        assert np.array_equal(got, oracle.sorted_pairs(*oracle.inner_join(b, p, False)))
