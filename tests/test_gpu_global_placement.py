"""Repeated build keys by one table in L2: a join with few CTAs of lookups takes
no longer behind other work, when its launches follow each other at once, than
alone."""
import numpy as np
import pytest
import torch

from oracle import oracle
from partitioned_join_b200 import api

pytestmark = pytest.mark.gpu


def dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def pairs(br, pr):
    return oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy())


def expect(b, p):
    return oracle.sorted_pairs(*oracle.inner_join(b, p, False))


@pytest.mark.parametrize("dtype", [np.int32, np.int64])
def test_few_ctas_do_not_crowd_together(dtype):
    # 32 CTAs of lookups behind a build of 256: joined at once after other work, no slower than with room to wait
    nb, n_probe, copies = 1 << 16, 1 << 14, 16
    rng = np.random.default_rng(4)
    b = (rng.permutation(nb) // copies * 0x1003F).astype(dtype)
    p = (rng.integers(0, nb // copies, n_probe) * 0x1003F).astype(dtype)
    j = api.Joiner(dev(b), dev(p), False)
    j.launch()
    before = torch.empty(1 << 26, dtype=torch.int32, device="cuda")
    t = {True: [], False: []}
    for busy in (True, False) * 6:
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        if busy:  # (the host is ahead: the launches follow each other at once)
            before.fill_(1)
        e0.record()
        j.launch()
        e1.record()
        torch.cuda.synchronize()
        t[busy].append(e0.elapsed_time(e1))
    assert min(t[True]) < 1.3 * min(t[False]), t
    assert np.array_equal(pairs(*j.result()), expect(b, p))
