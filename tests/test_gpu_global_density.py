"""The sizes at which a unique build side's table in L2 changes its rows a bucket."""
import numpy as np
import pytest
import torch

from oracle import oracle
from partitioned_join_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,line", [(np.int32, 1 << 21), (np.int64, 3 << 19)])
@pytest.mark.parametrize("more", [0, 1])
@pytest.mark.parametrize("n_probe", [3000, (1 << 21) + 77])
def test_both_sides_of_the_line(dtype, line, more, n_probe):
    rng = np.random.default_rng(line + more)
    b = (rng.permutation(2 * line)[: line + more].astype(np.int64) * 0x100000001B3).astype(dtype)
    p = np.where(rng.random(n_probe) < 0.6, rng.choice(b, n_probe), -1 - rng.integers(0, 1 << 30, n_probe)).astype(dtype)
    br, pr = api.partitioned_join(torch.from_numpy(b).cuda(), torch.from_numpy(p).cuda())
    got = oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy())
    assert np.array_equal(got, oracle.sorted_pairs(*oracle.inner_join(b, p, True)))
