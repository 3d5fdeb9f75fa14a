"""The planners' mark on a plan: as the planner wrote it, a plan for a build side
whose table stays in L2 joins without partitions; changed in any field, it runs
as written."""
import numpy as np
import pytest
import torch

from oracle import oracle
from partitioned_join_b200 import _lib, api, planner

pytestmark = pytest.mark.gpu

N_BUILD, N_PROBE = 1 << 18, 1 << 21


@pytest.fixture(scope="module")
def tables():
    rng = np.random.default_rng(1)
    b = rng.permutation(N_BUILD).astype(np.int32)
    p = rng.integers(0, 2 * N_BUILD, N_PROBE).astype(np.int32)
    return b, p, torch.from_numpy(b).cuda(), torch.from_numpy(p).cuda(), oracle.sorted_pairs(*oracle.inner_join(b, p, True))


def partitioned(bt, pt, plan, exp):
    """Joins under the plan; whether its partitioning stages ran."""
    j = api.Joiner(bt, pt, True, plan)
    j.launch()
    br, pr = j.result()
    assert np.array_equal(oracle.sorted_pairs(br.cpu().numpy(), pr.cpu().numpy()), exp)
    # (both sides' histogram, scan and scatter of 2^21 rows; empty stages are under 10 us together)
    return min(sum(j.launch_timed()[s] for s in ("probe_hist", "probe_scan", "probe_scatter")) for _ in range(5)) > 0.015


def planned(kind, bt, pt):
    if kind == "exact":
        return api.plan_exact(bt, pt)
    return planner.plan_learned(bt, pt, True, planner.load_weights())[0]


EDITS = {"hist_split": lambda p: setattr(p, "hist_split", p.hist_split % 4 + 1),
         "bits1": lambda p: setattr(p, "bits1", p.bits1 + 1),
         "probe_chunk": lambda p: setattr(p, "probe_chunk", p.probe_chunk + 16),
         "table_mode": lambda p: (setattr(p, "table_mode", _lib.TABLE_OPEN), setattr(p, "table_capacity", 8192)),
         "max_fill": lambda p: setattr(p, "max_fill", 0.4),
         "set_heavy": lambda p: p.set_heavy([5, 7]),
         "flags": lambda p: (setattr(p, "flags", 0), setattr(p, "hist_split", 3))}


@pytest.mark.parametrize("kind", ["exact", "learned"])
def test_an_unchanged_plan_takes_the_table(tables, kind):
    b, p, bt, pt, exp = tables
    plan = planned(kind, bt, pt)
    assert plan.flags & 1
    assert not partitioned(bt, pt, plan, exp)
    assert not partitioned(bt, pt, _lib.Plan.from_buffer_copy(plan), exp)  # (a copy, as one read from a file)
    plan.hist_split += 1
    plan.hist_split -= 1
    assert not partitioned(bt, pt, plan, exp)


@pytest.mark.parametrize("kind", ["exact", "learned"])
@pytest.mark.parametrize("edit", EDITS)
def test_a_changed_plan_runs_as_written(tables, kind, edit):
    b, p, bt, pt, exp = tables
    plan = planned(kind, bt, pt)
    EDITS[edit](plan)
    assert partitioned(bt, pt, plan, exp)


def test_heavy_keys_of_a_marked_plan_count(tables):
    b, p, bt, pt, exp = tables
    plan = planned("exact", bt, pt)
    plan.set_heavy([5, 7])
    assert partitioned(bt, pt, plan, exp)
    plan.heavy_keys[1] = 9
    assert partitioned(bt, pt, plan, exp)
