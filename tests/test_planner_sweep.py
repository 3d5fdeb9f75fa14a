"""The learned planner's sweep times schedules only where a planner's plan takes
one: above the build sides that are joined by one table in L2."""
import os
import re

import numpy as np
import pytest

from partitioned_join_b200 import planner

CSRC = os.path.join(os.path.dirname(planner.__file__), "csrc")


def test_the_sweep_starts_above_the_tables():
    text = open(os.path.join(CSRC, "pj_global.cuh")).read()
    row_bits = int(re.search(r"GT_ROW_BITS = (\d+);", text).group(1))
    assert "GT_MAX_BUILD = int64_t(1) << GT_ROW_BITS" in text
    assert planner.TABLE_LOG2_BUILD == row_bits
    for lowest in (18, 22, 22.5):
        lo, hi = planner.sweep_range(lowest, 28)
        assert int(2 ** np.float64(lo)) > 1 << row_bits and lo >= lowest and hi == 28
    with pytest.raises(ValueError):
        planner.sweep_range(18, 22)
