"""AMG setup: the hierarchies of levels whose pairing rounds run as one cluster launch (1 to 16 blocks,
isolated Dirichlet rows, rounds that stall and are redone, three-round levels) are those recorded from the
launch-per-step setup, row for row and entry for entry."""
import os
import sys

import numpy as np
import pytest

from parity import gpu_solve

sys.path.insert(0, os.path.join(os.path.dirname(__file__), "golden"))
from amg_levels import LEVELS  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", list(LEVELS))
def test_hierarchy_is_the_recorded_one(pkg, gpulib, workloads, name):
    dims, precision = name.split("_")
    dims = tuple(int(x) for x in dims.split("x"))
    prob = workloads.layered_lognormal(dims=dims, seed=9, sat=np.full(int(np.prod(dims)), 0.2))
    g = gpu_solve(pkg, prob, ltype=1, tol=1e-12, precision=int(precision))
    rows, entries = g["solver"].amg_info()
    assert rows == list(LEVELS[name][0])
    assert entries == list(LEVELS[name][1])
