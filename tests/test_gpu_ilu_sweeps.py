"""ILU0-CG (type 0) at the sizes where the triangular sweeps change form: all levels in one block with the
vector in shared memory, the vector in global memory (above 25,600 unknowns), and levels wider than one
fused step or run between narrow ones.  The sweeps and the factorisation keep the order of every sum,
so the iteration counts are the oracle's and the solutions agree to the solves' own accuracy: both stop
at the same residual reduction with iterates that differ by rounding, far below the 1e-9 asked here."""
import numpy as np
import pytest

from parity import gpu_solve, oracle_solve, relmax

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 1, 1), (9, 7, 5), (33, 3, 2), (19, 19, 19), (21, 21, 21), (40, 40, 24)])
def test_ilu_sweeps_match_oracle(pkg, gpulib, orc, workloads, dims):
    prob = workloads.layered_lognormal(dims=dims, seed=5, sat=np.full(int(np.prod(dims)), 0.3))
    g = gpu_solve(pkg, prob, ltype=0, tol=1e-12)
    o = oracle_solve(orc, prob, tol=1e-12)
    # the counts may part by a step or two once rounding has entered hundreds of iterations
    assert abs(g["stats"].iterations - o["iterations"]) <= max(1, o["iterations"] // 100)
    for k in ("p", "v", "pi"):
        assert relmax(g[k], o[k]) < 1e-9
