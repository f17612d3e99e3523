"""The AMG-CG recurrences in FP64 and mixed precision, at the sizes where their reductions change shape: two
blocks per SM of 256 threads (up to 78k unknowns on 152 SMs), of 512 and 1024 threads (155k, 311k), and
grid-stride beyond, with lengths that no block divides.

Both solves stop on a residual reduction of 1e-13 in FP64; their solutions differ by at most about 1e-13
times the condition of these systems (below 1e5), so 1e-8 is asked.  The mixed recurrence is CG on the same
system with rounded vectors: each step keeps the new direction conjugate to the last one, so it may need
some more steps, a quarter more at most."""
import numpy as np
import pytest

from parity import gpu_solve, relmax

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", [0, 1])
@pytest.mark.parametrize("dims", [(1, 1, 1), (29, 29, 29), (31, 30, 29), (41, 37, 33), (61, 53, 31), (97, 89, 41)])
def test_mixed_and_fp64_recurrences_agree(pkg, gpulib, workloads, dims, seed):
    prob = workloads.layered_lognormal(dims=dims, seed=seed, sat=np.full(int(np.prod(dims)), 0.3))
    a, b = (gpu_solve(pkg, prob, ltype=1, tol=1e-13, precision=q) for q in (0, 1))
    na, nb = a["stats"].iterations, b["stats"].iterations
    assert nb <= na + na // 4 + 3
    for k in ("p", "v", "pi"):
        assert relmax(b[k], a[k]) < 1e-8
    c = gpu_solve(pkg, prob, ltype=1, tol=1e-13, precision=1)
    for k in ("p", "v", "pi"):
        assert np.array_equal(b[k], c[k])


@pytest.mark.parametrize("dims", [(31, 30, 29), (61, 53, 31)])
def test_guarded_recurrence(pkg, gpulib, workloads, dims):
    """With hardly any coarse correction, and a replacement only once the FP32 residual has dropped by 1e-13, a
    stage lasts longer than 128 iterations: the recurrence goes on guarded.  The true residual gains at least
    four digits per stage (FP32 vectors), so four stages of FP64's count reach 1e-13."""
    prob = workloads.layered_lognormal(dims=dims, seed=3, sat=np.full(int(np.prod(dims)), 0.3))
    opt = dict(ltype=1, tol=1e-13, prolongate_factor=0.01)
    a = gpu_solve(pkg, prob, **opt)
    b = gpu_solve(pkg, prob, precision=1, inner_tolerance=1e-13, **opt)
    assert 128 < b["stats"].iterations <= 4 * a["stats"].iterations
    for k in ("p", "v", "pi"):
        assert relmax(b[k], a[k]) < 1e-8
