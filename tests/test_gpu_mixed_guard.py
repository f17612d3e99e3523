"""The guarded form of the mixed-precision CG, and its restarts, seen to run: a stage of more than 128 iterations
without a replacement turns it on, a direction of zero curvature starts anew from the preconditioned residual
(once; another one is a breakdown, so a matrix with negative curvature is refused).

The matrices are tridiagonal (2 + shift, -1): condition at most 4 / shift.  A solve to a residual reduction tol is
within condition * tol of the solution (2-norm).  CG needs about sqrt(condition) / 2 * ln(2 / tol) iterations
for tol; in FP32 vectors and stages of four digits at least, the guarded form at most four times that."""
import numpy as np
import pytest

sp = pytest.importorskip("scipy.sparse")

pytestmark = pytest.mark.gpu

NONFINITE = 3


def system(n, shift, seed=0):
    A = sp.diags([-np.ones(n - 1), (2.0 + shift) * np.ones(n), -np.ones(n - 1)], [-1, 0, 1]).tocsr()
    A.sort_indices()
    b = np.random.default_rng(seed).standard_normal(n)
    return A, b, np.linalg.solve(A.toarray(), b)


def close(x, ref, shift, tol):
    return np.linalg.norm(x - ref) <= 4.0 / shift * tol * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [400, 2000])
def test_long_stage_goes_on_guarded(pkg, gpulib, n):
    shift, tol = 0.01, 1e-11
    A, b, ref = system(n, shift)
    limit = 4 * int(np.sqrt(4.0 / shift) / 2 * np.log(2.0 / tol))
    rc, x, its, guarded = pkg.selftest_mixed_cg(A, b, tol, limit, 1e-13)
    assert rc == 0 and guarded and its > 128
    assert close(x, ref, shift, tol)
    # stages of three digits end before 128 iterations: the plain recurrence
    rc, x, its, guarded = pkg.selftest_mixed_cg(A, b, tol, limit, 1e-3)
    assert rc == 0 and not guarded
    assert close(x, ref, shift, tol)


@pytest.mark.parametrize("skip", [1, 2, 5, 20])
def test_zero_curvature_starts_anew(pkg, gpulib, skip):
    shift, tol = 0.2, 1e-11
    A, b, ref = system(600, shift)
    limit = 4 * int(np.sqrt(4.0 / shift) / 2 * np.log(2.0 / tol)) + 2
    rc, x, its, guarded = pkg.selftest_mixed_cg(A, b, tol, limit, 3e-3, skip, 1)
    assert rc == 0 and guarded
    assert close(x, ref, shift, tol)


@pytest.mark.parametrize("skip,skips", [(0, 1), (3, 2), (20, 2)])
def test_zero_curvature_of_a_fresh_direction_is_a_breakdown(pkg, gpulib, skip, skips):
    A, b, ref = system(600, 0.2)
    rc, x, its, _ = pkg.selftest_mixed_cg(A, b, 1e-11, 400, 3e-3, skip, skips)
    assert rc == NONFINITE
    assert np.all(np.isfinite(x)) and its <= skip + skips
    if skip == 0:
        assert np.all(x == 0.0)   # the direction without curvature changed nothing


@pytest.mark.parametrize("n", [50, 1000, 20000, 200000])
@pytest.mark.parametrize("diagonal", [1.0, 1.5, 1.9])
def test_negative_curvature_is_refused(pkg, gpulib, n, diagonal):
    """Tridiagonal (diagonal, -1): eigenvalues diagonal - 2 cos(t), a good part of them negative.  The solve gives
    up at the second direction of negative curvature, long before its iterates grow out of range."""
    A = sp.diags([-np.ones(n - 1), diagonal * np.ones(n), -np.ones(n - 1)], [-1, 0, 1]).tocsr()
    A.sort_indices()
    b = np.random.default_rng(n).standard_normal(n)
    rc, x, its, _ = pkg.selftest_mixed_cg(A, b, 1e-10, 20000, 3e-3)
    assert rc == NONFINITE
    assert np.linalg.norm(b - A @ x) <= 1e6 * np.linalg.norm(b)
