"""The fused ILU(0) sweeps wait for their bulk-copied records with a limit.  Each thread waits for itself, so one
thread's wait may run out where the others' do not: whichever thread it is (a row's, an idle one's, the one that
copies), the sweep reports the timeout and the context stays usable.  The same for the lanes of the smoother's
staged step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = 6


def exact():
    n = 48
    A = 2.5 * np.eye(n) - np.eye(n, k=1) - np.eye(n, k=-1)
    return np.linalg.solve(A, 1.0 + np.arange(n) / 8.0)


def check_normal(pkg, shared):
    rc, z = pkg.selftest_ilu_wait(-1, shared)
    assert rc == 0
    # ILU(0) of a tridiagonal matrix is its LU; condition 9, so a few roundings
    assert np.abs(z - exact()).max() <= 48 * 9 * 2.0 ** -53 * np.abs(z).max()


@pytest.mark.parametrize("shared", [True, False])
@pytest.mark.parametrize("thread", [0, 5, 31, 100, 255, 256, 287])
def test_any_threads_timeout_is_reported(pkg, gpulib, shared, thread):
    check_normal(pkg, shared)
    rc, _ = pkg.selftest_ilu_wait(thread, shared)
    assert rc == TIMEOUT
    check_normal(pkg, shared)


@pytest.mark.parametrize("lane", [0, 1, 17, 31])
def test_any_lanes_timeout_is_reported(pkg, gpulib, lane):
    rc, r, _, _ = pkg.selftest_bulk_wait(2 + lane)
    assert rc == TIMEOUT
    assert np.all(r == 2.0)   # the step wrote nothing
    assert pkg.selftest_bulk_wait(False)[0] == 0


def launches_per_iteration(pkg, workloads, dims):
    prob = workloads.layered_lognormal(dims=dims, seed=5, sat=np.full(int(np.prod(dims)), 0.3))
    s = pkg.PressureSolver()
    s.init(prob.grid, prob.perm.ravel(), (0.0, 0.0, 0.0), prob.bc_type)
    n = []
    for maxit in (2, 6):
        before = pkg.lib().porsol_launch_count()
        with pytest.raises(pkg.PorsolError) as e:
            s.solve(pkg.Fluid(*prob.fluid), prob.sat, prob.bc_type, prob.bc_value, prob.src,
                    opts=pkg.default_solve_opts(linsolver_type=0, residual_tolerance=1e-12, linsolver_maxit=maxit))
        assert e.value.code == 1   # stopped at the iteration limit
        n.append(pkg.lib().porsol_launch_count() - before)
    s.close()
    return (n[1] - n[0]) / 4


def test_wide_levels_keep_their_own_launches(pkg, gpulib, workloads):
    """One block takes longer over a level of more than 512 rows than a launch does: 10^3 cells are swept in one
    launch (with the CG's four), 36^3, whose middle levels hold 600 to 1000 rows, in hundreds."""
    assert launches_per_iteration(pkg, workloads, (10, 10, 10)) == 5
    assert launches_per_iteration(pkg, workloads, (36, 36, 36)) > 100
