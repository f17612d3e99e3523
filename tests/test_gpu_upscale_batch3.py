"""The batched CG that runs the three directions together, at the edges of its layout: sub-grids of less
than, about and many times one chunk of 2048 unknowns, one sub-grid alone, every preconditioner, and the
errors of a solve that stops early.

Each sub-grid and direction is solved to a residual reduction of 1e-12; the effective tensor's error is
that of a flux of the solve, below 1e-9 (FP64) and 1e-8 (mixed) as for the parity at size."""
import numpy as np
import pytest

from upscaling import oracle_keff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sides", [[2], [9], [3, 8, 9, 2, 13], [2] * 40])
@pytest.mark.parametrize("ltype,precision", [(1, 0), (1, 1), (0, 0), (2, 1)])
def test_directions_together_match_oracle(pkg, gpulib, orc, workloads, sides, ltype, precision):
    union, _, K = workloads.periodic_subgrids(seed=5, sides=sides)
    s = pkg.PressureSolver()
    o = pkg.default_solve_opts(residual_tolerance=1e-12, precision=precision, linsolver_type=ltype)
    keff, st = s.upscale_periodic(union, union.cellpos, union.partner, union.side, K.ravel(), o)
    again, st2 = s.upscale_periodic(union, union.cellpos, union.partner, union.side, K.ravel(), o)
    assert np.array_equal(keff, again) and st.iterations == st2.iterations
    for g in sorted({0, len(sides) // 2, len(sides) - 1}):
        c0, c1 = union.cellpos[g], union.cellpos[g + 1]
        ref = oracle_keff(orc, union.grids[g], K[c0:c1])
        assert np.abs(keff[g] - ref).max() < (1e-8 if precision else 1e-9) * np.abs(ref).max()
    s.close()


def test_stops_at_the_iteration_limit(pkg, gpulib, workloads):
    union, _, K = workloads.periodic_subgrids(seed=6, sides=[6, 11])
    s = pkg.PressureSolver()
    with pytest.raises(pkg.PorsolError) as e:
        s.upscale_periodic(union, union.cellpos, union.partner, union.side, K.ravel(),
                           pkg.default_solve_opts(residual_tolerance=1e-12, linsolver_maxit=3))
    assert e.value.code == 1
    keff, st = s.upscale_periodic(union, union.cellpos, union.partner, union.side, K.ravel(),
                                  pkg.default_solve_opts(residual_tolerance=1e-12))
    assert np.isfinite(keff).all() and st.iterations > 9
    s.close()


@pytest.mark.parametrize("schedule", ["batched", "persistent"])
def test_other_groupings_of_one_union(pkg, gpulib, workloads, schedule):
    """The unknown ranges stay from call to call: another grouping of the same union's cells, another union
    and the first ones again give what a new solver gives."""
    calls = []
    for seed, sides in ((5, [4, 6, 5]), (7, [6, 4])):
        union, _, K = workloads.periodic_subgrids(seed=seed, sides=sides)
        calls.append((union, union.cellpos, K))
        calls.append((union, np.ascontiguousarray(union.cellpos[[0, 1, -1]] if len(sides) > 2 else
                                                  union.cellpos[[0, -1]]), K))
    o = pkg.default_solve_opts(residual_tolerance=1e-11, precision=1)

    def run(s, c):
        if schedule == "persistent":
            s.set_upscale_schedule(pkg.UPSCALE_PERSISTENT, 512, 0)
        try:
            return s.upscale_periodic(c[0], c[1], c[0].partner, c[0].side, c[2].ravel(), o)[0]
        except pkg.PorsolError as e:
            assert len(c[1]) < 3 or c[1] is not c[0].cellpos
            return np.array([e.code])

    s = pkg.PressureSolver()
    for i in (0, 1, 1, 0, 2, 3, 0, 3):
        fresh = pkg.PressureSolver()
        assert np.array_equal(run(s, calls[i]), run(fresh, calls[i]))
        fresh.close()
    s.close()
