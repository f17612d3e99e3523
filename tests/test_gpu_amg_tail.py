"""The AMG levels that run as one cluster launch, at the sizes where their number and shape change: from
hierarchies of a single dense level to three cluster levels, rows that do not divide by the blocks, both
precisions, uneven rows (full tensors) and isolated Dirichlet rows.

The preconditioner only changes by the order of its sums, so the converged answer is the oracle's: at a
residual reduction of 1e-13 both sides are within about 1e-12 times the condition of the recovery
(below 1e3 here) of the exact solution."""
import numpy as np
import pytest

from parity import gpu_solve, oracle_solve, relmax

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dims", [(2, 2, 2), (5, 4, 3), (9, 7, 5), (17, 13, 11), (31, 23, 17), (40, 33, 21), (64, 5, 3)])
def test_cluster_levels_match_oracle(pkg, gpulib, orc, workloads, dims, precision):
    prob = workloads.layered_lognormal(dims=dims, seed=9, sat=np.full(int(np.prod(dims)), 0.2))
    g = gpu_solve(pkg, prob, ltype=1, tol=1e-13, precision=precision)
    o = oracle_solve(orc, prob, tol=1e-14, dirichlet_guess=True)
    for k in ("p", "v", "pi"):
        assert relmax(g[k], o[k]) < 1e-9
    assert g["stats"].iterations <= 60


@pytest.mark.parametrize("precision", [0, 1])
def test_cluster_levels_on_full_tensors(pkg, gpulib, orc, workloads, cart, precision):
    from tensor_mobility import tensor_problem
    g, K, lam, rlam, bct, bcv, src = tensor_problem(workloads, cart, dims=(23, 19, 13))
    s = pkg.PressureSolver()
    s.init(g, K.ravel(), (0.0, 0.0, 0.3), bct)
    s.solve(pkg.Fluid(pkg.FLUID_TENSOR, 1.0, 1.0, 0.0, 0.0), lam.ravel(), bct, bcv, src, mobdens=rlam.ravel(),
            opts=pkg.default_solve_opts(residual_tolerance=1e-13, precision=precision))
    o = orc.OraclePressure(g, bct)
    o.compute_inner_products(K.ravel(), (0.0, 0.0, 0.3))
    assert o.solve_tensor(lam.ravel(), rlam.ravel(), bct, bcv, src, tol=1e-14) == 0
    for a, b in zip(s.solution(), o.solution()):
        assert relmax(a, b) < 1e-9
