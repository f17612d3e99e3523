"""Rounding of the viscous transport sub-steps against extended precision (numpy's longdouble, 64 bits of mantissa
or more).

A sub-step adds one rounded increment to each saturation.  For s in [1/2, 1) the error of that addition is uniform
within 2^-54, its standard deviation 2^-53 / sqrt(12) = 0.29 * 2^-53; the increment itself is below 1/8 and carries
at most some eight roundings of its own, at most as much again.  Upstream weighting only averages what is there,
so after n sub-steps the saturations are off by less than sqrt(n) * 0.58 * 2^-53 in the root mean square: 6.5e-16
for the 100 here.  Coefficients that carry a rounding from sub-step to sub-step, or sums started from the saturation,
add up instead and exceed that."""
import numpy as np
import pytest

import capillary as cp

pytestmark = pytest.mark.gpu

L = np.longdouble


def divergence_free(rng, nx, ny, nz):
    """Half-face fluxes of a uniform flow along x plus the curl of a random potential, in multiples of 2^-20 (sums
    of a cell's fluxes are exact)."""
    q = 2.0 ** -20

    def potential(*shape):
        return np.round(0.4 * rng.standard_normal(shape) / q) * q

    Ax, Ay, Az = potential(nz + 1, ny + 1, nx), potential(nz + 1, ny, nx + 1), potential(nz, ny + 1, nx + 1)
    for A, axes in ((Ax, (0, 1)), (Ay, (0,)), (Az, (1,))):
        for ax in axes:
            A[tuple(slice(None) if k != ax else [0, -1] for k in range(3))] = 0.0
    qx = 1.0 + (Az[:, 1:] - Az[:, :-1]) - (Ay[1:] - Ay[:-1])
    qy = (Ax[1:] - Ax[:-1]) - (Az[:, :, 1:] - Az[:, :, :-1])
    qz = (Ay[:, :, 1:] - Ay[:, :, :-1]) - (Ax[:, 1:] - Ax[:, :-1])
    return np.stack([-qx[:, :, :-1], qx[:, :, 1:], -qy[:, :-1], qy[:, 1:], -qz[:-1], qz[1:]], axis=-1).reshape(-1, 6)


def extended(g, q, pv, s, sbc, time, n):
    nb = np.asarray(g.neighbour).reshape(-1, 6)
    q, s, w = q.astype(L), s.astype(L), L(time / n) / pv.astype(L)
    out = q >= 0

    def f(x):
        m0 = x * x / L(cp.MU1)
        return m0 / (m0 + (1 - x) * (1 - x) / L(cp.MU2))

    fb = f(L(sbc))
    for _ in range(n):
        fs = f(s)
        up = np.where(out, fs[:, None], np.where(nb >= 0, fs[np.maximum(nb, 0)], fb))
        s = s - w * (up * q).sum(1)
    return s


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_viscous_substeps_round_once(pkg, gpulib, cart, seed):
    rng = np.random.default_rng(seed)
    nx, ny, nz = 20, 16, 12
    g = cart.CartesianGrid(nx, ny, nz, 1.0 / nx, 1.0 / ny, 1.0 / nz)
    nc, nhf = g.num_cells, int(g.facepos[-1])
    K = np.zeros((nc, 9))
    K[:, 0] = K[:, 4] = K[:, 8] = 1.0
    poro = rng.uniform(0.1, 0.4, nc)
    q = divergence_free(rng, nx, ny, nz)
    sat, sbc = rng.uniform(0.3, 0.9, nc), 0.95
    T = pkg.TransportSolver()
    T.init(g, K.ravel(), poro, pkg.Fluid(pkg.FLUID_COREY2, cp.MU1, cp.MU2, cp.RHO1, cp.RHO2),
           np.full(nhf, pkg.BC_DIRICHLET, np.int32), np.full(nhf, sbc),
           opts=pkg.default_transport_opts(method_capillary=0, method_gravity=0, minimum_small_steps=100,
                                           maximum_small_steps=100))
    pv = np.asarray(g.volume) * poro
    through = np.maximum(q, 0).sum(1)
    time = 100 * 0.03 * (pv / through).min()      # increments below 1/8: f' is below 4 here
    s, st = T.solve(sat, time, q.ravel())
    assert st.small_steps == 100 and st.repeats == 0
    err = (s.astype(L) - extended(g, q, pv, sat, sbc, time, 100)).astype(float)
    assert np.sqrt((err ** 2).mean()) < 10.0 * 0.58 * 2.0 ** -53
    assert np.abs(np.asarray(s) - sat).max() > 0.1   # the flow did move
