"""The transport sub-step kernels against the oracle at the sizes where their layouts change: cells
with no, six and more than six inflow faces, partial warps, a single cell, boundary inflow, rock tables
searched inside, outside and at repeated rows.

The kernels' sums, quotients and table values differ from the oracle's by a few roundings of the
increment (at most 16 per face term), so after n sub-steps of at most 12 terms the saturations agree
to 12 * 16 * n * 2^-53 < 1e-12 for the n <= 40 used here."""
import numpy as np
import pytest

import capillary as cp
import hexgrids
from parity import relmax

pytestmark = pytest.mark.gpu


def star(leaves):
    """A hub with one face to each leaf; every leaf also has one boundary face."""
    rng = np.random.default_rng(leaves)
    nrm = rng.normal(size=(leaves, 3))
    nrm /= np.linalg.norm(nrm, axis=1, keepdims=True)
    hub = (1.0, np.zeros(3), [(1 + i, 0, 0.5, 0.5 * nrm[i], nrm[i]) for i in range(leaves)])
    leaf = [(0.5, nrm[i], [(0, 0, 0.5, 0.5 * nrm[i], -nrm[i]), (-1, 1, 0.5, 1.5 * nrm[i], nrm[i])])
            for i in range(leaves)]
    return hexgrids.FlatGrid([hub] + leaf)


def antisymmetric_flux(g, rng):
    """A flux per face, the same with opposite signs on its two half-faces."""
    cell = np.repeat(np.arange(g.num_cells), np.diff(g.facepos))
    q = rng.normal(size=len(cell))
    area = np.asarray(g.area)
    for c in range(g.num_cells):
        for h in range(g.facepos[c], g.facepos[c + 1]):
            n = g.neighbour[h]
            if n > c:
                back = [x for x in range(g.facepos[n], g.facepos[n + 1])
                        if g.neighbour[x] == c and np.allclose(g.fnormal[x], -g.fnormal[h])
                        and np.isclose(area[x], area[h])]
                free = [x for x in back if np.allclose(g.fcentroid[x], g.fcentroid[h])] or back
                q[free[0]] = -q[h]
    return q


GRIDS = {
    "one": lambda cart: cart.CartesianGrid(1, 1, 1),
    "line31": lambda cart: cart.CartesianGrid(31, 1, 1),
    "line33": lambda cart: cart.CartesianGrid(33, 1, 1),
    "box": lambda cart: cart.CartesianGrid(9, 7, 5),
    "star6": lambda cart: star(6),
    "star9": lambda cart: star(9),
    "refined": lambda cart: hexgrids.refined_top(),
}


def tables():
    t = [cp.rock_table(0.1, 0.9), cp.rock_table(0.2, 0.8, n=2), cp.rock_table(0.0, 1.0, n=11, ew=3.0, eo=1.5)]
    t[2] = np.insert(t[2], 5, t[2][5], axis=0)   # a repeated row
    return t


@pytest.mark.parametrize("name", list(GRIDS))
@pytest.mark.parametrize("form", ["viscous", "viscous_tables", "all_tables", "gravity"])
def test_substeps_match_oracle(pkg, gpulib, orc, cart, name, form):
    g = GRIDS[name](cart)
    nc, nhf = g.num_cells, int(g.facepos[-1])
    rng = np.random.default_rng(7 + nc)
    K = np.zeros((nc, 9))
    K[:, 0] = K[:, 4] = K[:, 8] = np.exp(rng.normal(0.0, 1.0, nc))
    poro = rng.uniform(0.1, 0.4, nc)
    q = antisymmetric_flux(g, rng)
    if name == "star9":
        q[:9] = -np.abs(q[:9])            # nine inflow faces of the hub
        q[9::2] = -q[:9]
    sat = rng.uniform(0.0, 1.0, nc)
    sat[: nc // 4] = rng.choice([0.0, 0.1, 0.2, 0.5, 0.9, 1.0], nc // 4)
    st, sv = np.full(nhf, pkg.BC_DIRICHLET, np.int32), rng.uniform(0.0, 1.0, nhf)
    inj = rng.normal(size=nc) * 0.1
    tab = form.endswith("tables")
    everything = form == "all_tables"
    grav = (0.0, 0.0, 0.0) if form.startswith("viscous") else (1e-4, -2e-4, 1e-3)
    opt = dict(method_capillary=int(everything), clamp_sat=1)
    T = pkg.TransportSolver()
    T.init(g, K.ravel(), poro, pkg.Fluid(pkg.FLUID_COREY2, cp.MU1, cp.MU2, cp.RHO1, cp.RHO2), st, sv,
           opts=pkg.default_transport_opts(**opt))
    fluid = orc.Fluid(cp.MU1, cp.MU2, cp.RHO1, cp.RHO2)
    if tab:
        rocks = np.arange(nc, dtype=np.int32) % 3
        T.set_rock_tables(tables(), rocks, True, 0.05)
        rt = orc.RockTables(tables(), rocks, True, 0.05)
        fluid = rt.fluid(cp.MU1, cp.MU2, cp.RHO1, cp.RHO2)
    O = orc.OracleTransport(g, K.ravel(), poro, fluid, st, sv, opts=orc.TransportOpts.defaults(**opt))
    t = 4.5 * O.cfl(q, grav)
    rc, s_orc, ns, _ = O.solve(sat, t, q, injection=inj, grav=grav)
    assert rc == 0 and 1 <= ns <= 40
    s_gpu, stats = T.solve(sat, t, q, injection=inj, grav=grav)
    assert stats.small_steps == ns
    assert relmax(s_gpu, s_orc) < 1e-12
