"""The work a user of this library has it do, as measurable cases.

A case is a dict of plain values.  Its kind names the call:

  pressure    IncompFlowSolverHybrid::solve + postProcessFluxes + getSolution on a kept solver (grid
              topology, inner products): cell pressures, half-face fluxes, face pressures
  adjoint     one inversion step: new permeabilities, forward solve, gradient of a mismatch objective
  upscale     effective permeability tensors of a batch of periodic sub-grids, new permeabilities per call
  transport   EulerUpstream::transportSolve over a given time with given fluxes
  capillary   ImplicitCapillarity::transportSolve

Linear systems are solved to a residual reduction of 1e-13, the tolerance of the repository's parity
tests, so that the outputs are the system's and not the stopping iteration's.  `host` cases call the
host-array entry points as the C++ drop-in does; the others keep their arrays on the device as a
device-resident simulator does.  exact() restates the discretisation in plain torch, in 64 bits.
"""
import functools
import importlib
import math

import numpy as np
import torch

lib = importlib.import_module("opm-porsol_gb300")
cartesian = importlib.import_module("opm-porsol_gb300.cartesian")

MD = 9.869233e-16          # m^2
TOL = 1e-13
F64 = torch.float64


# ------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: the plain drop-in on 1000 cells, ILU0-CG (the reference's type 0), host arrays
        dict(name="unit_cube_ilu0", kind="pressure", nx=10, ny=10, nz=10, field="iid", fluid="cellwise", host=True,
             mixed=False, solver=0),
        # a sector-model solve: small and ragged, gravity and wells, the default AMG-CG in FP64, host arrays
        dict(name="sector_gravity_fp64", kind="pressure", nx=31, ny=23, nz=17, field="layered", fluid="corey",
             host=True, mixed=False, solver=1, gravity=True, wells=True),
        # a deformed (corner-point like) grid with full tensors and tensor mobilities, host arrays
        dict(name="tensor_hex_mixed", kind="pressure", nx=61, ny=47, nz=29, field="full", fluid="tensor", host=True,
             mixed=True, solver=1, hexgrid=True, gravity=True),
        # two-phase pressure solve on 500k anisotropic cells, device-resident
        dict(name="anisotropic_500k_mixed", kind="pressure", nx=100, ny=100, nz=50, field="anisotropic",
             fluid="corey", host=False, mixed=True, solver=1),
        # the headline: 1M layered cells, every step of an IMPES run; mixed and the plain FP64 drop-in
        dict(name="layered_1m_mixed", kind="pressure", nx=200, ny=200, nz=25, field="layered", fluid="corey",
             host=False, mixed=True, solver=1),
        dict(name="layered_1m_fp64", kind="pressure", nx=200, ny=200, nz=25, field="layered", fluid="corey",
             host=False, mixed=False, solver=1),
        # one step of a permeability inversion on 131k cells (both directions of the path)
        dict(name="adjoint_131k_mixed", kind="adjoint", nx=64, ny=64, nz=32, mixed=True),
        # batched upscaling: uneven sub-grids, hierarchy schedule (mixed) and the persistent launch
        dict(name="upscale_48_mixed", kind="upscale", num=48, nmin=8, nmax=32, mixed=True, persistent=False),
        dict(name="upscale_192_persistent", kind="upscale", num=192, nmin=5, nmax=17, mixed=False, persistent=True),
        # explicit viscous transport between two pressure solves, about 100 sub-steps, device-resident
        dict(name="transport_1m", kind="transport", nx=200, ny=200, nz=25, substeps=100, rock=False, host=False),
        # the same with gravity, rock tables and the capillary term on a ragged box, host arrays
        dict(name="transport_rock_167k", kind="transport", nx=83, ny=65, nz=31, substeps=12, rock=True, host=True),
        # implicit capillary step of a coupled run, two rocks
        dict(name="capillary_250k_mixed", kind="capillary", nx=100, ny=100, nz=25, mixed=True),
    ]


def draw(rng):
    def cells(lo, hi, nz_lo, nz_hi):
        """Uneven dimensions whose product is log-uniform in [lo, hi]."""
        n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        nz = rng.randint(nz_lo, nz_hi)
        a = math.sqrt(n / nz) * math.exp(rng.uniform(-0.4, 0.4))
        nx = max(5, min(400, round(a)))
        ny = max(5, min(400, round(n / nz / nx)))
        return dict(nx=nx, ny=ny, nz=nz)

    kind = rng.choice(["pressure"] * 5 + ["adjoint", "upscale", "upscale", "transport", "transport", "capillary"])
    mixed = rng.random() < 0.5
    if kind == "pressure":
        form = rng.choice(["ilu0", "corey", "corey", "aniso", "tensor"])
        if form == "ilu0":
            return dict(kind=kind, **cells(300, 6000, 5, 12), field="iid", fluid="cellwise", host=True, mixed=False,
                        solver=0)
        if form == "tensor":
            return dict(kind=kind, **cells(2e3, 1.2e5, 7, 30), field="full", fluid="tensor", host=True, mixed=mixed,
                        solver=1, hexgrid=rng.random() < 0.6, gravity=rng.random() < 0.5)
        host = rng.random() < 0.4
        return dict(kind=kind, **cells(2e3, 9e5, 9, 45), field="layered" if form == "corey" else "anisotropic",
                    fluid="corey", host=host, mixed=mixed, solver=2 if rng.random() < 0.15 else 1,
                    gravity=rng.random() < 0.3, wells=rng.random() < 0.3)
    if kind == "adjoint":
        return dict(kind=kind, **cells(4e3, 2.5e5, 9, 33), mixed=mixed)
    if kind == "upscale":
        persistent = rng.random() < 0.5
        nmax = rng.randint(9, 17 if persistent else 26)
        return dict(kind=kind, num=rng.randint(5, 150 if persistent else 40), nmin=rng.randint(5, 8), nmax=nmax,
                    mixed=mixed, persistent=persistent)
    if kind == "transport":
        rock = rng.random() < 0.5
        return dict(kind=kind, **cells(1e3, 2.5e5 if rock else 9e5, 5, 33), rock=rock, host=rng.random() < 0.5,
                    substeps=rng.randint(4, 12) if rock else rng.randint(5, 100))
    return dict(kind=kind, **cells(4e3, 2.5e5, 9, 30), mixed=mixed)


def work(case):
    """Inputs read once and outputs written once.  The packed inner products (21 values a cell) are an
    input of a pressure solve; flops are those of assembly and recovery (or of the sub-steps' upstream
    terms), the part that does not depend on the solver."""
    kind = case["kind"]
    if kind == "upscale":
        nc = float((_sides(case) ** 3).sum())
        return {"bytes": nc * (72 + 6 * 4 + 6 * 4) + 72.0 * case["num"], "flops": 3 * nc * 500}
    nc = float(case["nx"] * case["ny"] * case["nz"])
    nhf, n = 6 * nc, 3 * nc
    if kind == "transport":
        return {"bytes": 16 * nc + 8 * nhf + (80 * nc if case["rock"] else 8 * nc),
                "flops": nc * case["substeps"] * (400.0 if case["rock"] else 40.0)}
    if kind == "capillary":
        return {"bytes": 21 * 8 * nc + 16 * nc + 8 * nhf + 4 * nhf + 8 * nhf + 12 * nc, "flops": nc * 700}
    if case.get("fluid") == "tensor":   # rebuilt per solve from geometry, permeability and the mobility tensors
        static = 56 * nhf + 104 * nc + (144 if case.get("gravity") else 72) * nc
    else:
        static = 21 * 8 * nc + 8 * nc
    b = static + 8 * nc + 12 * nhf + 8 * nc + 8 * nhf + 8 * n
    if kind == "adjoint":
        b += 72 * nc + 8 * nhf + 24 * nc
    return {"bytes": b, "flops": nc * 500.0 * (2 if kind == "adjoint" else 1)}


# ------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=3)
def _grid(nx, ny, nz, size, hexgrid):
    """The grid is geometry alone and the same for every seed: kept between preparations."""
    if not hexgrid:
        return cartesian.CartesianGrid(nx, ny, nz, *(s / n for s, n in zip(size, (nx, ny, nz))))

    def bend(x):
        y = x.copy()
        y[:, 0] += 0.04 * np.sin(2 * np.pi * x[:, 1]) * np.sin(np.pi * x[:, 2])
        y[:, 1] += 0.04 * np.sin(2 * np.pi * x[:, 2]) * np.sin(np.pi * x[:, 0])
        y[:, 2] += 0.04 * np.sin(2 * np.pi * x[:, 0]) * np.sin(np.pi * x[:, 1])
        return y * np.asarray(size)
    return cartesian.HexGrid(nx, ny, nz, bend)


def _grid_of(case):
    # physical boxes for the transport with gravity and capillarity, unit cubes otherwise
    size = (10.0 * case["nx"], 10.0 * case["ny"], 2.0 * case["nz"]) if case.get("rock") else (1.0, 1.0, 1.0)
    return _grid(case["nx"], case["ny"], case["nz"], size, bool(case.get("hexgrid")))


def _correlated(rng, dims, cells, sigma):
    """Gaussian field with correlation length `cells`, periodic, scaled to standard deviation sigma."""
    nx, ny, nz = dims
    f = np.fft.rfftn(rng.standard_normal((nz, ny, nx)))
    w = 1.0
    for ax, n in enumerate((nz, ny, nx)):
        k = np.fft.rfftfreq(n) if ax == 2 else np.fft.fftfreq(n)
        g = np.exp(-2.0 * (np.pi * cells * k) ** 2)
        w = w * g.reshape([-1 if a == ax else 1 for a in range(3)])
    z = np.fft.irfftn(f * w, s=(nz, ny, nx), axes=(0, 1, 2))
    return ((z - z.mean()) / z.std() * sigma).ravel()


def _permeability(rng, case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    nc = nx * ny * nz
    field = case.get("field", "layered")
    K = np.zeros((nc, 9))
    if field == "iid":
        k = np.exp(rng.normal(math.log(100 * MD), 1.0, nc))
    elif field == "correlated":
        k = np.exp(math.log(100 * MD) + _correlated(rng, (nx, ny, nz), 4.0, 1.0))
    elif field == "anisotropic":
        k = np.exp(math.log(100 * MD) + _correlated(rng, (nx, ny, nz), 5.0, 2.0))
    elif field == "full":
        A = rng.normal(size=(nc, 3, 3)) * 0.4
        K3 = (np.eye(3) + np.einsum("cij,ckj->cik", A, A)) * (100 * MD * np.exp(rng.normal(0.0, 1.0, nc)))[:, None, None]
        return K3.reshape(nc, 9)
    else:
        means = rng.normal(math.log(100 * MD), 1.0, nz)
        k = np.exp(rng.normal(np.repeat(means, nx * ny), 2.0))
    K[:, 0] = K[:, 4] = k
    K[:, 8] = 0.1 * k if field == "anisotropic" else k
    return K


MU, RHO = (1e-3, 1e-2), (1000.0, 850.0)


def _pressure_inputs(case, seed):
    rng = np.random.default_rng(seed)
    g = _grid_of(case)
    nc = g.num_cells
    d = dict(K=_permeability(rng, case))
    d["grav"] = (0.0, 0.0, 9.81e-4) if case.get("gravity") else (0.0, 0.0, 0.0)
    d["bct"] = np.where((g.side == 1) | (g.side == 2), lib.BC_DIRICHLET, lib.BC_NEUMANN).astype(np.int32)
    d["bcv"] = np.where(g.side == 1, 1.0, 0.0)
    d["src"] = np.zeros(nc)
    if case.get("wells"):
        at = rng.choice(nc, 6, replace=False)
        d["src"][at] = np.array([1, 1, 1, -1, -1, -1]) * 1e-11
    d["mobdens"] = None
    fluid = case.get("fluid", "cellwise")
    if fluid == "corey":
        # a flood under way: water behind a ragged front, connate water ahead of it
        front = 0.5 + 0.2 * rng.standard_normal(nc)
        d["sat"] = np.clip(np.where(g.ccentroid[:, 0] < 0.4, 0.3 + 0.5 * front, 0.1 * front), 0.0, 1.0)
        d["fluid"] = lib.Fluid(lib.FLUID_COREY2, *MU, *RHO)
    elif fluid == "tensor":
        K3 = d["K"].reshape(nc, 3, 3)
        a = rng.uniform(50.0, 200.0, nc)[:, None, None]
        b = rng.uniform(0.0, 50.0, nc)[:, None, None] / np.trace(K3, axis1=1, axis2=2)[:, None, None]
        d["sat"] = (a * np.eye(3) + b * K3).reshape(nc, 9)
        d["mobdens"] = (1000.0 * a * np.eye(3) + 850.0 * b * K3).reshape(nc, 9)
        d["fluid"] = lib.Fluid(lib.FLUID_TENSOR, 1.0, 1.0, 0.0, 0.0)
    else:
        d["sat"] = np.ones(nc)
        d["mobdens"] = np.zeros(nc)
        d["fluid"] = lib.Fluid(lib.FLUID_CELLWISE, 1.0, 1.0, 0.0, 0.0)
    return d


def _adjoint_inputs(case, seed):
    case = dict(case, field="correlated")
    d = _pressure_inputs(case, seed)
    rng = np.random.default_rng(seed + 77)
    nc = len(d["src"])
    obs = rng.choice(nc, 50, replace=False)
    d["w"] = np.zeros(nc)
    d["w"][obs] = 1.0
    d["target"] = np.zeros(nc)
    d["target"][obs] = rng.normal(0.5, 0.1, 50)
    d["u"] = np.where(_grid_of(case).side == 2, 1.0, 0.0)
    return d


def _sides(case):
    """The batch's shape belongs to the case, not to the seed: a program upscales realisations of it."""
    r = np.random.default_rng(1000 * case["num"] + 10 * case["nmax"] + case["nmin"])
    return r.integers(case["nmin"], case["nmax"] + 1, size=case["num"])


@functools.lru_cache(maxsize=3)
def _union(sides):
    return cartesian.UnionGrid([cartesian.CartesianGrid(n, n, n, unique_bids=True) for n in sides])


def _union_of(case):
    return _union(tuple(int(n) for n in _sides(case)))


def _upscale_perm(case, seed):
    """Full tensors: log-normal principal values (sigma 1.5) on uniformly random axes."""
    r = torch.Generator(device="cuda").manual_seed(int(seed))
    nc = _union_of(case).num_cells
    q = torch.randn(nc, 4, generator=r, device="cuda", dtype=F64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).view(nc, 3, 3)
    lam = torch.exp(math.log(100 * MD) + 1.5 * torch.randn(nc, 3, generator=r, device="cuda", dtype=F64))
    K = torch.einsum("cij,cj,ckj->cik", R, lam, R)
    return (0.5 * (K + K.transpose(1, 2))).reshape(nc, 9).cpu().numpy()


def _rocks():
    def table(lo, hi, n, jmax, ew, eo):
        s = np.linspace(lo, hi, n)
        e = (s - lo) / (hi - lo)
        return np.column_stack([s, e ** ew, (1 - e) ** eo, jmax * (1 - e) ** 2 + 0.05 * (1 - e)])
    return [table(0.1, 0.9, 17, 2.0, 2.0, 2.0), table(0.15, 0.85, 11, 3.0, 3.0, 1.5)]


def _flux(rng, case, g):
    """Half-face fluxes without divergence: a layered flow along x plus the curl of a random vector
    potential that vanishes on the box's walls.  Both half-faces of a face carry the same value."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    hx, hy, hz = g.h
    u = np.exp(rng.normal(0.0, 0.7, nz)) * (1e-6 if case.get("rock") else 1e-10)
    s = 0.5 * u.mean() * min(hy, hz)
    Ay = s * rng.standard_normal((nz + 1, ny, nx + 1)) * hy      # potential times edge length
    Az = s * rng.standard_normal((nz, ny + 1, nx + 1)) * hz
    Ax = s * rng.standard_normal((nz + 1, ny + 1, nx)) * hx
    Ay[[0, -1]] = 0.0
    Az[:, [0, -1]] = 0.0
    Ax[[0, -1]] = 0.0
    Ax[:, [0, -1]] = 0.0
    qx = u[:, None, None] * hy * hz + (Az[:, 1:] - Az[:, :-1]) - (Ay[1:] - Ay[:-1])        # (nz, ny, nx+1)
    qy = (Ax[1:] - Ax[:-1]) - (Az[:, :, 1:] - Az[:, :, :-1])                              # (nz, ny+1, nx)
    qz = (Ay[:, :, 1:] - Ay[:, :, :-1]) - (Ax[:, 1:] - Ax[:, :-1])                        # (nz+1, ny, nx)
    q = np.stack([-qx[:, :, :-1], qx[:, :, 1:], -qy[:, :-1], qy[:, 1:], -qz[:-1], qz[1:]], axis=-1)
    return np.ascontiguousarray(q.reshape(-1))


def _transport_inputs(case, seed):
    rng = np.random.default_rng(seed)
    g = _grid_of(case)
    nc = g.num_cells
    d = dict(K=_permeability(rng, case), poro=rng.uniform(0.15, 0.3, nc), flux=_flux(rng, case, g))
    d["sat_type"] = np.full(g.num_half_faces, lib.BC_DIRICHLET, np.int32)
    x = g.ccentroid[:, 0] / (g.h[0] * case["nx"])
    if case["rock"]:
        d["sat"] = rng.uniform(0.35, 0.6, nc)
        d["sat_value"] = np.full(g.num_half_faces, 0.85)
        d["cell_rock"] = ((np.arange(nc) // (case["nx"] * case["ny"])) % 2).astype(np.int32)
        d["tables"], d["sct"], d["grav"] = _rocks(), 1e-3, (0.0, 0.0, 9.81)
    else:
        d["sat"] = np.clip(0.9 - 2.0 * x, 0.0, 1.0) * rng.uniform(0.8, 1.0, nc)
        d["sat_value"] = np.ones(g.num_half_faces)
        d["cell_rock"], d["tables"], d["sct"], d["grav"] = None, None, 1.0, (0.0, 0.0, 0.0)
    d["fluid"] = lib.Fluid(lib.FLUID_COREY2, *MU, *RHO)
    # the report step: that many steps of the CFL bound
    d["time"] = (case["substeps"] - 0.5) * _cfl_step(case, g, d)
    return d


def _capillary_inputs(case, seed):
    rng = np.random.default_rng(seed)
    g = _grid_of(case)
    nc = g.num_cells
    d = dict(K=_permeability(rng, case), poro=rng.uniform(0.15, 0.3, nc), flux=_flux(rng, case, g))
    d["flux"] *= 0.1   # the pressure drop of 1 Pa over the unit box that the capillary pressure competes with
    d["sat"] = rng.uniform(0.3, 0.6, nc)
    d["sat_type"] = np.full(g.num_half_faces, lib.BC_DIRICHLET, np.int32)
    d["sat_value"] = np.full(g.num_half_faces, 0.85)
    d["cell_rock"] = ((np.arange(nc) // (case["nx"] * case["ny"])) % 2).astype(np.int32)
    d["tables"], d["sct"], d["grav"] = _rocks(), 1e-6, (0.0, 0.0, 0.0)
    d["bct"] = np.where((g.side == 1) | (g.side == 2), lib.BC_DIRICHLET, lib.BC_NEUMANN).astype(np.int32)
    d["bcv"] = np.where(g.side == 1, 1.0, 0.0)
    d["fluid"] = lib.Fluid(lib.FLUID_COREY2, *MU, *RHO)
    return d


# ------------------------------------------------------------------------------------ the calls
class _Device:
    """A device array of the library, readable as a tensor while its solver lives."""

    def __init__(self, pointer, n):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(pointer, False), version=3, strides=None)


def _view(pointer, n):
    return torch.as_tensor(_Device(pointer, n), device="cuda")


def prepare(case, seed):
    s = dict(case=case)
    kind = case["kind"]
    precision = lib.MIXED if case.get("mixed") else lib.FP64
    if kind == "upscale":
        u = _union_of(case)
        s["union"], s["K"] = u, _upscale_perm(case, seed).ravel()
        P = s["P"] = lib.PressureSolver()
        P.set_upscale_schedule(lib.UPSCALE_PERSISTENT if case["persistent"] else lib.UPSCALE_AMG)
        s["opts"] = lib.default_solve_opts(residual_tolerance=TOL, precision=precision, linsolver_maxit=6000)
        # the batch's topology and schedule belong to the handle: one coarse call builds them
        first = lib.default_solve_opts(residual_tolerance=1e-2, precision=precision, linsolver_maxit=6000)
        P.upscale_periodic(u, u.cellpos, u.partner, u.side, s["K"], first)
        return s
    g = s["grid"] = _grid_of(case)
    if kind == "transport":
        d = s["d"] = _transport_inputs(case, seed)
        T = s["T"] = lib.TransportSolver()
        T.init(g, d["K"].ravel(), d["poro"], d["fluid"], d["sat_type"], d["sat_value"],
               opts=lib.default_transport_opts(method_gravity=int(case["rock"]), method_capillary=int(case["rock"])))
        if d["tables"] is not None:
            T.set_rock_tables(d["tables"], d["cell_rock"], True, d["sct"])
        if not case["host"]:
            s["sat0"], s["flux"] = (torch.from_numpy(d[k]).cuda() for k in ("sat", "flux"))
            s["sat"] = torch.empty_like(s["sat0"])
            torch.cuda.synchronize()
        return s
    if kind == "capillary":
        d = s["d"] = _capillary_inputs(case, seed)
        T = s["T"] = lib.TransportSolver()
        T.init(g, d["K"].ravel(), d["poro"], d["fluid"], d["sat_type"], d["sat_value"])
        T.set_rock_tables(d["tables"], d["cell_rock"], True, d["sct"])
        P = s["P"] = lib.PressureSolver()
        P.init(g, d["K"].ravel(), (0.0, 0.0, 0.0), d["bct"])
        s["opts"] = lib.default_capillary_opts(residual_tolerance=TOL, precision=precision)
        return s
    d = s["d"] = _adjoint_inputs(case, seed) if kind == "adjoint" else _pressure_inputs(case, seed)
    P = s["P"] = lib.PressureSolver()
    P.init(g, d["K"].ravel(), d["grav"], d["bct"])
    s["opts"] = lib.default_solve_opts(residual_tolerance=TOL, precision=precision, linsolver_type=case.get("solver", 1))
    if kind == "pressure" and not case["host"]:
        for k in ("sat", "bct", "bcv", "src"):
            s[k] = torch.from_numpy(d[k]).cuda()
        torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "upscale":
        u = s["union"]
        return s["P"].upscale_periodic(u, u.cellpos, u.partner, u.side, s["K"], s["opts"])[0]
    d = s["d"]
    if kind == "transport":
        if case["host"]:
            return s["T"].solve(d["sat"], d["time"], d["flux"], grav=d["grav"])[0]
        s["sat"].copy_(s["sat0"])
        torch.cuda.current_stream().synchronize()   # the solver has a stream of its own
        s["T"].solve_device(s["sat"].data_ptr(), d["time"], s["flux"].data_ptr(), grav=d["grav"])
        return s["sat"]
    if kind == "capillary":
        return s["T"].capillary_solve(s["P"], d["sat"], d["flux"], d["bct"], d["bcv"], opts=s["opts"])[0]
    P = s["P"]
    if kind == "adjoint":
        P.compute_inner_products(d["K"].ravel(), d["grav"])
        P.solve(d["fluid"], d["sat"], d["bct"], d["bcv"], d["src"], mobdens=d["mobdens"], opts=s["opts"])
        J, grad, _ = P.adjoint_gradient(d["w"], d["target"], d["u"])
        return dict(J=J, gradient=grad)
    if case["host"]:
        P.solve(d["fluid"], d["sat"], d["bct"], d["bcv"], d["src"], mobdens=d["mobdens"], opts=s["opts"])
        P.post_process_fluxes()
        p, v, f = P.solution()
    else:
        P.solve_device(d["fluid"], s["sat"].data_ptr(), s["bct"].data_ptr(), s["bcv"].data_ptr(), s["src"].data_ptr(),
                       opts=s["opts"])
        P.post_process_fluxes()
        g = s["grid"]
        # the library's arrays are valid until the next solve: a simulator keeps its own copy
        p, v, f = (_view(a, n).clone() for a, n in zip(P.solution_device(), (g.num_cells, g.num_half_faces, P.n)))
        torch.cuda.current_stream().synchronize()   # read before the solver's own stream writes them again
    return dict(pressure=p, outflux=v, face_pressure=f)


# ------------------------------------------------------------------------------------ 64-bit values
def exact(case, seed):
    kind = case["kind"]
    if kind == "transport":
        g, d = _grid_of(case), _transport_inputs(case, seed)
        return _exact_transport(case, g, d)
    if kind == "capillary":
        return _exact_capillary(case, _grid_of(case), _capillary_inputs(case, seed))
    if kind == "upscale":
        return _exact_upscale(_union_of(case), _upscale_perm(case, seed))
    d = _adjoint_inputs(case, seed) if kind == "adjoint" else _pressure_inputs(case, seed)
    g = _grid_of(case)
    if kind == "adjoint":
        return _exact_adjoint(g, d)
    M = _Mimetic(g, d["K"], *_mobilities(case, d), d["grav"], d["src"], d["bct"], d["bcv"])
    x = M.solve()
    p, v = M.recover(x)
    return dict(pressure=p, outflux=M.average(v), face_pressure=M.face_pressure(x))


def _t(a, dtype=F64):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda").to(dtype)


def _mobilities(case, d):
    """(lambda, sum rho lambda) per cell as 3x3 tensors or scalars."""
    if case.get("fluid") == "tensor":
        return _t(d["sat"]).view(-1, 3, 3), _t(d["mobdens"]).view(-1, 3, 3)
    if case.get("fluid") == "corey":
        s = _t(d["sat"])
        m1, m2 = s * s / MU[0], (1 - s) ** 2 / MU[1]
        return m1 + m2, RHO[0] * m1 + RHO[1] * m2
    return _t(d["sat"]), _t(d["mobdens"])


def _inner(g, K):
    """W = (N K N^T + 2 tr(K) A (I - Q Q^T) A) / |c| per cell and N, for six-faced cells."""
    a = g.arrays()
    nc = a["num_cells"]
    area = _t(a["area"]).view(nc, 6)
    N = _t(a["fnormal"]).view(nc, 6, 3) * area[:, :, None]
    X = (_t(a["fcentroid"]).view(nc, 6, 3) - _t(a["ccentroid"]).view(nc, 1, 3)) * area[:, :, None]
    X = X / X.norm(dim=1, keepdim=True)
    G = torch.linalg.inv(X.transpose(1, 2) @ X)
    P = torch.eye(6, dtype=F64, device="cuda") - X @ G @ X.transpose(1, 2)
    tr = K.diagonal(dim1=1, dim2=2).sum(1)
    W = N @ K @ N.transpose(1, 2) + 2 * tr[:, None, None] * area[:, :, None] * P * area[:, None, :]
    return W / _t(a["volume"])[:, None, None], N


def _pcg(A, d, b, blk, nblk):
    """Jacobi-CG for the columns of b, one recurrence per block and column, restarted from the true
    residual until that no longer falls."""
    one = nblk == 1

    def dot(u, v):
        w = u * v
        if one:
            return w.sum(0, keepdim=True)
        return torch.zeros(nblk, w.shape[1], dtype=F64, device="cuda").index_add_(0, blk, w)

    def each(c):
        return c if one else c[blk]

    x = torch.zeros_like(b)
    start = dot(b, b)
    start = torch.where(start > 0, start, torch.ones_like(start))
    last = torch.full_like(start, math.inf)
    best = x
    for _ in range(4):
        r = b - A @ x
        now = dot(r, r)
        if bool((now >= 0.25 * last).all()):
            break
        last, best = now, x.clone()
        z = r / d
        p, rz = z.clone(), dot(r, z)
        goal = 1e-31 * start
        for it in range(20000):
            q = A @ p
            pq = dot(p, q)
            go = (pq > 0) & (dot(r, r) > goal)                # a block that has converged stands still
            al = each(torch.where(go, rz / torch.where(go, pq, torch.ones_like(pq)), torch.zeros_like(pq)))
            x = x + al * p
            r = r - al * q
            z = r / d
            rz2 = dot(r, z)
            p = z + each(torch.where(rz > 0, rz2 / torch.where(rz > 0, rz, torch.ones_like(rz)), torch.zeros_like(rz))) * p
            rz = rz2
            if it % 50 == 49 and bool((dot(r, r) <= goal).all()):
                break
    return best


class _Mimetic:
    """The hybrid system of half-face pressures pi = x[dof] + off: S_c = B - F F^T / L, B = lambda W(K)."""

    def __init__(self, g, K, lam, rlam, grav, src, bct, bcv, dof=None, off=None, pinned=None):
        nc = g.num_cells
        K = _t(K).view(nc, 3, 3)
        gv = torch.tensor(grav, dtype=F64, device="cuda")
        if lam.dim() == 3:
            W, N = _inner(g, lam @ K)
            self.B = W
            Kg = (rlam @ (K @ gv)[:, :, None])[:, :, 0]
        else:
            W, N = _inner(g, K)
            self.B = W * lam[:, None, None]
            Kg = (K @ gv) * rlam[:, None]
        self.gf = (N @ Kg[:, :, None])[:, :, 0]
        self.F = self.B.sum(1)
        self.L = self.F.sum(1)
        self.g = _t(src) - self.gf.sum(1)
        self.nb = torch.as_tensor(g.neighbour, device="cuda").long().view(nc, 6)
        bct = _t(bct, torch.long).view(nc, 6)
        bcv = _t(bcv).view(nc, 6)
        bnd = self.nb < 0
        self.dirichlet = bnd & (bct == lib.BC_DIRICHLET)
        h = torch.where(bnd & (bct == lib.BC_NEUMANN), bcv, torch.zeros_like(bcv))
        # faces numbered at their first half-face, internal before boundary
        cell = torch.arange(nc, device="cuda")[:, None].expand(nc, 6)
        lf = torch.arange(6, device="cuda")[None].expand(nc, 6)
        first = (self.nb > cell)
        num = torch.cumsum(first.reshape(-1), 0).view(nc, 6) - 1
        self.twin = torch.where(bnd, torch.full_like(self.nb, -1), self.nb * 6 + (lf ^ 1))
        ni = int(first.sum())
        nbd = torch.cumsum(bnd.reshape(-1), 0).view(nc, 6) - 1 + ni
        self.dof = torch.where(bnd, nbd, torch.where(first, num, num.reshape(-1)[self.twin.clamp(min=0)]))
        self.n = ni + int(bnd.sum())
        self.off = torch.where(self.dirichlet, bcv, torch.zeros_like(bcv))
        if dof is not None:
            self.dof, self.off = dof(self.dof), off
        S = self.B - self.F[:, :, None] * self.F[:, None, :] / self.L[:, None, None]
        rl = self.gf - h + (self.g / self.L)[:, None] * self.F
        loc = rl - (S @ self.off[:, :, None])[:, :, 0]
        free = torch.ones(self.n, dtype=torch.bool, device="cuda")
        free[self.dof[self.dirichlet]] = False
        if pinned is not None:
            free[self.dof[pinned, 0]] = False      # one pressure of a periodic box is arbitrary: 0
        self.free = free
        used = torch.zeros(self.n, dtype=torch.bool, device="cuda")
        used[self.dof.reshape(-1)] = True
        self.b = self.gather(loc)
        i = self.dof[:, :, None].expand(nc, 6, 6).reshape(-1)
        j = self.dof[:, None, :].expand(nc, 6, 6).reshape(-1)
        v = S.reshape(-1)
        keep = (free[i] & free[j])
        i, j, v = i[keep], j[keep], v[keep]
        rest = torch.nonzero(~(free & used)).view(-1)
        i, j, v = torch.cat([i, rest]), torch.cat([j, rest]), torch.cat([v, torch.ones_like(rest, dtype=F64)])
        A = torch.sparse_coo_tensor(torch.stack([i, j]), v, (self.n, self.n)).coalesce()
        ii, vv = A.indices(), A.values()
        on = ii[0] == ii[1]
        self.d = torch.ones(self.n, dtype=F64, device="cuda")
        self.d[ii[0][on]] = vv[on]
        self.A = A.to_sparse_csr()

    def gather(self, loc):
        b = torch.zeros(self.n, dtype=F64, device="cuda").index_add_(0, self.dof.reshape(-1), loc.reshape(-1))
        return torch.where(self.free, b, torch.zeros_like(b))

    def solve(self, b=None):
        b = self.b if b is None else b
        return _pcg(self.A, self.d[:, None], b[:, None], None, 1)[:, 0]

    def half(self, x):
        return torch.where(self.dirichlet, torch.zeros_like(self.off), x[self.dof]) + self.off

    def recover(self, x):
        pi = self.half(x)
        p = (self.g + (self.F * pi).sum(1)) / self.L
        v = (self.B @ (p[:, None] - pi)[:, :, None])[:, :, 0] + self.gf
        return p, v.reshape(-1)

    def average(self, v):
        t = self.twin.reshape(-1)
        return torch.where(t >= 0, 0.5 * (v - v[t.clamp(min=0)]), v)

    def face_pressure(self, x):
        out = torch.zeros(self.n, dtype=F64, device="cuda")
        out[self.dof.reshape(-1)] = self.half(x).reshape(-1)
        return out


def _exact_adjoint(g, d):
    M = _Mimetic(g, d["K"], _t(d["sat"]), _t(d["mobdens"]), d["grav"], d["src"], d["bct"], d["bcv"])
    w, target, u = _t(d["w"]), _t(d["target"]), _t(d["u"]).view(-1, 6)
    pi0 = M.half(M.solve())

    def cellwise(theta, pi):
        """J of the cells and S pi - b, with B scaled by exp(theta)."""
        B = M.B * torch.exp(theta)[:, None, None]
        F = B.sum(1)
        L = F.sum(1)
        p = (M.g + (F * pi).sum(1)) / L
        v = (B @ (p[:, None] - pi)[:, :, None])[:, :, 0]
        return (w * (p - target) ** 2).sum() + (u * v).sum(), -v

    theta = torch.zeros(g.num_cells, dtype=F64, device="cuda")
    pi = pi0.clone().requires_grad_(True)
    J, _ = cellwise(theta, pi)
    y, = torch.autograd.grad(J, pi)
    mu = M.solve(-M.gather(y))
    mu = torch.where(M.dirichlet, torch.zeros_like(pi0), mu[M.dof])
    theta.requires_grad_(True)
    J, res = cellwise(theta, pi0)
    grad, = torch.autograd.grad(J + (mu * res).sum(), theta)
    return dict(J=float(J.detach()), gradient=grad)


def _exact_upscale(u, K):
    nc, ng = u.num_cells, len(u.grids)
    side = torch.as_tensor(u.side, device="cuda").long()
    bid = torch.as_tensor(u.bid, device="cuda").long()
    partner = torch.as_tensor(u.partner, device="cuda").long()
    of_bid = torch.zeros(int(bid.max()) + 1, dtype=torch.long, device="cuda")
    hfs = torch.nonzero(bid > 0).view(-1)
    of_bid[bid[hfs]] = hfs
    low = torch.nonzero((side > 0) & (side % 2 == 1)).view(-1)
    high = of_bid[partner[low]]

    def shared(dof):                     # a face of a low side takes the unknown of its partner
        dof = dof.reshape(-1).clone()
        dof[low] = dof[high]
        return dof.view(nc, 6)

    first = torch.as_tensor(u.cellpos[:-1].astype(np.int64), device="cuda")
    one, zero = torch.ones(nc, dtype=F64, device="cuda"), torch.zeros(nc, dtype=F64, device="cuda")
    bct, none = np.full(u.num_half_faces, lib.BC_PERIODIC, np.int32), np.zeros(u.num_half_faces)
    systems = []
    for a in range(3):
        off = torch.zeros(u.num_half_faces, dtype=F64, device="cuda")
        off[side == 2 * a + 1] = 1.0
        systems.append(_Mimetic(u, K, one, zero, (0.0, 0.0, 0.0), zero.cpu().numpy(), bct, none, shared, off.view(nc, 6),
                                first))
    pos = torch.as_tensor(np.repeat(np.arange(ng), np.diff(u.cellpos)), device="cuda")
    M = systems[0]
    blk = torch.zeros(M.n, dtype=torch.long, device="cuda")
    blk[M.dof.reshape(-1)] = pos[:, None].expand(nc, 6).reshape(-1)
    x = _pcg(M.A, M.d[:, None], torch.stack([s.b for s in systems], 1), blk, ng)
    K = torch.zeros(ng, 3, 3, dtype=F64, device="cuda")
    of = pos[:, None].expand(nc, 6).reshape(-1)
    area, fc = _t(u.area), _t(u.fcentroid)
    for a, s in enumerate(systems):
        _, v = s.recover(x[:, a])
        for i in range(3):
            at = side == 2 * i + 2
            Q = torch.zeros(ng, dtype=F64, device="cuda").index_add_(0, of[at], v[at])
            Ai = torch.zeros(ng, dtype=F64, device="cuda").index_add_(0, of[at], area[at])
            hi = torch.zeros(ng, dtype=F64, device="cuda").scatter_reduce_(0, of, fc[:, a], "amax", include_self=False)
            lo = torch.zeros(ng, dtype=F64, device="cuda").scatter_reduce_(0, of, fc[:, a], "amin", include_self=False)
            K[:, i, a] = (hi - lo) * Q / Ai
    return K


def _interp(x, y, v):
    """Piecewise linear, end values outside."""
    x, y = _t(x), _t(y)
    k = torch.searchsorted(x, v.contiguous(), right=True).clamp(1, len(x) - 1)
    w = ((v - x[k - 1]) / (x[k] - x[k - 1])).clamp(0.0, 1.0)
    return (1 - w) * y[k - 1] + w * y[k]


class _Rock:
    """Phase mobilities and capillary pressure per cell: the tables, or kr = s^2, (1 - s)^2."""

    def __init__(self, d):
        self.tables = d["tables"]
        if self.tables is not None:
            self.rock = _t(d["cell_rock"], torch.long)
            K = _t(d["K"])
            self.skp = torch.sqrt((K[:, 0] + K[:, 4] + K[:, 8]) / (3 * _t(d["poro"])))
            self.sct = d["sct"]

    def pick(self, cells, f):
        out = None
        for r, t in enumerate(self.tables):
            v = f(t)
            out = v if out is None else torch.where(self.rock[cells] == r, v, out)
        return out

    def mob(self, phase, cells, s):
        if self.tables is None:
            return s * s / MU[0] if phase == 0 else (1 - s) ** 2 / MU[1]
        return self.pick(cells, lambda t: _interp(t[:, 0], t[:, 1 + phase], s)) / MU[phase]

    def pc(self, s):
        every = torch.arange(len(s), device="cuda")
        return self.pick(every, lambda t: _interp(t[:, 0], t[:, 3], s)) * self.sct / self.skp

    def sat_of_pc(self, pc):
        every = torch.arange(len(pc), device="cuda")
        v = pc * self.skp / self.sct
        return self.pick(every, lambda t: _interp(t[::-1, 3].copy(), t[::-1, 0].copy(), v))


class _Upstream:
    """The upstream residual of EulerUpstreamResidual over faces; Dirichlet saturations on the boundary."""

    def __init__(self, g, d, gravity, capillary):
        nc = g.num_cells
        self.nc, self.gravity, self.capillary, self.rock = nc, gravity, capillary, _Rock(d)
        nb = torch.as_tensor(g.neighbour, device="cuda").long()
        cell = torch.arange(nc, device="cuda").repeat_interleave(6)
        f = torch.nonzero((nb < 0) | (nb > cell)).view(-1)
        self.bnd = nb[f] < 0
        self.c0, self.c1 = cell[f], torch.where(self.bnd, cell[f], nb[f])
        self.n = _t(g.fnormal)[f]
        self.area = _t(g.area)[f]
        self.q = _t(d["flux"])[f]
        self.sv = _t(d["sat_value"])[f]
        K = _t(d["K"]).view(nc, 3, 3)
        self.Kav = 0.5 * (K[self.c0] + K[self.c1]) if gravity or capillary else None
        if gravity:
            self.gi = (self.Kav @ torch.tensor(d["grav"], dtype=F64, device="cuda")) * (RHO[0] - RHO[1])
        if capillary:
            cc, fc = _t(g.ccentroid), _t(g.fcentroid)
            lf = f % 6
            fn = torch.where(self.bnd, f, nb[f] * 6 + (lf ^ 1))
            a, b = cc[self.c0] - fc[f], cc[self.c1] - fc[fn]
            self.dist = a.norm(dim=1) + b.norm(dim=1)
            r = b + fc[f] - cc[self.c0]
            self.dir = r / r.norm(dim=1, keepdim=True).clamp(min=1e-300)
            self.Kdir = (self.n * (self.Kav @ self.dir[:, :, None])[:, :, 0]).sum(1)

    def __call__(self, s):
        rk, c0, c1, q, n = self.rock, self.c0, self.c1, self.q, self.n
        s0, s1 = s[c0], torch.where(self.bnd, self.sv, s[c1])
        up = q >= 0

        def at(phase, first):
            return rk.mob(phase, torch.where(first, c0, c1), torch.where(first, s0, s1))

        if self.gravity:
            ng = (n * self.gi).sum(1)
            triv0 = self.area * ng >= 0                       # phase 0 is the trivial one
            m_triv = torch.where(triv0, at(0, up), at(1, up))
            shift = torch.where(triv0, -self.area * m_triv * ng, self.area * m_triv * ng)
            other = q + shift >= 0
            m0 = torch.where(triv0, m_triv, at(0, other))
            m1 = torch.where(triv0, at(1, other), m_triv)
        else:
            m0, m1 = at(0, up), at(1, up)
        dS = m0 / (m0 + m1) * q * (n * n).sum(1)
        inside = (~self.bnd).to(F64)
        if self.gravity:
            dS = dS + inside * self.area * m0 * m1 / (m0 + m1) * ng
        if self.capillary:
            a = 0.5 * (s0 + s1)
            a0 = 0.5 * (rk.mob(0, c0, a) + rk.mob(0, c1, a))
            a1 = 0.5 * (rk.mob(1, c0, a) + rk.mob(1, c1, a))
            pc = rk.pc(s)
            dS = dS + inside * self.area * a0 * a1 / (a0 + a1) * (pc[c1] - pc[c0]) / self.dist * self.Kdir
        return torch.zeros(self.nc, dtype=F64, device="cuda").index_add_(0, c0, -dS).index_add_(0, c1, inside * dS)


def _cfl_step(case, g, d):
    """The time step that EulerUpstream's CFL bounds allow (Courant number 0.5)."""
    nc = g.num_cells
    s = np.arange(257) / 256.0
    K, poro = d["K"], d["poro"]
    pv = g.volume * poro
    rocks = [None] if d["tables"] is None else d["tables"]
    fv, fg, fc = 1e100, 1e100, 0.0
    for r, t in enumerate(rocks):
        if t is None:
            l1, l2 = s * s / MU[0], (1 - s) ** 2 / MU[1]
        else:
            l1, l2 = np.interp(s, t[:, 0], t[:, 1]) / MU[0], np.interp(s, t[:, 0], t[:, 2]) / MU[1]
        f, gg = l1 / (l1 + l2), l1 * l2 / (l1 + l2)
        fv = min(fv, 1.0 / (np.abs(np.diff(f)).max() * 256))
        fg = min(fg, 1.0 / (np.abs(np.diff(gg)).max() * 256))
        if t is not None:
            mine = d["cell_rock"] == r
            kmin = ((K[mine, 0] + K[mine, 4] + K[mine, 8]) / 3).min()
            slope = np.abs(np.diff(t[:, 3]) / np.diff(t[:, 0])).max()
            fc = max(fc, gg.max() * slope * d["sct"] / math.sqrt(kmin / poro[mine].max()))
    q = d["flux"].reshape(nc, 6)
    through = np.maximum(np.maximum(q, 0).sum(1), np.maximum(-q, 0).sum(1))
    dt = (fv * pv / through).min()
    if case.get("rock"):
        nb = g.neighbour.reshape(nc, 6)
        k = K[:, [0, 4, 8]]                                   # diagonal, so face by face one axis
        ax = np.array([0, 0, 1, 1, 2, 2])
        kf = np.where(nb < 0, k[:, ax], 0.5 * (k[:, ax] + k[np.maximum(nb, 0)][:, np.arange(6), ax]))
        n = g.fnormal.reshape(nc, 6, 3)[:, np.arange(6), ax]
        gf = g.area.reshape(nc, 6) * n * kf * np.asarray(d["grav"])[ax] * (RHO[0] - RHO[1])
        out = np.maximum(gf, 0).sum(1)
        dt = min(dt, (fg * pv / np.maximum(out, 1e-300)).min())
        x = (g.fcentroid.reshape(nc, 6, 3) - g.ccentroid[:, None])[:, np.arange(6), ax]
        dt = min(dt, (x * x / kf).min() / fc)
    return 0.5 * dt


def _exact_transport(case, g, d):
    R = _Upstream(g, d, case["rock"], case["rock"])
    step = _cfl_step(case, g, d)
    n = max(1, math.ceil(d["time"] / step))
    s, ipv = _t(d["sat"]), d["time"] / n / (_t(d["poro"]) * _t(g.volume))
    for _ in range(n):
        s = s + ipv * R(s)
        if bool(((s > 1.001) | (s < -0.001)).any()):
            return None                                       # the step-doubling retry
    return s


def _exact_capillary(case, g, d):
    rk = _Rock(d)
    s = _t(d["sat"])
    every = torch.arange(len(s), device="cuda")
    m1, m2 = rk.mob(0, every, s), rk.mob(1, every, s)
    cm = (m1 * m2 / (m1 + m2)).clamp(min=1e-10)
    src = -_Upstream(g, d, False, False)(s)
    M = _Mimetic(g, d["K"], cm, cm, (0.0, 0.0, 0.0), src.cpu().numpy(), d["bct"], d["bcv"])
    pc, _ = M.recover(M.solve())
    pv = _t(d["poro"]) * _t(g.volume)

    def miss(shift):
        return float((pv * (rk.sat_of_pc(pc + shift) - s)).sum())

    step = float(pc.max() - pc.min())
    f0, lo, hi = miss(0.0), None, None
    x = step
    for _ in range(100):
        if f0 * miss(x) <= 0:
            lo, hi = min(0.0, x), max(0.0, x)
            break
        x *= -2.0
    flo = miss(lo)
    for _ in range(200):
        mid = 0.5 * (lo + hi)
        if mid in (lo, hi):
            break
        f = miss(mid)
        if f * flo > 0:
            lo, flo = mid, f
        else:
            hi = mid
    return rk.sat_of_pc(pc + 0.5 * (lo + hi))
