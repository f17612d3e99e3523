"""The AMG setup as cluster launches and as a launch per step make the same hierarchy: every level's matrix, row
lengths, diagonal, aggregates and member lists agree bit for bit, whether the device holds clusters of 16 blocks,
of 8 or none (the setup then takes the launches instead of failing).  Matrices with few and many entries a row (one
to several lanes), equal strengths, couplings of both signs (rounds that stall), isolated rows, and rows at the
edges of blocks and of the largest cluster level.

The coarsest inverse comes from two algorithms (Gauss-Jordan by the cluster, Cholesky otherwise).  These
matrices are diagonally dominant by a twentieth of their couplings, so the condition of a coarse level of n <= 160
rows is below 2e4, and each inverse is within n * 2e4 * 2^-53 of the exact one."""
import numpy as np
import pytest

sp = pytest.importorskip("scipy.sparse")

pytestmark = pytest.mark.gpu


def stencil(dims, full, kind, seed):
    nx, ny, nz = dims
    n = nx * ny * nz
    rng = np.random.default_rng(seed)
    idx = np.arange(n).reshape(nz, ny, nx)
    offs = [(0, 0, 1), (0, 1, 0), (1, 0, 0)]
    if full:
        offs = [(a, b, c) for a in (0, 1) for b in (-1, 0, 1) for c in (-1, 0, 1) if (a, b, c) > (0, 0, 0)]
    i, j = [], []
    for a, b, c in offs:
        lo = idx[: nz - a, max(0, -b): ny - max(0, b), max(0, -c): nx - max(0, c)]
        hi = idx[a:, max(0, b): ny - max(0, -b), max(0, c): nx - max(0, -c)]
        i.append(lo.ravel())
        j.append(hi.ravel())
    i, j = np.concatenate(i), np.concatenate(j)
    w = -np.ones(len(i)) if kind == "equal" else -rng.uniform(0.1, 1.0, len(i))
    if kind == "signs":
        w *= np.where(rng.random(len(i)) < 0.6, -1.0, 1.0)
    if kind == "isolated":
        off = rng.random(n) < 0.1
        keep = ~(off[i] | off[j])
        i, j, w = i[keep], j[keep], w[keep]
    d = np.zeros(n)
    np.add.at(d, i, np.abs(w))
    np.add.at(d, j, np.abs(w))
    d = 1.05 * d + (d == 0)
    A = sp.coo_matrix((np.concatenate([w, w, d]), (np.concatenate([i, j, np.arange(n)]),
                                                   np.concatenate([j, i, np.arange(n)])))).tocsr()
    A.sort_indices()
    return A


CASES = [((5, 4, 3), False, "random"), ((32, 32, 1), False, "equal"), ((41, 25, 1), False, "random"),
         ((17, 13, 11), True, "random"), ((23, 19, 21), False, "signs"), ((31, 30, 29), False, "isolated"),
         ((25, 24, 23), True, "signs"), ((48, 32, 32), False, "random"), ((40, 33, 38), False, "equal")]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("dims,full,kind", CASES)
def test_cluster_and_launch_paths_agree(pkg, gpulib, dims, full, kind, precision):
    A = stencil(dims, full, kind, 3)
    for round3 in (0, 30000):
        rows, hashes, inv = pkg.selftest_amg_setup(A, precision, 16, round3)
        for clusters in (8, 0):
            rows2, hashes2, inv2 = pkg.selftest_amg_setup(A, precision, clusters, round3)
            assert rows2 == rows
            assert hashes2 == hashes
            n = len(inv)
            assert np.abs(inv2 - inv).max() <= 2 * n * 2e4 * 2.0 ** -53 * np.abs(inv).max()
