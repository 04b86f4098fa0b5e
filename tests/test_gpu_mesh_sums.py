"""How far the mesh pass's sums are from 64 bits: cells that mostly lie outside
the mesh, whose signed terms cancel, against the oracle.

A cell's points are rounded to u = 2^-24 of its radius, about a cell's size.
So the barycentre of a part is off by about u of that size, and the volume of a
part with the share f, which is f^(1/3) of the size across, by about 3 u /
f^(1/3) of itself.  Bounds on the root mean square: twice u (a radius is up to
twice the size), and 3 u / f^(1/3)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


def slab_problem(meshgen, n):
    P = meshgen.cube_problem(5, 10, seed=2, jitter=0.15)
    tets = P.tets[P.verts[P.tets].mean(1)[:, 2] < 430.0]
    return P.verts, tets, np.random.default_rng(12).uniform(5.0, 995.0, (n, 3)).astype(np.float32)


def moments(pkg, verts, tets, sites, **kw):
    with pkg.Engine(verts, tets, sites, **kw) as e:
        e.iterate(1, update=False)
        vol, mom = e.moments()
        _, ids = e.sites()
    v, m = np.empty_like(vol), np.empty_like(mom)
    v[ids], m[ids] = vol, mom
    return v, m


def check(vol, mom, want, wmom, n):
    cell = 1e9 / n
    share = want / cell
    for lo, hi in ((0.01, 0.1), (0.1, 0.5), (0.5, 9.0)):
        w = (share > lo) & (share <= hi)
        assert w.sum() > 25
        e = (vol[w] / want[w] - 1) * np.cbrt(share[w])
        b = np.linalg.norm(mom[w] / vol[w, None] - wmom[w] / want[w, None], axis=1) / np.cbrt(cell)
        assert np.sqrt((e * e).mean()) < 3 * U, (lo, "volume")
        assert np.sqrt((b * b).mean()) < 2 * U, (lo, "barycentre")


@pytest.mark.parametrize("site_k", [16, 96])
def test_exact_form(pkg, meshgen, oracle, site_k):
    pkg.build()
    n = 4000
    verts, tets, sites = slab_problem(meshgen, n)
    vol, mom = moments(pkg, verts, tets, sites, site_k=site_k, tet_k=20, exact=True)
    q = np.flatnonzero(vol > 0)
    r = oracle.complete_cells(sites, q, verts, tets, k0=96)
    assert r["complete"].all()
    check(vol[q], mom[q], r["vol"], r["mom"], n)


@pytest.mark.parametrize("method", ["cell_tet", "site_major"])
@pytest.mark.parametrize("tet_k", [7, 40])
def test_reference_forms(pkg, meshgen, oracle, tet_k, method):
    pkg.build()
    n = 4000
    verts, tets, sites = slab_problem(meshgen, n)
    vol, mom = moments(pkg, verts, tets, sites, site_k=96, tet_k=tet_k, method=method)
    nbr = oracle.knn_grid(sites, None, 96)
    cand = oracle.knn_grid(sites, oracle.tet_centroids(verts, tets), tet_k, exclude_self=False)
    r = oracle.cell_tet(sites, nbr, verts, tets, cand)
    check(vol, mom, r["vol"], r["mom"], n)
