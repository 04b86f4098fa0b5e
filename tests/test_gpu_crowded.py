"""Sites crowded into a few cells of the grid, beside spread ones: the order, the
neighbours and the cells around the crowds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def crowds(n, sizes, width, seed=0):
    """n sites in [0,1000]^3, of which sizes[i] in a cube of that width each."""
    rng = np.random.default_rng(seed)
    p = rng.uniform(5.0, 995.0, (n, 3))
    b = 0
    for m in sizes:
        p[b:b + m] = rng.uniform(150.0, 850.0, 3) + rng.uniform(0.0, width, (m, 3))
        b += m
    return p[rng.permutation(n)].astype(np.float32)


@pytest.mark.parametrize("n,sizes", [(700, [257, 256]), (5000, [255, 256, 257, 300, 511, 1025]), (40_000, [20_000, 9_000]),
                                     (65_536, [65_536]), (65_536, [33_000, 300, 31_000]), (65_537, [40_000])])
def test_order_within_crowded_cells(pkg, n, sizes):
    """Cells on both sides of the line between comparing and counting bits,
    several to a block and many blocks to one."""
    pkg.build()
    p = crowds(n, sizes, 0.01, seed=n)
    kn = pkg.KnProblem(p, k=16)
    perm, dim = kn.permutation().astype(np.int64), kn.dim
    kn.close()
    c = np.floor(p * np.float32(dim) / np.float32(1000.0)).astype(np.int64).clip(0, dim - 1)
    assert np.array_equal(perm, np.lexsort((np.arange(n), c[:, 0] + dim * (c[:, 1] + dim * c[:, 2]))))


@pytest.mark.parametrize("k", [16, 32, 64])
@pytest.mark.parametrize("n,sizes,width", [(20_000, [800, 900, 1500], 20.0), (20_000, [10_000], 0.5), (66_000, [30_000, 2000], 25.0)])
def test_neighbours_beside_a_crowd(pkg, n, sizes, width, k):
    """Queries in and around the crowds, on both sides of the line at 27 K sites
    in a block, against brute force."""
    pkg.build()
    p = crowds(n, sizes, width, seed=k)
    kn = pkg.KnProblem(p, k=k)
    kn.solve()
    perm, rows = kn.permutation().astype(np.int64), kn.knearests().astype(np.int64)
    kn.close()
    d = p.astype(np.float64)
    _, block = np.unique(np.floor(d / 60.0), axis=0, return_inverse=True)
    full = np.bincount(block)[block]
    near = np.argsort(-full[perm], kind="stable")
    for q in np.concatenate([near[::len(near) // 60], np.random.default_rng(1).choice(n, 40, replace=False)]):
        d2 = ((d - d[perm[q]]) ** 2).sum(1)
        d2[perm[q]] = np.inf
        assert np.allclose(np.sort(d2[perm[rows[q]]]), np.sort(d2)[:k], rtol=1e-6, atol=0.0)


@pytest.mark.parametrize("n,sizes,width", [(6000, [3000], 2.0), (20_000, [6000, 200], 10.0), (30_000, [12_000], 0.5)])
def test_cells_beside_a_crowd(pkg, meshgen, oracle, n, sizes, width):
    """Cells that the K neighbours left open, completed by the 64-vertex pass or,
    where the search spans the grid, by the 256-vertex pass, against the
    oracle's exact cells.  Points are rounded to u = 2^-24 of a cell's radius R,
    and further along the line that planes at a small angle nearly share: a cell
    at the rim of a crowd is a needle sqrt(V / R) wide, with faces at that angle
    over R, and its points are good to u R over the angle along it, which is
    u R^3 / V of its volume, and of R for its barycentre."""
    pkg.build()
    P = meshgen.cube_problem(8, 10, seed=3)
    sites = crowds(n, sizes, width, seed=n)
    with pkg.Engine(P.verts, P.tets, sites, site_k=64, tet_k=20, exact=True) as e:
        e.iterate(1, update=False)
        vol, mom = e.moments()
        _, ids = e.sites()
        fl, st = e.buffer("site_flags"), e.stats()
    v, m, f = np.empty_like(vol), np.empty_like(mom), np.empty_like(fl)
    v[ids], m[ids], f[ids] = vol, mom, fl
    done = np.flatnonzero((f & pkg.SITE_COMPLETED) != 0)
    large = (f[done] & pkg.SITE_REDO) != 0
    # (a few whose search a float cut ends, as for the 256-vertex pass alone, say so)
    assert st["unresolved"] < 5 and large.any() and (~large).any()
    # the largest of those at 256 vertices, and a sample of the others
    q = np.concatenate([done[large][np.argsort(-v[done[large]])][:60], done[~large][:: max(1, (~large).sum() // 200)]])
    r = oracle.complete_cells(sites, q, P.verts, P.tets, k0=256, kmax=16_384)
    ok = r["complete"] & (r["vol"] > 0)  # (the oracle drops cells beyond its capacity)
    assert ok.sum() > 60
    vol, bary = r["vol"][ok], r["mom"][ok] / r["vol"][ok, None]
    radius = np.cbrt(vol) + 2.0 * np.linalg.norm(bary - sites[q][ok], axis=1)
    bound = np.maximum(1e-5, 2.0 ** -24 * radius ** 3 / vol)
    assert (np.abs(v[q][ok] / vol - 1) / bound).max() < 1.0
    off = np.linalg.norm(m[q][ok] / v[q][ok, None] - bary, axis=1)
    assert (off / (radius * bound)).max() < 1.0
