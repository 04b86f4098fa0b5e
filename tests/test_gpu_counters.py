"""The counters of a pass: every candidate pair is culled or clipped, every
clipped one contributes or is empty, whichever passes its site went through
(half the sites of the slab lie outside the mesh: slivers are given back), and
the misses of the tet-cell method are its pairs'."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def slab(meshgen, n, seed):
    P = meshgen.cube_problem(5, 10, seed=2, jitter=0.15)
    tets = P.tets[P.verts[P.tets].mean(1)[:, 2] < 430.0]
    return P.verts, tets, np.random.default_rng(seed).uniform(5.0, 995.0, (n, 3)).astype(np.float32)


def stats(pkg, v, t, s, **kw):
    with pkg.Engine(v, t, s, **kw) as e:
        e.iterate(1, update=False)
        return e.stats()


@pytest.mark.parametrize("kw", [dict(exact=True, site_k=96), dict(exact=True, site_k=24), dict(tet_k=40, site_k=90),
                                dict(tet_k=40, site_k=90, method="site_major")])
def test_pairs_add_up(pkg, meshgen, kw):
    pkg.build()
    v, t, s = slab(meshgen, 4000, 12)
    st = stats(pkg, v, t, s, **{"tet_k": 20, **kw})
    assert st["boundary_fail"] == st["tri_overflow"] == st["unresolved"] == 0 and st["redo"] > 0
    assert st["candidates"] == st["culled"] + st["clipped"]
    assert st["clipped"] == st["empty"] + st["contrib"] and st["contrib"] > 0


@pytest.mark.parametrize("site_k", [12, 32, 90])
@pytest.mark.parametrize("mesh", ["cube", "slab", "torus"])
def test_misses_of_the_tet_cell_method_are_of_pairs(pkg, meshgen, mesh, site_k):
    """Against the general path (robust), which clips each pair: a pair within
    rounding of the line may differ, or one that only touches."""
    pkg.build()
    n = 3000
    if mesh == "slab":
        v, t, s = slab(meshgen, n, 5)
    else:
        P = meshgen.cube_problem(9, n, seed=3, jitter=0.1) if mesh == "cube" else meshgen.torus_problem(n, grid=24, seed=3)
        v, t, s = P.verts, P.tets, P.sites
    got, want = (stats(pkg, v, t, s, site_k=site_k, tet_k=30, method="site_major", robust_predicates=r)["security_miss"]
                 for r in (False, True))
    assert abs(got - want) <= 0.001 * want + 1, (got, want)
