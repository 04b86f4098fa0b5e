"""The mesh pass of the exact form (the part of a cell inside the mesh from its
edges and the mesh's open triangles) against the general path, which clips a
copy of the cell by every tet (the robust option keeps that path): meshes
whose faces do not all pair up, and cells from a few vertices to tets far
larger or smaller than them.

Both paths place a cell's vertices in single precision from the same planes:
a volume is off by a few 1e-7 of the cell's own radius cubed, here bounded by
1e-5 of the volume plus 1e-6 of the median cell (slivers of cells that mostly
lie outside the mesh carry their whole cell's rounding)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def volumes(pkg, verts, tets, sites, **kw):
    with pkg.Engine(verts, tets, sites, exact=True, **kw) as e:
        e.iterate(1, update=False)
        vol, mom = e.moments()
        _, ids = e.sites()
        st = e.stats()
    v, m = np.empty_like(vol), np.empty_like(mom)
    v[ids], m[ids] = vol, mom
    return v, m, st


def shuffled(P, rng):
    """The same mesh, its vertices numbered in another order."""
    order = rng.permutation(len(P.verts))
    where = np.empty_like(order)
    where[order] = np.arange(len(order))
    return P.verts[order], where[P.tets].astype(np.int32)


def meshes(meshgen):
    rng = np.random.default_rng(3)
    P = meshgen.cube_problem(5, 10, seed=2, jitter=0.15)
    v, t = P.verts, P.tets
    yield "plain", v, t
    yield ("renumbered",) + shuffled(P, rng)
    # a crack: the tets of one half have vertices of their own
    half = v[t].mean(1)[:, 0] < 480.0
    yield "cracked", np.concatenate([v, v]), np.where(half[:, None], t + len(v), t).astype(np.int32)
    # holes: a tenth of the tets missing; and a tenth there twice
    keep = rng.random(len(t)) > 0.1
    yield "holes", v, t[keep]
    yield "doubled", v, np.concatenate([t, t[~keep]])
    # tets that are not positively oriented count for nothing
    bad = t.copy()
    bad[~keep] = bad[~keep][:, [0, 2, 1, 3]]
    yield "inverted", v, bad
    # every other tet: each cube's diagonal planes are open, and edges of the
    # box that bounds an open cell lie in some of them
    yield "every other", v, t[::2]
    # part of the box only: many sites outside the mesh
    yield "slab", v, t[v[t].mean(1)[:, 2] < 350.0]


@pytest.mark.parametrize("n", [130, 2500, 20011])
def test_mesh_pass_matches_clipping_by_every_tet(pkg, meshgen, n):
    pkg.build()
    rng = np.random.default_rng(n)
    sites = rng.uniform(5.0, 995.0, (n, 3)).astype(np.float32)
    for name, v, t in meshes(meshgen):
        got, mom, st = volumes(pkg, v, t, sites, site_k=min(96, n - 1), tet_k=20)
        ref, rmom, _ = volumes(pkg, v, t, sites, site_k=min(96, n - 1), tet_k=20, robust_predicates=True)
        assert st["unresolved"] == 0, name
        scale = np.median(ref[ref > 0])
        err = np.abs(got - ref) - 1e-5 * ref
        assert err.max() < 1e-6 * scale, (name, err.max() / scale, int(err.argmax()))
        # moments about the site: the same, at a cell's reach
        reach = 4.0 * (1e9 / n) ** (1 / 3)
        d = np.abs((mom - got[:, None] * sites) - (rmom - ref[:, None] * sites))
        assert d.max() < reach * (1e-5 * ref.max() + 1e-6 * scale), name


@pytest.mark.parametrize("method", ["cell_tet", "site_major"])
@pytest.mark.parametrize("tet_k", [1, 7, 40])
@pytest.mark.parametrize("n", [130, 2500])
def test_reference_form_sums_over_the_candidate_tets_only(pkg, meshgen, n, tet_k, method):
    """A site's sum is over the tets that count it among their tet_k nearest:
    with few candidates most tets that meet a cell are left out, and their
    faces close the sum.  Terms are of the size of a cell's radius cubed,
    about three cell volumes, each rounded to 1e-7 of it and some dozens of
    them: 2e-6 of the mean cell."""
    pkg.build()
    rng = np.random.default_rng(n + tet_k)
    sites = rng.uniform(5.0, 995.0, (n, 3)).astype(np.float32)
    for name, v, t in meshes(meshgen):
        if name == "inverted" and method == "site_major":
            continue  # tets are positively oriented; that method's general path starts from the tet
        kw = dict(site_k=min(96, n - 1), tet_k=tet_k, method=method)
        out = []
        for robust in (False, True):
            with pkg.Engine(v, t, sites, robust_predicates=robust, **kw) as e:
                e.iterate(1, update=False)
                vol, mom = e.moments()
                _, ids = e.sites()
                assert e.stats()["candidates"] == tet_k * len(t)
            o = np.empty_like(vol)
            o[ids] = vol
            out.append(o)
        err = np.abs(out[0] - out[1]) - 1e-5 * out[1]
        assert err.max() < 2e-6 * 1e9 / n, (name, err.max() * n / 1e9, int(err.argmax()))


def test_sites_whose_cell_has_next_to_nothing_of_the_mesh(pkg, meshgen):
    """Half the sites lie outside the mesh: cells that miss it keep their site
    where it is, and those that reach it move to the same point as in the
    general path.  A cell with the part f of its volume inside has its terms
    rounded to 1e-7 of a volume from a point of that part: where f > 1e-6 of
    the mean cell the barycentre is good to 1e-2 of the cell's size, and where
    f > 1e-2 to 1e-4 of it."""
    pkg.build()
    P = meshgen.cube_problem(5, 10, seed=2, jitter=0.15)
    t = P.tets[P.verts[P.tets].mean(1)[:, 2] < 430.0]
    rng = np.random.default_rng(12)
    n = 4000
    sites = rng.uniform(5.0, 995.0, (n, 3)).astype(np.float32)
    out = []
    for robust in (False, True):
        with pkg.Engine(P.verts, t, sites, site_k=96, tet_k=20, exact=True, robust_predicates=robust) as e:
            e.iterate(1)
            vol, _ = e.moments()
            _, ids = e.sites()
            v = np.empty_like(vol)
            v[ids] = vol
            out.append((v, e.sites_original().astype(np.float64)))
    cell = 1e9 / n
    assert ((out[0][0] > 1e-6 * cell) == (out[1][0] > 1e-6 * cell)).mean() > 0.999
    none = (out[0][0] == 0)
    assert none.sum() > n // 4
    assert np.array_equal(out[0][1][none], sites[none].astype(np.float64))
    d = np.linalg.norm(out[0][1] - out[1][1], axis=1) / cell ** (1 / 3)
    f = np.minimum(out[0][0], out[1][0]) / cell
    assert d[f > 1e-6].max() < 1e-2
    assert d[f > 1e-2].max() < 1e-4
