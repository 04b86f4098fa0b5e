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
