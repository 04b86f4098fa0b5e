"""Which faces of a mesh are open: faces are known by their corners' positions
and found by hashing.  Meshes stored tet by tet, each with four vertices of its
own, give the bits of the same mesh with shared vertices numbered in the order
of their first appearance (all their faces would be open if vertices were told
apart by index); problems of a batch share no face; a vertex common to all tets
costs no more than any other."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def shared_and_apart(P):
    """The mesh with its vertices numbered as they first appear, and apart."""
    _, first = np.unique(P.tets.ravel(), return_index=True)
    order = P.tets.ravel()[np.sort(first)]
    where = np.empty(len(P.verts), np.int64)
    where[order] = np.arange(len(order))
    v, t = P.verts[order], where[P.tets].astype(np.int32)
    return (v, t), (np.ascontiguousarray(v[t.ravel()]), np.arange(t.size, dtype=np.int32).reshape(-1, 4))


@pytest.mark.parametrize("form", ["exact", "reference", "site_major"])
@pytest.mark.parametrize("mesh", ["cube", "torus"])
def test_a_mesh_stored_tet_by_tet(pkg, meshgen, mesh, form):
    pkg.build()
    n = 3000
    P = meshgen.cube_problem(7, n, seed=3, jitter=0.1) if mesh == "cube" else meshgen.torus_problem(n, grid=24, seed=3)
    kw = dict(exact=True) if form == "exact" else dict(tet_k=30, method="cell_tet" if form == "reference" else form)
    got = []
    for v, t in shared_and_apart(P):
        with pkg.Engine(v, t, P.sites, site_k=64, **kw) as e:
            e.iterate(1, update=False)
            vol, mom = e.moments()
            # (the cells taken whole are found on the host, by index)
            whole = e.buffer("site_flags") & pkg.SITE_INTERIOR if form == "exact" else np.zeros(n)
            got.append((vol, mom, whole != 0))
    cut = ~got[0][2]
    assert cut.sum() > n // 8 and not got[1][2].any()
    assert np.array_equal(got[0][0][cut], got[1][0][cut]) and np.array_equal(got[0][1][cut], got[1][1][cut])
    assert np.allclose(got[0][0], got[1][0], rtol=1e-5)


def test_problems_of_a_batch_share_no_face(pkg, meshgen):
    pkg.build()
    P = meshgen.cube_problem(5, 900, seed=3, jitter=0.1)
    shared, apart = shared_and_apart(P)
    got = {0: [], 1: []}
    for problems in ([0], [0, 1], [1, 0, 0]):
        with pkg.Batch([(*(shared, apart)[p], P.sites) for p in problems], site_k=64, tune_grid=False) as b:
            b.iterate(1)
            for i, p in enumerate(problems):
                got[p].append(b.result(i)[0])
    for x in got.values():
        assert all(np.array_equal(y, x[0]) for y in x)
    assert np.abs(got[0][0] - got[1][0]).max() < 1e-3


def test_a_fan_around_one_vertex(pkg):
    """A ball of 200,000 tets from its centre, vertex 0."""
    pkg.build()
    a = 316
    th, ph = np.linspace(0.1, np.pi - 0.1, a + 1), np.linspace(0.0, 2.0 * np.pi, a, endpoint=False)
    ring = np.stack([np.sin(th)[:, None] * np.cos(ph), np.sin(th)[:, None] * np.sin(ph),
                     np.cos(th)[:, None] * np.ones(a)], -1).reshape(-1, 3)
    v = (np.concatenate([np.zeros((1, 3)), ring]) * 400.0 + 500.0).astype(np.float32)
    i, j = (x.ravel() for x in np.meshgrid(np.arange(a), np.arange(a), indexing="ij"))
    at = lambda r, c: 1 + r * a + c % a
    t = np.concatenate([np.stack([0 * i, at(i, j), at(i + 1, j), at(i, j + 1)], 1),
                        np.stack([0 * i, at(i, j + 1), at(i + 1, j), at(i + 1, j + 1)], 1)]).astype(np.int32)
    x = v.astype(np.float64)[t]
    det = np.einsum("ij,ij->i", np.cross(x[:, 1] - x[:, 0], x[:, 2] - x[:, 0]), x[:, 3] - x[:, 0])
    t[det < 0] = t[det < 0][:, [0, 2, 1, 3]]
    sites = np.random.default_rng(1).uniform(150.0, 850.0, (400, 3)).astype(np.float32)
    with pkg.Engine(v, t, sites, site_k=64, tet_k=20, exact=True) as e:
        e.iterate(1, update=False)
        vol, _ = e.moments()
    # (each of some thousand tets of a cell rounds its planes to 1e-7)
    assert abs(vol.sum() / (np.abs(det).sum() / 6.0) - 1.0) < 1e-5
