"""The clip form that runs: `tet_pieces` is an option of the exact form, and the
shape that an engine or a batch reports is the one in use."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_reported_form_is_the_one_in_use(pkg, meshgen):
    pkg.build()
    P, Q = meshgen.cube_problem(6, 800, seed=2), meshgen.cube_problem(1, 3000, seed=8)
    for p, kw, pieces in ((P, {}, 0), (P, dict(robust_predicates=True), 1), (Q, {}, 1)):
        kw = dict(site_k=64, tet_pieces=True, **kw)
        with pkg.Engine(p.verts, p.tets, p.sites, exact=True, tet_k=6, **kw) as e:
            assert e.shape()["tet_pieces"] == pieces
        with pkg.Batch([(p.verts, p.tets, p.sites)], tune_grid=False, **kw) as b:
            assert b.shape()["tet_pieces"] == pieces


@pytest.mark.parametrize("method", ["cell_tet", "site_major"])
def test_the_option_means_nothing_to_the_reference_forms(pkg, meshgen, method):
    pkg.build()
    P = meshgen.cube_problem(1, 3000, seed=8)
    got = []
    for pieces in (False, True):
        with pkg.Engine(P.verts, P.tets, P.sites, site_k=64, tet_k=100, method=method, tet_pieces=pieces) as e:
            e.iterate(1, update=False)
            got.append(e.moments())
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
