"""The robust option's first filter (pairs of floats) and what it hands to the
exact signs: lattices whose spacing is no dyadic fraction are cospherical up
to the rounding of their positions, so most near-zero tests are decided by the
filter, and every cell must come out whole.  A cell is its lattice box
clipped to the mesh's; positions are rounded to 6e-5 of 1,000, spacings are
at least 70, so a box's side is good to 2e-6 and its volume to 6e-6."""
import numpy as np
import pytest

from conftest import lattice_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["exact", "reference", "pieces"])
@pytest.mark.parametrize("n_side", [7, 12, 14])
def test_lattices_of_rounded_positions(pkg, meshgen, n_side, form):
    pkg.build()
    P, vol, bary = lattice_problem(meshgen, n_side)
    kw = dict(exact=form != "reference", tet_pieces=form == "pieces")
    with pkg.Engine(P.verts, P.tets, P.sites, site_k=96, tet_k=100, robust_predicates=True, **kw) as e:
        e.iterate(1, update=False)
        got, mom = e.moments()
        _, ids = e.sites()
        st = e.stats()
    v, m = np.empty_like(got), np.empty_like(mom)
    v[ids], m[ids] = got, mom
    assert st["boundary_fail"] == 0 and st["tri_overflow"] == 0 and st["needs_exact"] > 0
    assert np.abs(v / vol - 1).max() < 1e-5
    assert np.abs(m / v[:, None] - bary).max() < 1e-5 * 1000
