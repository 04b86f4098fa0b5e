"""Tets of a grid cell in id order, whatever order the scatter left them in:
few sites in many tets (thousands of tets a cell, below and above one warp and
one block) give the same bits in two engines, and the mesh's volume."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["exact", "reference"])
@pytest.mark.parametrize("cells,n", [(2, 3), (4, 5), (17, 3), (20, 64), (33, 700)])
def test_same_bits_and_whole_volume(pkg, meshgen, cells, n, form):
    pkg.build()
    p = meshgen.cube_problem(cells, n, seed=cells, jitter=0.1)
    got = []
    for _ in range(2):
        e = pkg.Engine(p.verts, p.tets, p.sites, site_k=min(64, n - 1), exact=form == "exact")
        e.iterate(1, update=False)
        vol, mom = e.moments()
        got.append((vol.copy(), mom.copy()))
        e.close()
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    # the reference form may miss pairs beyond its candidates; a cell's edge is
    # summed from its lengths in up to 3 x 33 tets, each rounded to 6e-8 of it
    if form == "exact":
        v = p.verts.astype(np.float64)[p.tets]
        whole = np.abs(np.einsum("ij,ij->i", np.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]), v[:, 3] - v[:, 0])).sum() / 6
        assert abs(got[0][0].sum() - whole) < 1e-5 * whole
