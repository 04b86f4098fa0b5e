"""Grid order by (cell, id) on both sides of the line between the counting
placement (up to 65,536 sites) and the radix passes, with tiles of 128 keys
and more, spread sites and clusters that put thousands in one cell: the order
and the neighbours against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def order_of(p, dim):
    c = np.floor(p * np.float32(dim) / np.float32(1000.0)).astype(np.int64).clip(0, dim - 1)
    return np.lexsort((np.arange(len(p)), c[:, 0] + dim * (c[:, 1] + dim * c[:, 2])))


@pytest.mark.parametrize("kind", ["uniform", "one cell", "outside"])
@pytest.mark.parametrize("n", [5, 129, 4097, 65536, 65537, 311_297])
def test_order_and_neighbours(pkg, n, kind):
    pkg.build()
    rng = np.random.default_rng(n)
    p = rng.uniform(0.0, 1000.0, (n, 3))
    if kind == "one cell":
        m = min(n - n // 4, 6000)
        p[:m] = 500.0 + rng.uniform(0.0, 0.5, (m, 3))
    if kind == "outside":
        p[::7] = rng.uniform(-80.0, 1080.0, (len(p[::7]), 3))
    p = p.astype(np.float32)
    k = min(17, n - 1)
    kn = pkg.KnProblem(p, k=k)
    kn.solve()
    perm, rows, dim = kn.permutation().astype(np.int64), kn.knearests().astype(np.int64), kn.dim
    kn.close()
    assert np.array_equal(perm, order_of(p, dim))
    # the neighbours of some, by (squared distance, id) as the search rounds it
    for q in rng.choice(n, min(n, 40), replace=False):
        d = p - p[perm[q]]
        d2 = (d[:, 0].astype(np.float64) ** 2 + d[:, 1].astype(np.float64) ** 2 + d[:, 2].astype(np.float64) ** 2)
        d2[perm[q]] = np.inf
        got = np.sort(d2[perm[rows[q]]])
        assert np.allclose(got, np.sort(d2)[:k], rtol=1e-6, atol=0.0)
