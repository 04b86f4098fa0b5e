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
