"""The fixed-point FP64 operator makes the same bits every time: its blocks
renormalise twice from words in shared memory, and a block whose warps read the
first words late must not see the second ones.  Equality, no tolerance: every
sum of the operator and of CG has a fixed order."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# one thread a column (the smallest block, one warp and more) and three
@pytest.mark.parametrize("dims", [(9, 8, 9, 8), (11, 10, 10, 10), (7, 7, 7, 12), (2, 2, 2, 16),
                                  (3, 3, 3, 7), (2, 2, 2, 2)])
def test_repeated_passes_are_bitwise_equal(dims):
    import nekbone_gb300 as nb
    mesh = nb.Nekbone(*dims, mask_mode=1)
    rng = np.random.default_rng(sum(dims))
    # values and metrics that differ by powers of two from point to point, so
    # that the two renormalisations differ from element to element
    u = rng.standard_normal(mesh.n) * 2.0 ** rng.integers(-20, 20, mesh.n)
    g = rng.standard_normal(6 * mesh.n) * 2.0 ** rng.integers(-20, 20, 6 * mesh.n)
    c = mesh.set_multiplicity()
    w = mesh.ax(u, g)
    x = mesh.cg(u, g, c, 2)[:4]
    for _ in range(5):
        assert np.array_equal(mesh.ax(u, g), w)
        for a, b in zip(mesh.cg(u, g, c, 2)[:4], x):
            assert np.array_equal(a, b, equal_nan=True)
