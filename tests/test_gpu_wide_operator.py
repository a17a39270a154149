"""The FP64 CG pass with three threads a column (small elements and small
meshes): element counts on both sides of the rule's lines, box and general
metric, against the oracle's CG: x to 1e-12 after 8 iterations, the tolerance
of the other CG tests (the smallest box has 8 unknowns: its residual is zero by
then, to rounding)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nb():
    import nekbone_gb300 as m
    return m


@pytest.mark.parametrize("dims", [(1, 1, 1, 4), (2, 2, 2, 5), (3, 2, 2, 6), (2, 2, 2, 7),
                                  (10, 10, 6, 8), (11, 11, 5, 8), (3, 2, 2, 9), (10, 10, 10, 10),
                                  (11, 10, 10, 10), (4, 4, 19, 11), (5, 4, 19, 12),
                                  (4, 4, 9, 14), (9, 17, 1, 16), (2, 4, 19, 16)])
@pytest.mark.parametrize("metric", ["box", "general"])
def test_cg_matches_oracle(nb, dims, metric):
    mesh = nb.Nekbone(*dims, mask_mode=1)
    ctx = O.Ctx(*dims, mask_mode=1, nthreads=8)
    c, g = mesh.set_multiplicity(), mesh.setup_g()
    if metric == "general":
        # symmetric positive definite: the box's weights times a fixed matrix
        # that varies from element to element
        v = g.reshape(mesh.nelt, -1, 6)
        s = np.random.default_rng(1).uniform(0.8, 1.2, (mesh.nelt, 1))
        w = v[..., 0].copy()
        for q, f in enumerate((1.0, 0.1, -0.05, 1.1, 0.15, 0.9)):
            v[..., q] = w * f * s
    f = mesh.set_f(c)
    x = mesh.cg(f, g, c, 8)[0]
    o = ctx.cg(f, g, c, 8)
    assert np.abs(x - o["x"]).max() <= 1e-12 * np.abs(o["x"]).max()
