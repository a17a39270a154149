"""The FP64 operator in fixed point (order 2) at every lx1, odd ones too,
against the oracle's operator in the reference's summation order.

Tolerance: each of the six contraction stages and the metric step is off by
a few units of 2^-55 of the element's largest value, and the FP64 evaluation
it is compared with by lx1 roundings of 2^-53 of its largest term; with
|D|'s row sums up to ~lx1^2/2 twice over, 1e-13 of max|w| leaves a factor of
ten above both."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nb():
    import nekbone_gb300 as m
    return m


@pytest.mark.parametrize("lx", range(2, 17))
@pytest.mark.parametrize("field", ["random", "largest_gradient"])
def test_every_order_matches_oracle(nb, lx, field):
    mesh = nb.Nekbone(2, 3, 2, lx, mask_mode=1)
    ctx = O.Ctx(2, 3, 2, lx, mask_mode=1)
    rng = np.random.default_rng(lx)
    g = rng.standard_normal(6 * mesh.n)
    if field == "random":
        u = rng.standard_normal(mesh.n)
    else:
        # every line of one direction in turn has the signs of D's first row:
        # the largest derivative that values of this size can have
        sgn = np.sign(mesh.dxm1.reshape(lx, lx).T[0]) + 0.0
        sgn[sgn == 0] = 1.0
        e = np.ones((mesh.nelt, lx, lx, lx))
        for q in range(mesh.nelt):
            e[q] *= sgn.reshape([(1, 1, lx), (1, lx, 1), (lx, 1, 1)][q % 3])
        u = e.reshape(-1)
    nb.Nekbone.set_order(2)
    w, wo = mesh.ax(u, g), ctx.ax(u, g)
    assert np.abs(w - wo).max() <= 1e-13 * np.abs(wo).max()
    assert not mesh.ax(np.zeros(mesh.n), g).any()


@pytest.mark.parametrize("lx", [3, 9, 15])
@pytest.mark.parametrize("mask_mode", [0, 1])
def test_odd_order_cg_matches_oracle(nb, lx, mask_mode):
    mesh = nb.Nekbone(4, 3, 3, lx, mask_mode=mask_mode)
    ctx = O.Ctx(4, 3, 3, lx, mask_mode=mask_mode)
    c, g = mesh.set_multiplicity(), mesh.setup_g()
    f = mesh.set_f(c)
    x = mesh.cg(f, g, c, 15)[0]
    xo = ctx.cg(f, g, c, 15)["x"]
    assert np.abs(x - xo).max() <= 1e-12 * np.abs(xo).max()
