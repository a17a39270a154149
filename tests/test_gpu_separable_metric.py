"""The FP64 operator on a separable metric (a box of equal cubes: one
contraction a direction with K = D^T b D, nb_ax_fx.cuh) against the oracle's
operator and CG, and the metrics that are nearly of that form, which take the
general operator: every call gives the oracle's result whichever form runs.

Tolerance 1e-13 of max|w|, as for the general fixed-point operator
(test_gpu_fixed_point.py): K's entries are up to lx1^2/4 times larger against
the result than D's, its tables and values hold two bits more, and the 64-bit
sums are rounded once instead of three times."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

DIMS = (3, 2, 2)


@pytest.fixture(scope="module")
def nb():
    import nekbone_gb300 as m
    return m


def metrics(mesh, kind):
    """setup_g's metric, or one changed so that it is not of the form."""
    g = mesh.setup_g()
    v = g.reshape(mesh.nelt, -1, 6)
    if kind == "scaled":
        v *= 0.37
    elif kind == "one_value":
        v[-1, -1, 0] *= 1 + 1e-9
    elif kind == "not_cubic":
        v[..., 3] *= 2.0
    elif kind == "off_diagonal":
        v[0, 5, 1] = 1e-3 * v[0, 5, 0]
    elif kind == "not_a_product":
        v[:, 7, :] *= 1.5
    elif kind == "negative":
        v *= -1.0
    return g


@pytest.mark.parametrize("lx", [2, 4, 6, 8, 10, 12, 14, 16])
@pytest.mark.parametrize("kind", ["box", "scaled", "one_value", "not_cubic", "off_diagonal",
                                  "not_a_product", "negative"])
def test_ax_matches_oracle(nb, lx, kind):
    mesh = nb.Nekbone(*DIMS, lx, mask_mode=1)
    ctx = O.Ctx(*DIMS, lx, mask_mode=1)
    g = metrics(mesh, kind)
    rng = np.random.default_rng(lx)
    smooth = np.cos(0.3 * np.arange(mesh.glo_num.max() + 1))[mesh.glo_num]
    for u in (rng.uniform(-1, 1, mesh.n), smooth, np.zeros(mesh.n)):
        w, wo = mesh.ax(u, g), ctx.ax(u, g)
        assert np.abs(w - wo).max() <= 1e-13 * np.abs(wo).max()


@pytest.mark.parametrize("lx", [4, 10, 16])
@pytest.mark.parametrize("mask_mode", [0, 1])
@pytest.mark.parametrize("kind", ["box", "one_value"])
def test_cg_matches_oracle(nb, lx, mask_mode, kind):
    mesh = nb.Nekbone(*DIMS, lx, mask_mode=mask_mode)
    ctx = O.Ctx(*DIMS, lx, mask_mode=mask_mode)
    g, c = metrics(mesh, kind), mesh.set_multiplicity()
    f = mesh.set_f(c)
    x, r = mesh.cg(f, g, c, 8)[:2]
    o = ctx.cg(f, g, c, 8)
    assert np.abs(x - o["x"]).max() <= 1e-12 * np.abs(o["x"]).max()
    assert np.abs(r - o["r"]).max() <= 1e-12 * np.abs(o["r"]).max()


@pytest.mark.parametrize("metric", ["box", "one_value"])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_values_that_are_not_finite_reach_the_result(nb, metric, bad):
    mesh = nb.Nekbone(*DIMS, 8, mask_mode=1)
    g = metrics(mesh, metric)
    u = np.random.default_rng(0).uniform(-1, 1, mesh.n)
    u[8 ** 3 + 100] = bad
    assert not np.isfinite(mesh.ax(u, g)[8 ** 3:2 * 8 ** 3]).all()
