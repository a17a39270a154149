"""The separable metric's operator, reached through solves (a plain apply takes
the general form): w of one CG iteration is one apply of it."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

LD = np.longdouble


@pytest.fixture(scope="module")
def nb():
    import nekbone_gb300 as m
    return m


# meshes on both sides of the line between three threads a column and one
@pytest.mark.parametrize("dims", [(2, 2, 2, 4), (3, 2, 2, 8), (9, 9, 8, 8), (2, 3, 2, 12),
                                  (7, 7, 7, 12), (6, 6, 5, 14), (2, 2, 3, 16), (6, 6, 5, 16)])
@pytest.mark.parametrize("field", ["random", "smooth"])
def test_apply_is_as_exact_as_fp64_sums(nb, dims, field):
    """Against extended precision, beside the oracle's FP64 sums on the same
    input.  Both round w itself and a few units of its largest terms: 1.0 to
    1.5 times the oracle's error (2-norm), so twice bounds it.  With D or the
    weights made symmetric it is 4 to 30 times from lx1 = 8 on."""
    *ex, lx = dims
    mesh, ctx = nb.Nekbone(*dims, mask_mode=1), O.Ctx(*dims, mask_mode=1, nthreads=8)
    c, g = mesh.set_multiplicity(), mesh.setup_g()
    ids = mesh.glo_num - mesh.glo_num.min()
    mask = np.ones(mesh.n)
    ctx.maskit(mask)
    u = (np.random.default_rng(lx).standard_normal(ids.max() + 1) if field == "random"
         else np.cos(0.01 / lx * np.arange(ids.max() + 1)))[ids] * mask
    w, wo = mesh.cg(u, g, c, 1)[2], ctx.cg(u.copy(), g, c, 1)["w"]
    # the 2 x 2 x 2 elements at the corner, at the points that only they have
    D = np.asarray(mesh.dxm1).reshape(lx, lx).astype(LD)
    D = D if abs(D.sum(1)).max() < abs(D.sum(0)).max() else D.T
    el = [i + ex[0] * (j + ex[1] * k) for k in (0, 1) for j in (0, 1) for i in (0, 1)]
    sub = (np.asarray(el)[:, None] * lx ** 3 + np.arange(lx ** 3)).ravel()
    sh = (8, lx, lx, lx)

    def along(M, v, axis):
        return np.moveaxis(np.tensordot(v, M, axes=(axis, 1)), -1, axis)

    G, U = g.reshape(-1, 6)[sub].astype(LD).reshape(sh + (6,)), u[sub].astype(LD).reshape(sh)
    W = sum(along(D.T, G[..., m] * along(D, U, a), a) for m, a in ((0, 3), (3, 2), (5, 1)))
    total, copies = np.zeros(ids.max() + 1, LD), np.zeros(ids.max() + 1)
    np.add.at(total, ids[sub], W.ravel())
    np.add.at(copies, ids[sub], 1.0)
    W = (total[ids[sub]] + LD(0.1) * U.ravel()) * mask[sub]
    own = copies[ids[sub]] == np.rint(1 / c[sub])

    def err(v):
        return float(np.sqrt(((v[sub] - W)[own] ** 2).sum() / (W[own] ** 2).sum()))

    assert err(wo) < 1e-14          # the same operator
    assert err(w) <= 2 * err(wo), (err(w), err(wo))
