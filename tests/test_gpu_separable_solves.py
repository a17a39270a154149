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


def box_metric(mesh, kind):
    """setup_g's metric, or one changed so that it is of the form no longer
    (or still, "scaled" and "box")."""
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


KINDS = ["box", "scaled", "one_value", "not_cubic", "off_diagonal", "not_a_product", "negative"]


@pytest.mark.parametrize("dims", [(3, 2, 2, 2), (3, 2, 2, 4), (2, 2, 2, 6), (3, 2, 2, 8),
                                  (9, 9, 8, 8), (3, 2, 2, 10), (11, 10, 10, 10), (3, 2, 2, 12),
                                  (7, 7, 7, 12), (3, 2, 2, 14), (6, 6, 5, 14), (3, 2, 2, 16),
                                  (6, 6, 5, 16)])
@pytest.mark.parametrize("kind", KINDS)
def test_every_metric_gives_the_oracles_apply(nb, dims, kind):
    """1e-13 of max|w|, the fixed-point operator's tolerance; a metric taken for
    separable that is not is off by 1e-9 and more."""
    mesh, ctx = nb.Nekbone(*dims, mask_mode=1), O.Ctx(*dims, mask_mode=1, nthreads=8)
    c, g = mesh.set_multiplicity(), box_metric(mesh, kind)
    f = np.random.default_rng(dims[3]).uniform(-1, 1, mesh.glo_num.max() + 1)[mesh.glo_num]
    got, o = mesh.cg(f, g, c, 1), ctx.cg(f, g, c, 1)
    assert np.abs(got[2] - o["w"]).max() <= 1e-13 * np.abs(o["w"]).max()
    assert np.array_equal(got[3], o["p"])


@pytest.mark.parametrize("dims", [(3, 2, 2, 8), (7, 7, 7, 12), (3, 2, 2, 16)])
@pytest.mark.parametrize("skew", [0.0, 1.8e-14, 4e-14])
def test_weights_that_are_not_symmetric(nb, dims, skew):
    """The first weight larger than the last by skew, on both sides of the 2e-14
    up to which the form is taken.  w against the oracle's FP64 sums (2-norm),
    each within 3e-16 of the exact one where the form is taken: 1e-15; 1e-14
    for the general form, whose 55 bits leave up to 5e-15 at lx1 = 16."""
    lx = dims[3]
    mesh, ctx = nb.Nekbone(*dims, mask_mode=1), O.Ctx(*dims, mask_mode=1, nthreads=8)
    c, g = mesh.set_multiplicity(), mesh.setup_g()
    h = lx // 2
    b = g.reshape(mesh.nelt, lx, lx, lx, 6)[0, h, h, :, 0].copy()
    b = 0.5 * (b + b[::-1])
    b[0] *= 1 + skew
    block = np.zeros((lx, lx, lx, 6))
    block[..., 0] = b[:, None, None] * b[:, None] * b
    block[..., 3] = block[..., 5] = block[..., 0]
    g = np.tile(block.ravel(), mesh.nelt)
    f = np.random.default_rng(lx).standard_normal(mesh.glo_num.max() + 1)[mesh.glo_num]
    w, wo = mesh.cg(f, g, c, 1)[2], ctx.cg(f, g, c, 1)["w"]
    err = np.sqrt(((w - wo) ** 2).sum() / (wo ** 2).sum())
    assert err <= (1e-15 if skew < 2e-14 else 1e-14), err


@pytest.mark.parametrize("dims", [(3, 2, 2, 8), (9, 9, 8, 8), (3, 2, 2, 9), (3, 2, 2, 13)])
@pytest.mark.parametrize("kind", ["box", "one_value"])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_values_that_are_not_finite(nb, dims, kind, bad):
    """One value of f: x, r and p of CG are finite where the oracle's are, w
    nowhere that the oracle's is not (a block with such a value is all NaN)."""
    mesh, ctx = nb.Nekbone(*dims, mask_mode=1), O.Ctx(*dims, mask_mode=1, nthreads=8)
    c, g = mesh.set_multiplicity(), box_metric(mesh, kind)
    f = np.random.default_rng(0).uniform(-1, 1, mesh.glo_num.max() + 1)[mesh.glo_num]
    lx = dims[3]
    f[lx ** 3 + 2 + lx * 3 + lx * lx * 2] = bad      # inside the second element
    for niter in (1, 3):
        got, o = mesh.cg(f, g, c, niter), ctx.cg(f, g, c, niter)
        for q, name in ((0, "x"), (1, "r"), (3, "p")):
            assert np.array_equal(np.isfinite(got[q]), np.isfinite(o[name])), name
        assert not (np.isfinite(got[2]) & ~np.isfinite(o["w"])).any()
