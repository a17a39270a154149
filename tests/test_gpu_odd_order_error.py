"""The error that the odd orders' fixed-point operator leaves in CG, against a
solve in extended precision, beside the error of the oracle's FP64 sums on the
same inputs: no larger.  After 16 iterations both are about 2.5e-16 (2-norm,
mean over right-hand sides; the spread of a mean of three is a tenth), so 1.5
times the oracle's bounds it; an operator whose lines lose half a unit at every
point leaves 2.5 to 4 times as much."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

DIMS, NITER = (2, 2, 2), 16
LD = np.longdouble


def extended_cg(D, g, c, f, mask, ids, lx):
    """NITER iterations of cg.f:36-75 in extended precision."""
    sh = (f.size // lx ** 3, lx, lx, lx)
    D, g, c = D.astype(LD), g.astype(LD).reshape(sh + (6,)), c.astype(LD).reshape(sh)

    def along(M, u, axis):
        return np.moveaxis(np.tensordot(u, M, axes=(axis, 1)), -1, axis)

    def ax(u):
        r, s, t = along(D, u, 3), along(D, u, 2), along(D, u, 1)
        w = along(D.T, g[..., 0] * r + g[..., 1] * s + g[..., 2] * t, 3)
        w += along(D.T, g[..., 1] * r + g[..., 3] * s + g[..., 4] * t, 2)
        w += along(D.T, g[..., 2] * r + g[..., 4] * s + g[..., 5] * t, 1)
        total = np.zeros(ids.max() + 1, LD)
        np.add.at(total, ids, w.ravel())
        return (total[ids].reshape(sh) + LD(0.1) * u) * mask

    x, r, p = np.zeros(sh, LD), f.reshape(sh).astype(LD) * mask, np.zeros(sh, LD)
    rz0, rz = LD(1), (r * c * r).sum()
    for it in range(NITER):
        p = r + (rz / rz0 if it else LD(0)) * p
        w = ax(p)
        a = rz / (w * c * p).sum()
        x, r = x + a * p, r - a * w
        rz0, rz = rz, (r * c * r).sum()
    return x.ravel()


@pytest.mark.parametrize("lx", [5, 9, 11])
def test_error_in_cg_is_no_larger_than_the_oracles(lx):
    import nekbone_gb300 as nb
    mesh, ctx = nb.Nekbone(*DIMS, lx, mask_mode=1), O.Ctx(*DIMS, lx, mask_mode=1)
    c, g, ids = mesh.set_multiplicity(), mesh.setup_g(), mesh.glo_num - mesh.glo_num.min()
    mask = np.ones(mesh.n)
    ctx.maskit(mask)
    mask = mask.reshape(-1, lx, lx, lx)
    D = np.asarray(mesh.dxm1).reshape(lx, lx)
    D = D if abs(D.sum(1)).max() < abs(D.sum(0)).max() else D.T   # rows differentiate a constant
    mine, oracle = [], []
    for seed in range(3):
        f = np.random.default_rng(seed).standard_normal(ids.max() + 1)[ids]
        ref = extended_cg(D, g, c, f, mask, ids, lx)
        for err, x in ((mine, mesh.cg(f, g, c, NITER)[0]),
                       (oracle, ctx.cg(f.copy(), g, c, NITER)["x"])):
            err.append(float(np.sqrt(((x - ref) ** 2).sum() / (ref ** 2).sum())))
    assert np.mean(oracle) < 1e-15   # the reference is the same problem
    assert np.mean(mine) <= 1.5 * np.mean(oracle), (mine, oracle)
