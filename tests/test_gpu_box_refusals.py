"""Right-hand sides with one copy of a shared point that differs, on a box whose
update would otherwise take the sums over copies: the copy next to each face of
the middle element, one on an edge and one at a corner, in turn the lower and
the upper of its pair.  All outputs of cg against the oracle, to 1e-12 as in the
other CG tests (the assembled form would be off by 1e-2)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

# which end of the element (0 first, 1 inside, 2 last) along x, y, z
POINTS = [(0, 1, 1), (2, 1, 1), (1, 0, 1), (1, 2, 1), (1, 1, 0), (1, 1, 2), (0, 2, 1), (1, 2, 2),
          (0, 0, 0), (2, 2, 2), (2, 0, 2)]


@pytest.mark.parametrize("lx", [6, 7, 10])
@pytest.mark.parametrize("mask_mode", [0, 1])
@pytest.mark.parametrize("where", POINTS)
@pytest.mark.parametrize("fp32", [False, True])
def test_one_copy_differs(lx, mask_mode, where, fp32):
    torch = pytest.importorskip("torch")
    import nekbone_gb300 as nb
    host, ctx = nb.Nekbone(3, 3, 3, lx, mask_mode=1), O.Ctx(3, 3, 3, lx, mask_mode=mask_mode)
    c, g = host.set_multiplicity(), host.setup_g()
    f = np.random.default_rng(lx).uniform(-1, 1, host.glo_num.max() + 1)[host.glo_num]
    i, j, k = ((0, 2, lx - 1)[a] for a in where)
    at = 13 * lx ** 3 + i + lx * (j + lx * k)
    assert c[at] < 1                        # it has copies, and none is masked:
    copies = np.flatnonzero(host.glo_num == host.glo_num[at])
    full = np.ones(host.n)
    O.Ctx(3, 3, 3, lx, mask_mode=1).maskit(full)
    assert full[copies].all() and copies.size > 1
    f[at] += 1e3 if fp32 else 0.25
    m = nb.DeviceMesh(3, 3, 3, lx, mask_mode=mask_mode)
    typ = torch.float32 if fp32 else torch.float64
    fd, gd, cd = (torch.tensor(v, dtype=typ, device="cuda") for v in (f, g, c))
    for _ in range(2):                      # the first builds the reference's mask list
        v = {q: torch.zeros(m.n, dtype=typ, device="cuda") for q in "xrwpz"}
        torch.cuda.synchronize()
        a = [t.data_ptr() for t in (v["x"], fd, gd, cd, v["r"], v["w"], v["p"])]
        m.cg_f32(*a, 2) if fp32 else m.cg(*a, v["z"].data_ptr(), 2)
        nb.sync()
        o = ctx.cg(f.copy(), g, c, 2)
        for name in "xrwp":
            err = np.abs(v[name].cpu().numpy() - o[name]).max() / np.abs(o[name]).max()
            # FP32: two applies of sums of 8 lx1 terms at 6e-8, grown tenfold at most
            assert err <= (1e-4 if fp32 else 1e-12), (name, err)
