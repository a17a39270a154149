"""cg with the right-hand side in one of the solve's own vectors: x is cleared,
whatever it holds, and the result is that of separate vectors, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 2, 4, 8), (2, 3, 2, 9), (3, 3, 3, 12), (2, 2, 2, 13)])
@pytest.mark.parametrize("mask_mode", [0, 1])
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("where", ["r", "w", "p"])
def test_rhs_in_a_work_vector(dims, mask_mode, fp32, where):
    torch = pytest.importorskip("torch")
    import nekbone_gb300 as nb
    m = nb.DeviceMesh(*dims, mask_mode=mask_mode)
    host = nb.Nekbone(*dims, mask_mode=1)
    c, g = host.set_multiplicity(), host.setup_g()
    f = np.random.default_rng(3).uniform(-1, 1, host.glo_num.max() + 1)[host.glo_num]
    typ = torch.float32 if fp32 else torch.float64
    fd, gd, cd = (torch.tensor(v, dtype=typ, device="cuda") for v in (f, g, c))

    def solve(alias):
        v = {k: torch.full((m.n,), 7.5, dtype=typ, device="cuda") for k in "xrwpz"}
        rhs = fd
        if alias:
            v[alias].copy_(fd)
            rhs = v[alias]
        torch.cuda.synchronize()
        a = [t.data_ptr() for t in (v["x"], rhs, gd, cd, v["r"], v["w"], v["p"])]
        m.cg_f32(*a, 4) if fp32 else m.cg(*a, v["z"].data_ptr(), 4)
        nb.sync()
        return [v[k].cpu().numpy() for k in "xrwp"]

    solve(None)   # the first solve builds the reference's mask list
    want = solve(None)
    assert np.isfinite(want[0]).all() and np.abs(want[0]).max() > 0
    for got, ref in zip(solve(where), want):
        assert np.array_equal(got, ref)
