"""CG on a box where the update takes the sums over copies itself (no pass
writes them back): every output of cg against the oracle, on boxes with one
element in a direction, odd and even lx1, in both mask modes, and for right-
hand sides and multiplicities that the form refuses (a copy that differs, c
that is not the inverse multiplicity), which take the general iteration.

Tolerance: 1e-12 relative after at most 12 iterations, as the other CG tests
assert after 100 (FP64); 2e-4 for FP32 (12 iterations of sums of at most
8 lx1 terms at 6e-8 each, grown by the residual's fall of at most 1e-1)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nb():
    import nekbone_gb300 as m
    return m


def rel(a, b):
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


@pytest.mark.parametrize("dims", [(3, 3, 3, 6), (4, 1, 2, 5), (1, 3, 1, 8), (2, 2, 2, 3),
                                  (5, 4, 3, 10), (1, 1, 1, 9)])
@pytest.mark.parametrize("mask_mode", [0, 1])
@pytest.mark.parametrize("kind", ["continuous", "copy_differs", "other_c"])
@pytest.mark.parametrize("niter", [1, 2, 5])
def test_cg_matches_oracle(nb, dims, mask_mode, kind, niter):
    mesh = nb.Nekbone(*dims, mask_mode=mask_mode)
    ctx = O.Ctx(*dims, mask_mode=mask_mode)
    c, g = mesh.set_multiplicity(), mesh.setup_g()
    rng = np.random.default_rng(sum(dims))
    f = rng.uniform(-1, 1, mesh.glo_num.max() + 1)[mesh.glo_num]
    if kind == "copy_differs":
        f[np.flatnonzero(c < 1)[-1:]] += 0.25
    if kind == "other_c":
        c = c * rng.uniform(0.5, 1.0, c.size)
    for _ in range(2):   # the first call builds the reference's mask list
        x, r, w, p, z, _ = mesh.cg(f, g, c, niter)
        o = ctx.cg(f, g, c, niter)
        for name, got in (("x", x), ("r", r), ("w", w), ("p", p)):
            assert rel(got, o[name]) <= 1e-12, (name, rel(got, o[name]))


@pytest.mark.parametrize("dims", [(3, 4, 2, 6), (2, 3, 4, 12), (3, 2, 2, 7)])
@pytest.mark.parametrize("niter", [1, 6])
def test_cg_f32_follows_oracle(nb, dims, niter):
    torch = pytest.importorskip("torch")
    m = nb.DeviceMesh(*dims, mask_mode=1)
    ctx = O.Ctx(*dims, mask_mode=1)
    c, g = ctx.set_multiplicity(), ctx.setup_g()
    host = nb.Nekbone(*dims, mask_mode=1)
    f = np.random.default_rng(1).uniform(-1, 1, host.glo_num.max() + 1)[host.glo_num]
    o = ctx.cg(f, g, c, niter)
    dev = [torch.tensor(v, dtype=torch.float32, device="cuda") for v in (f, g, c)]
    x, r, w, p = (torch.zeros(m.n, dtype=torch.float32, device="cuda") for _ in range(4))
    m.cg_f32(*(t.data_ptr() for t in (x, *dev, r, w, p)), niter)
    nb.sync()
    for name, got in (("x", x), ("r", r), ("w", w), ("p", p)):
        assert rel(got.cpu().numpy(), o[name]) <= 2e-4, name
