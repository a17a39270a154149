"""The batched inner CG where its update takes the sums over copies (a
residual that is equal at all copies of every point), and right-hand sides
that it refuses (a copy that differs, a value on the mask), which take the
general iteration: the solutions against the single mesh's FP64 CG, the
refused ones after three cycles against the single mesh's mixed solver, which
makes the same iterations.

Both solve to 1e-10 of |f|; A's smallest eigenvalue is above 1e-3 of its
largest on these boxes, so x agrees to 1e-6 relative.  Without convergence the
two solvers' 60 FP32 iterations differ by their sums' rounding (1e-7 each):
1e-3."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BOXES = [(2, 3, 2, 4), (3, 1, 2, 6), (1, 1, 1, 8), (2, 2, 3, 8), (3, 2, 2, 10), (2, 2, 2, 12),
         (7, 2, 3, 4)]


class View:
    def __init__(self, ptr, n):
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False),
                                         "version": 2}


@pytest.mark.parametrize("kind", ["continuous", "copy_differs", "on_the_mask"])
@pytest.mark.parametrize("paired", [True, False])
def test_solutions(kind, paired):
    torch = pytest.importorskip("torch")
    import nekbone_gb300 as nb
    b = nb.Batch(BOXES)
    b.setup(5)
    xp, fp = b.arrays()[:2]
    f = torch.as_tensor(View(fp, b.n), device="cuda")
    x = torch.as_tensor(View(xp, b.n), device="cuda")
    for p, box in enumerate(BOXES):
        at, n, lx = b.problem(p)
        l3 = lx ** 3
        if kind == "copy_differs" and n > l3:
            # the last point of the first element's x-row that has a copy
            f[at + l3 - 1] += 0.25
        elif kind == "on_the_mask":
            f[at] = 0.5
    fh = f.clone()
    nb.set_paired_update(paired)
    try:
        b.solve(1e-10, 20, 50 if kind == "continuous" else 3)
        res = [b.result(p) for p in range(len(BOXES))]
    finally:
        nb.set_paired_update(True)
    for p, box in enumerate(BOXES):
        at, n, lx = b.problem(p)
        m = nb.DeviceMesh(*box, mask_mode=1)
        g, c = (torch.empty(k * n, dtype=torch.float64, device="cuda") for k in (6, 1))
        m.setup_g(g.data_ptr())
        m.set_multiplicity(c.data_ptr())
        fm = fh[at:at + n].clone()
        xo = torch.zeros(n, dtype=torch.float64, device="cuda")
        if kind == "continuous":
            assert res[p][2] <= 1e-10
            m.cg_tol(xo.data_ptr(), fm.data_ptr(), g.data_ptr(), c.data_ptr(), 1e-12, 2000, 5)
            err = float((x[at:at + n] - xo).abs().max() / xo.abs().max())
            assert err <= 1e-6, (box, err)
        elif kind == "copy_differs" and min(box[:3]) > 1:
            # (else the corner is masked, which nb_cg_mixed applies to its
            # right-hand side and the batch does not)
            m.cg_mixed(xo.data_ptr(), fm.data_ptr(), g.data_ptr(), c.data_ptr(), 1e-10, 20, 3)
            err = float((x[at:at + n] - xo).abs().max() / xo.abs().max())
            assert err <= 1e-3, (box, err)
        assert bool(torch.isfinite(x[at:at + n]).all())
