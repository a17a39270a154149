"""The closed-form assembly of a box's boundary points (k_box_dssum, k_box_rest)
against jl's gather-scatter on the same numbering: dssum bitwise in both
precisions, and the operator's second pass through a numbering in another
element order (the boundary groups instead) against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def nb():
    import nekbone_gb300 as m
    return m


@pytest.mark.parametrize("dims", [(3, 2, 4, 6), (1, 1, 1, 4), (5, 1, 1, 3), (2, 2, 2, 2),
                                  (4, 3, 5, 9), (2, 3, 2, 16)])
@pytest.mark.parametrize("dtype", ["float64", "float32"])
def test_dssum_is_the_gather_scatter(nb, dims, dtype):
    torch = pytest.importorskip("torch")
    m = nb.DeviceMesh(*dims, mask_mode=1)
    host = nb.Nekbone(*dims, mask_mode=1)
    u = np.random.default_rng(3).uniform(-1, 1, m.n).astype(dtype)
    d = torch.tensor(u, device="cuda")
    m.dssum(d.data_ptr(), dom=1 if dtype == "float64" else 2)
    nb.sync()
    h = nb.gs_setup(host.glo_num)
    nb.gs_op(h, u, 1, 0)
    nb.gs_free(h)
    assert np.array_equal(d.cpu().numpy(), u)


@pytest.mark.parametrize("dims", [(3, 2, 2, 6), (2, 3, 2, 5)])
@pytest.mark.parametrize("order", [0, 2])
def test_ax_in_another_element_order(nb, dims, order):
    nelt = dims[0] * dims[1] * dims[2]
    lglel = np.random.default_rng(7).permutation(np.arange(1, nelt + 1)).astype(np.int32)
    mesh = nb.Nekbone(*dims, mask_mode=1, lglel=lglel)
    ctx = O.Ctx(*dims, mask_mode=1)
    rng = np.random.default_rng(8)
    g, u = rng.standard_normal(6 * mesh.n), rng.standard_normal(mesh.n)
    at = lglel - 1

    try:
        mesh.set_order(order)
        w = mesh.ax(u.reshape(nelt, -1)[at].reshape(-1).copy(),
                    g.reshape(nelt, -1)[at].reshape(-1).copy()).reshape(nelt, -1)
    finally:
        mesh.set_order(nb.DEFAULT_ORDER)
    wo = ctx.ax(u, g).reshape(nelt, -1)[at]
    # (the copies are summed in another order: rounding, not bits)
    assert np.abs(w - wo).max() <= 1e-13 * np.abs(wo).max()
