"""What this framework is measured on: passes through its public entry points
(the solvers, the operator and the gather-scatter on device vectors, and the
drop-in routine on host arrays) over the range of meshes that they serve.

A case names a kind of pass, the box of elements, lx1 (points per direction),
the metric ("box": every element the same, as setup_g makes it; "deformed":
a smooth deformation of the box, a full symmetric metric at every point) and
the iterations or the tolerance.  Inputs and the 64-bit results to compare
with are made here with torch and numpy alone.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import nekbone_gb300 as nb

# CG passes run 50 iterations: half of the reference driver's 100, so that
# the residual and the direction that come back are still far above rounding.
NITER = 50
# Solves to a tolerance go to 1e-12: what comes back is the solution to more
# digits than it is compared to.
TOL = 1e-12


def listed():
    return [
        # one operator application on a mesh of a few elements: a code that
        # calls the operator from its own loop; latency and launches
        dict(name="ax_smallest", kind="ax", ex=2, ey=2, ez=2, lx=6, metric="box"),
        # the reference's own example: 4x4x4 elements of order 9
        dict(name="cg_example", kind="cg", ex=4, ey=4, ez=4, lx=10, metric="box", niter=NITER),
        # an odd number of points per direction (the driver sweeps all
        # orders) on a ragged box
        dict(name="cg_odd_order", kind="cg", ex=12, ey=10, ez=9, lx=9, metric="box", niter=NITER),
        # a deformed mesh of medium size
        dict(name="cg_deformed", kind="cg", ex=16, ey=16, ez=16, lx=8, metric="deformed",
             niter=NITER),
        # the benchmark configuration: 32x32x32 elements, lx1 = 12
        dict(name="cg_headline", kind="cg", ex=32, ey=32, ez=32, lx=12, metric="box",
             niter=NITER),
        # the drop-in routine called with host arrays and the reference's
        # own mask, as the Fortran driver calls it
        dict(name="cg_dropin_host", kind="dropin", ex=8, ey=8, ez=8, lx=10, metric="box",
             niter=NITER),
        # the operator alone on a deformed mesh, FP64 and FP32
        dict(name="ax_deformed", kind="ax", ex=16, ey=16, ez=16, lx=12, metric="deformed"),
        dict(name="ax_fp32_deformed", kind="ax_f32", ex=16, ey=16, ez=16, lx=16,
             metric="deformed"),
        # the mixed-precision solver at the size of a production mesh
        dict(name="mixed_solve", kind="mixed", ex=24, ey=24, ez=24, lx=12, metric="box", tol=TOL),
        # the multigrid-preconditioned solver with the FP32 smoother
        dict(name="hsmg_pcg", kind="pcg", ex=16, ey=16, ez=16, lx=12, metric="deformed", tol=TOL),
        # many uneven problems solved together
        dict(name="batch_uneven", kind="batch", problems=64, most=1024, shapes=1, tol=TOL),
        # the gather-scatter alone on a resident FP64 field
        dict(name="dssum", kind="dssum", ex=24, ey=20, ez=22, lx=10, metric="box"),
    ]


def draw(rng: random.Random):
    kind = rng.choices(["cg", "ax", "mixed", "dropin", "pcg", "batch", "ax_f32", "dssum"],
                       [32, 18, 12, 10, 8, 8, 6, 6])[0]
    if kind == "batch":
        return dict(kind=kind, problems=rng.randint(4, 96), most=rng.choice([256, 512, 1024]),
                    shapes=rng.randrange(10 ** 6), tol=TOL)
    lx = rng.choice([8, 10, 12]) if kind == "pcg" else rng.randint(4, 16)
    # points of the mesh, spread over the logarithm
    least, largest = {"cg": (1e3, 3e7), "ax": (1e3, 3e7), "mixed": (1e4, 2e7), "dropin": (1e3, 2e6),
                   "pcg": (5e4, 7e6), "ax_f32": (1e4, 3e7), "dssum": (1e4, 3e7)}[kind]
    nelt = max(1.0, math.exp(rng.uniform(math.log(least), math.log(largest))) / lx ** 3)
    side = nelt ** (1 / 3)
    # (the preconditioner's levels want more than one element a direction)
    low = 2 if kind == "pcg" else 1
    ex = max(low, round(side * rng.uniform(0.7, 1.4)))
    ey = max(low, round(side * rng.uniform(0.7, 1.4)))
    ez = max(low, round(nelt / (ex * ey)))
    case = dict(kind=kind, ex=ex, ey=ey, ez=ez, lx=lx,
                metric="box" if kind in ("dropin", "dssum") else rng.choice(["box", "deformed"]))
    if kind in ("cg", "dropin"):
        # (a box of few elements has few distinct modes: CG is through with it
        # in few iterations, and what then comes back is rounding)
        few = min(ex, ey, ez)
        most = 10 if few == 1 else 15 if few < 4 else 30 if few < 6 or lx < 6 else NITER
        case["niter"] = rng.randint(8, most)
    if kind in ("mixed", "pcg"):
        case["tol"] = TOL
    return case


# ------------------------------------------------------------------ inputs --
DEV = "cuda"


def gll(n):
    """GLL points, weights and derivative matrix D(i, m) of n points."""
    leg = np.polynomial.legendre.Legendre.basis(n - 1)
    d1 = leg.deriv()
    d2 = d1.deriv()
    x = np.concatenate([[-1.0], np.sort(d1.roots().real), [1.0]])
    for _ in range(3):
        x[1:-1] -= d1(x[1:-1]) / d2(x[1:-1])
    x = (x - x[::-1]) / 2
    v = leg(x)
    w = 2.0 / (n * (n - 1) * v * v)
    d = np.zeros((n, n))
    for i in range(n):
        for m in range(n):
            if i != m:
                d[i, m] = v[i] / v[m] / (x[i] - x[m])
    d[0, 0], d[-1, -1] = -n * (n - 1) / 4, n * (n - 1) / 4
    return x, w, d


def global_ids(ex, ey, ez, lx):
    """The box number of every local point, (ez, ey, ex, k, j, i) flattened,
    and the sizes of the global grid."""
    def line(ne):
        e = torch.arange(ne, device=DEV)[:, None] * (lx - 1)
        return e + torch.arange(lx, device=DEV)[None, :]
    nx, ny, nz = ex * (lx - 1) + 1, ey * (lx - 1) + 1, ez * (lx - 1) + 1
    gx, gy, gz = line(ex), line(ey), line(ez)
    ids = (gx[None, None, :, None, None, :] + gy[None, :, None, None, :, None] * nx
           + gz[:, None, None, :, None, None] * (nx * ny))
    return ids.reshape(-1), (nz, ny, nx)


def multiplicity(ex, ey, ez, lx):
    """c: one over the number of copies of every local point."""
    def line(ne):
        c = torch.ones(ne, lx, dtype=torch.float64, device=DEV)
        c[1:, 0] = 0.5
        c[:-1, -1] = 0.5
        return c
    cx, cy, cz = line(ex), line(ey), line(ez)
    return (cx[None, None, :, None, None, :] * cy[None, :, None, None, :, None]
            * cz[:, None, None, :, None, None]).reshape(-1)


def field(case, seed):
    """A continuous field, uniform in [-1, 1) at every global point inside
    and zero on the boundary of the box."""
    ids, (nz, ny, nx) = global_ids(case["ex"], case["ey"], case["ez"], case["lx"])
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    v = torch.rand(nz, ny, nx, dtype=torch.float64, device=DEV, generator=gen) * 2 - 1
    for a in (0, -1):
        v[a] = 0
        v[:, a] = 0
        v[:, :, a] = 0
    return v.reshape(-1)[ids]


def metric(case, seed):
    """g(6, point): w |J| J^-1 J^-T of the box or of a smooth deformation."""
    ex, ey, ez, lx = case["ex"], case["ey"], case["ez"], case["lx"]
    x, w, _ = gll(lx)
    w = torch.tensor(w, device=DEV)
    www = (w[None, None, :] * w[None, :, None]) * w[:, None, None]
    n = ex * ey * ez * lx ** 3
    g = torch.zeros(n, 6, dtype=torch.float64, device=DEV)
    if case["metric"] == "box":
        for q in (0, 3, 5):
            g[:, q] = www.reshape(-1).repeat(ex * ey * ez)
        return g.reshape(-1)
    # X = xi + sum_q a_q sin(k_q . xi + phi_q), elements of size 2
    rng = np.random.default_rng(seed)
    size = (2.0 * ex, 2.0 * ey, 2.0 * ez)
    pts = torch.tensor(x, device=DEV)

    def line(ne):
        return 2.0 * torch.arange(ne, device=DEV, dtype=torch.float64)[:, None] + 1 + pts[None, :]
    cx = line(ex)[None, None, :, None, None, :]
    cy = line(ey)[None, :, None, None, :, None]
    cz = line(ez)[:, None, None, :, None, None]
    jac = [[torch.full((1,), float(a == b), dtype=torch.float64, device=DEV) for b in range(3)]
           for a in range(3)]
    for _ in range(2):
        k = [2 * math.pi * int(rng.integers(1, 3)) / s for s in size]
        a = rng.uniform(-1, 1, 3) * 0.06 / max(k)
        t = torch.cos(k[0] * cx + k[1] * cy + k[2] * cz + rng.uniform(0, 2 * math.pi)).reshape(-1)
        for d in range(3):
            for b in range(3):
                jac[d][b] = jac[d][b] + a[d] * k[b] * t
    cof = [[jac[(a + 1) % 3][(b + 1) % 3] * jac[(a + 2) % 3][(b + 2) % 3]
            - jac[(a + 1) % 3][(b + 2) % 3] * jac[(a + 2) % 3][(b + 1) % 3] for b in range(3)]
           for a in range(3)]
    det = sum(jac[0][b] * cof[0][b] for b in range(3))
    scale = www.reshape(-1).repeat(ex * ey * ez) / det
    for q, (a, b) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
        g[:, q] = scale * sum(cof[d][a] * cof[d][b] for d in range(3))
    return g.reshape(-1)


def boxes(case):
    """The batch's problems: elements log-uniform from 8, uneven boxes."""
    rng = random.Random(case["shapes"])
    out = []
    for _ in range(case["problems"]):
        nelt = math.exp(rng.uniform(math.log(8), math.log(case["most"])))
        a = max(1, round(nelt ** (1 / 3) * rng.uniform(0.7, 1.4)))
        b = max(1, round(nelt ** (1 / 3) * rng.uniform(0.7, 1.4)))
        out.append((a, b, max(1, round(nelt / (a * b))), rng.choice([6, 8, 10, 12])))
    return out


def part(box, i):
    """Problem i of a batch as a case of its own (its seed goes with it)."""
    return dict(ex=box[0], ey=box[1], ez=box[2], lx=box[3], metric="box")


def part_seed(seed, i):
    return seed * 1000 + i


class DeviceArray:
    """A library vector of n doubles, for torch.as_tensor (the tensor keeps
    this object, and this object the vector's owner)."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (ptr, False),
                                         "version": 2}


class State:
    pass


def prepare(case, seed):
    s = State()
    s.kind, s.case = case["kind"], case
    if s.kind == "batch":
        s.batch = nb.Batch(boxes(case))
        s.batch.setup(seed)
        s.batch.set_inner_tol(1e-5)
        x, f = s.batch.arrays()[:2]
        s.x = torch.as_tensor(DeviceArray(s.batch, x, s.batch.n), device=DEV)
        f = torch.as_tensor(DeviceArray(s.batch, f, s.batch.n), device=DEV)
        for i, box in enumerate(s.batch.boxes):
            at, n, _ = s.batch.problem(i)
            f[at:at + n] = field(part(box, i), part_seed(seed, i))
        return s
    dims = case["ex"], case["ey"], case["ez"], case["lx"]
    f = field(case, seed)
    n = f.numel()
    if s.kind == "dropin":
        s.mesh = nb.Nekbone(*dims, mask_mode=0)
        s.f = f.cpu().numpy()
        s.g = metric(case, seed).cpu().numpy()
        s.c = multiplicity(*dims).cpu().numpy()
        s.work = tuple(np.zeros(n) for _ in range(5))
        return s
    s.mesh = nb.DeviceMesh(*dims, mask_mode=1)
    s.f = f
    if s.kind == "dssum":
        s.w = torch.empty_like(f)
        return s
    s.g = metric(case, seed)
    if s.kind == "ax_f32":
        s.f, s.g = s.f.float(), s.g.float()
    if s.kind in ("ax", "ax_f32"):
        s.w = torch.empty_like(s.f)
        return s
    s.c = multiplicity(*dims)
    s.x = torch.empty_like(f)
    if s.kind == "cg":
        s.r, s.w, s.p, s.z = (torch.empty_like(f) for _ in range(4))
    if s.kind == "pcg":
        # levels of 12 -> 6 -> 3 points; the reference's own choice below
        s.mesh.mg_setup([2, 5, 11] if case["lx"] == 12 else None, precision=32)
    return s


def run(s):
    m, case = getattr(s, "mesh", None), s.case
    if s.kind == "ax":
        m.ax(s.w.data_ptr(), s.f.data_ptr(), s.g.data_ptr())
        return s.w
    if s.kind == "ax_f32":
        m.ax_f32(s.w.data_ptr(), s.f.data_ptr(), s.g.data_ptr())
        return s.w
    if s.kind == "dssum":
        # (the library's stream orders with the default stream)
        s.w.copy_(s.f)
        m.dssum(s.w.data_ptr())
        return s.w
    if s.kind == "cg":
        m.cg(*(t.data_ptr() for t in (s.x, s.f, s.g, s.c, s.r, s.w, s.p, s.z)), case["niter"])
        return {"x": s.x, "r": s.r, "w": s.w, "p": s.p}
    if s.kind == "dropin":
        x, r, w, p, _, _ = m.cg(s.f, s.g, s.c, case["niter"], work=s.work)
        return {"x": x, "r": r, "w": w, "p": p}
    if s.kind == "mixed":
        m.cg_mixed(*(t.data_ptr() for t in (s.x, s.f, s.g, s.c)), case["tol"])
        return s.x
    if s.kind == "pcg":
        m.pcg_tol(*(t.data_ptr() for t in (s.x, s.f, s.g, s.c)), case["tol"])
        return s.x
    s.batch.solve(case["tol"], inner_iters=80)
    return s.x


# ------------------------------------------------------------- 64-bit value --
class Reference:
    """The operator A = mask(QQ^T A_L + 0.1 I) and its CG in torch, FP64."""

    def __init__(self, case, g, mask):
        self.shape = (-1, case["lx"], case["lx"], case["lx"])
        self.ids, grid = global_ids(case["ex"], case["ey"], case["ez"], case["lx"])
        self.size = math.prod(grid)
        self.g = [t.contiguous().reshape(self.shape) for t in g.reshape(-1, 6).unbind(1)]
        self.mask = mask
        self.D = torch.tensor(gll(case["lx"])[2], device=DEV)

    def dssum(self, u):
        t = torch.zeros(self.size, dtype=torch.float64, device=DEV)
        return t.index_add_(0, self.ids, u)[self.ids]

    def along(self, M, u):
        """M applied along i, j and k of every element."""
        n = M.shape[0]
        return u @ M.T, M @ u, (M @ u.reshape(-1, n, n * n)).reshape(u.shape)

    def ax(self, u):
        g, D = self.g, self.D
        ur, us, ut = self.along(D, u.reshape(self.shape))
        w = (g[0] * ur + g[1] * us + g[2] * ut) @ D
        w = w + D.T @ (g[1] * ur + g[3] * us + g[4] * ut)
        n = D.shape[0]
        t = (g[2] * ur + g[4] * us + g[5] * ut).reshape(-1, n, n * n)
        w = w + (D.T @ t).reshape(w.shape)
        return (self.dssum(w.reshape(-1)) + 0.1 * u) * self.mask

    def cg(self, f, c, niter, tol=0.0):
        x, r, p = torch.zeros_like(f), f * self.mask, torch.zeros_like(f)
        rtz = first = 1.0
        for it in range(niter):
            last, rtz = rtz, float((r * c).dot(r))
            first = rtz if it == 0 else first
            if rtz <= tol * tol * first:
                break
            p = r + (rtz / last if it else 0.0) * p
            w = self.ax(p)
            alpha = rtz / float((w * c).dot(p))
            x += alpha * p
            r -= alpha * w
        return {"x": x, "r": r, "w": w, "p": p}


def exact(case, seed):
    if case["kind"] == "batch":
        out = []
        # the concatenated vectors hold the problems in order of lx1
        every = sorted(enumerate(boxes(case)), key=lambda b: b[1][3])
        for i, box in every:
            one = dict(part(box, i), kind="mixed", tol=case["tol"])
            out.append(exact(one, part_seed(seed, i)))
        return torch.cat(out)
    dims = case["ex"], case["ey"], case["ez"], case["lx"]
    f = field(case, seed)
    if case["kind"] == "dssum":
        ids, grid = global_ids(*dims)
        t = torch.zeros(math.prod(grid), dtype=torch.float64, device=DEV)
        return t.index_add_(0, ids, f)[ids]
    g = metric(case, seed)
    # zero on the boundary of the box ...
    ids, (nz, ny, nx) = global_ids(*dims)
    inside = torch.zeros(nz, ny, nx, dtype=torch.float64, device=DEV)
    inside[1:-1, 1:-1, 1:-1] = 1
    mask = inside.reshape(-1)[ids]
    if case["kind"] == "dropin":
        # ... with the reference's own mask in its first element alone
        mask[case["lx"] ** 3:] = 1
    if case["kind"] == "ax_f32":
        f, g = f.float().double(), g.float().double()
    A = Reference(case, g, mask)
    if case["kind"] in ("ax", "ax_f32"):
        return A.ax(f)
    c = multiplicity(*dims)
    if case["kind"] in ("cg", "dropin"):
        return A.cg(f, c, case["niter"])
    return A.cg(f, c, 400, case["tol"])["x"]


def work(case):
    """Per pass: the vectors and the metric that it cannot do without, and
    the operator's 12 lx1 + 19 and the vectors' 15 operations a point."""
    if case["kind"] == "batch":
        n = sum(b[0] * b[1] * b[2] * b[3] ** 3 for b in boxes(case))
        flops = sum(b[0] * b[1] * b[2] * b[3] ** 3 * (12 * b[3] + 34) for b in boxes(case))
        # about 120 FP32 iterations: r, x, p read and written, the metric read
        return {"bytes": 120 * 48 * n, "flops": 120 * flops}
    n = case["ex"] * case["ey"] * case["ez"] * case["lx"] ** 3
    per = 12 * case["lx"] + 19
    if case["kind"] == "dssum":
        return {"bytes": 16 * n, "flops": n}
    if case["kind"] == "ax":
        return {"bytes": 64 * n, "flops": per * n}
    if case["kind"] == "ax_f32":
        return {"bytes": 32 * n, "flops": per * n}
    if case["kind"] in ("cg", "dropin"):
        return {"bytes": 96 * n * case["niter"], "flops": (per + 15) * n * case["niter"]}
    if case["kind"] == "mixed":
        # about 140 FP32 iterations
        return {"bytes": 48 * n * 140, "flops": (per + 15) * n * 140}
    # about 90 preconditioned FP64 iterations
    return {"bytes": 96 * n * 90, "flops": 2 * (per + 15) * n * 90}
