"""Performance cases of the GPK step and of the modules around it.

Each case is a plain dict; `kind` selects the public path it takes:

  growth     GPKGrid.step_n of a grain-growth grid: the microstructure is
             loaded from host arrays and advanced by `steps` steps (a run
             between two outputs); labels, alpha and the step's fields stay on
             the device, where the caller reads them
  geometry   GPKGrid.geometry: normals, curvature and competitors of a label
             field, without a step
  solidify   GPKGrid.step_graph of FP64 solidification with solute
             partitioning
  sweep      GPKBatch.step_graph of many small 2-D lamellar instances
  elastic    SpectralElasticity.solve on device tensors
  calibrate  AdjointProblem.gradient, the calibration loss and its gradient
  alcu       one step of the Al-Cu transport and remap chain on device tensors

`listed` are the sizes in use: the benchmark's workloads, the sizes of the
tests and odd ones.  `draw` spreads the same kinds over their ranges.
"""
from __future__ import annotations

import math
import os
import sys
import types

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "python")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

import gpk  # noqa: E402
from gpk import alcu  # noqa: E402
from gpk.spectral import variant_eigenstrains  # noqa: E402
from gpk_b200 import sweep  # noqa: E402

SETTLE = 16  # steps evolved before a growth state is used: the first crossings come at step 8


def listed():
    return [
        # a small 2-D polycrystal, as the known-answer tests and quick studies run: launches and latency
        dict(name="growth2d_64", kind="growth", nz=1, ny=64, nx=64, grains=16, sigma=1.5, precision="f32", steps=8),
        # an ordinary 2-D grain-growth run at the grid's default sigma
        dict(name="growth2d_512", kind="growth", nz=1, ny=512, nx=512, grains=500, sigma=2.0, precision="f32",
             steps=8),
        # a ragged 3-D box at the default sigma: no extent is a multiple of a tile
        dict(name="growth3d_ragged", kind="growth", nz=90, ny=101, nx=117, grains=300, sigma=2.0, precision="f32",
             steps=8),
        # the FP64 mode with the direct stencil
        dict(name="growth3d_f64_96", kind="growth", nz=96, ny=96, nx=96, grains=216, sigma=1.5, precision="f64",
             steps=8),
        # the benchmark's workload: 256^3, 4096 grains, sigma 1.5
        dict(name="growth3d_256", kind="growth", nz=256, ny=256, nx=256, grains=4096, sigma=1.5, precision="f32",
             steps=8),
        # wide smoothing (sigma 5), which selects the separable geometry
        dict(name="growth3d_sigma5", kind="growth", nz=128, ny=128, nx=128, grains=24, sigma=5.0, precision="f32",
             steps=8),
        # curvature of a polycrystal in FP64 with the throughput geometry (measurement of a snapshot)
        dict(name="curvature3d_f64", kind="geometry", nz=144, ny=160, nx=130, grains=700, sigma=1.5,
             precision="f64", kernel="separable_tiles"),
        # solidification with solute partitioning, FP64, as the coupled benchmark without its elastic solve
        dict(name="solidify3d_128", kind="solidify", n=128, radius=20, steps=16),
        # a parameter sweep of small 2-D instances as one graph
        dict(name="sweep2d_48", kind="sweep", instances=48, first=5000, steps=8),
        # the spectral elastic solve of the coupled benchmark
        dict(name="elastic3d_128", kind="elastic", n0=128, n1=128, n2=128, inclusions=12),
        # the calibration case: 512^2, 256 grains, 64 precipitates
        dict(name="calibrate2d_512", kind="calibrate", n=512, grains=256, precipitates=64),
        # the Al-Cu chain on a field of theta-prime plates
        dict(name="alcu3d_160", kind="alcu", n0=160, n1=160, n2=160, plates=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["growth", "growth", "growth", "growth", "coarse", "geometry", "solidify", "sweep", "elastic",
                       "calibrate", "alcu"])
    if kind == "growth":
        f64 = rng.random() < 0.3
        sigma = rng.choice([1.0, 1.25, 1.5, 2.0, 2.2])
        if rng.random() < 0.5:
            nz, ny, nx = 1, _log(rng, 48, 900), _log(rng, 48, 900)
            grains = max(4, ny * nx // _log(rng, 120, 1500))
        else:
            top = 120 if f64 else 210
            nz, ny, nx = (_log(rng, 32, top) for _ in range(3))
            grains = max(4, nz * ny * nx // _log(rng, 1500, 9000))
        return dict(kind="growth", nz=nz, ny=ny, nx=nx, grains=grains, sigma=sigma,
                    precision="f64" if f64 else "f32", steps=8)
    if kind == "coarse":
        nz, ny, nx = (_log(rng, 64, 160) for _ in range(3))
        return dict(kind="growth", nz=nz, ny=ny, nx=nx, grains=max(4, nz * ny * nx // _log(rng, 60000, 150000)),
                    sigma=rng.choice([4.75, 5.0, 5.5, 6.0]), precision="f32", steps=8)
    if kind == "geometry":
        f64 = rng.random() < 0.7
        nz, ny, nx = (_log(rng, 40, 180) for _ in range(3))
        return dict(kind="geometry", nz=nz, ny=ny, nx=nx, grains=max(4, nz * ny * nx // _log(rng, 1500, 9000)),
                    sigma=rng.choice([1.0, 1.5, 2.0]), precision="f64" if f64 else "f32",
                    kernel="separable_tiles" if f64 else "tiled")
    if kind == "solidify":
        n = _log(rng, 48, 160)
        return dict(kind="solidify", n=n, radius=rng.randint(5, n // 4), steps=16)
    if kind == "sweep":
        return dict(kind="sweep", instances=rng.randint(6, 64), first=rng.randint(0, 4000), steps=8)
    if kind == "elastic":
        if rng.random() < 0.4:
            n0, n1 = _log(rng, 64, 1024), _log(rng, 64, 1024)
            return dict(kind="elastic", n0=n0, n1=n1, n2=0, inclusions=rng.randint(2, 20))
        n0, n1, n2 = (_log(rng, 32, 160) for _ in range(3))
        return dict(kind="elastic", n0=n0, n1=n1, n2=n2, inclusions=rng.randint(2, 20))
    if kind == "calibrate":
        n = _log(rng, 96, 640)
        return dict(kind="calibrate", n=n, grains=max(8, n * n // _log(rng, 500, 2000)),
                    precipitates=max(4, n * n // _log(rng, 3000, 9000)))
    n0, n1, n2 = (_log(rng, 48, 192) for _ in range(3))
    return dict(kind="alcu", n0=n0, n1=n1, n2=n2, plates=max(2, n0 * n1 * n2 // _log(rng, 30000, 90000)))


# ---------------------------------------------------------------------------
# device views of a grid's fields
# ---------------------------------------------------------------------------
class _Field:
    def __init__(self, grid, name):
        dt = {"phi": "<i4", "phi_comp": "<i4", "mask": "|u1"}.get(name, "<f4" if grid.precision == "f32" else "<f8")
        self.grid = grid  # the memory belongs to the grid
        self.__cuda_array_interface__ = {"shape": (grid.Nz, grid.Ny, grid.Nx), "typestr": dt, "version": 2,
                                         "data": (grid.device_ptr(name), False)}


def _view(grid, name):
    return torch.as_tensor(_Field(grid, name), device="cuda")


def _pinned(array):
    t = torch.empty(array.shape, dtype=torch.from_numpy(array).dtype, pin_memory=True)
    t.numpy()[...] = array
    return t.numpy()


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _growth_grid(case, seed):
    grid = gpk.GPKGrid(case["nz"], case["ny"], case["nx"], 1.0, gpk.thermo.isotropic(1.0, 1.0), 0.0, case["sigma"],
                       precision=case["precision"])
    rng = np.random.default_rng([seed, 1])
    n, shape = case["grains"], (case["nz"], case["ny"], case["nx"])
    seeds = np.stack(np.unravel_index(rng.choice(math.prod(shape), n, replace=False), shape))
    grid.voronoi_seeds(seeds, rng.uniform(0.0, math.pi / 2, n).astype(np.float32))
    grid.set("alpha", 1.0)
    return grid


def _plates(case, rng):
    """int8 labels of theta-prime plates: thin along the variant's axis, aspect 8, periodic."""
    shape = (case["n0"], case["n1"], case["n2"])
    lab = np.zeros(shape, dtype=np.int8)
    for k in range(case["plates"]):
        centre, v = [int(rng.integers(0, e)) for e in shape], 1 + k % 3
        axes = np.full(3, 6.0 * rng.uniform(0.9, 2.2))
        axes[v - 1] /= 8.0
        half = [min(int(math.ceil(a)), (e - 1) // 2) for a, e in zip(axes, shape)]
        offs = [np.arange(-h, h + 1) for h in half]
        win = np.ix_(*[(centre[a] + offs[a]) % shape[a] for a in range(3)])
        d2 = sum(((offs[a] / axes[a]) ** 2).reshape([-1 if b == a else 1 for b in range(3)]) for a in range(3))
        sub = lab[win]
        sub[d2 <= 1.0] = v
        lab[win] = sub
    return lab


ALCU = types.SimpleNamespace(dx=1.5e-9, diffusivity=1.66e-20, c_matrix_eq=3.7189506575706577e-4, c_theta=1.0 / 3.0,
                             composition_extension_sigma_cells=0.75)
ALCU_DT, ALCU_REMAP_SIGMA = 10.0, 0.70
CUBIC = dict(c11=108e9, c12=62e9, c44=28e9)
CALIBRATE = dict(m_fixed=1.0, sigma0=1e-3, c11=1.08, c12=0.62, c44=0.28, energy_weight=1e-6)


def _elastic_shape(case):
    return tuple(e for e in (case["n0"], case["n1"], case["n2"]) if e)


def _elastic_fractions(case, seed):
    """Three variants' fractions: smooth-edged ellipsoidal inclusions on a periodic field."""
    rng = np.random.default_rng([seed, 2])
    shape = _elastic_shape(case)
    f = torch.zeros((3,) + shape, dtype=torch.float64, device="cuda")
    axes = [torch.arange(e, dtype=torch.float64, device="cuda") for e in shape]
    for k in range(case["inclusions"]):
        d2 = 0.0
        for a, e in enumerate(shape):
            d = torch.remainder(axes[a] - rng.uniform(0, e) + 0.5 * e, e) - 0.5 * e
            r = rng.uniform(2.0, max(3.0, 0.12 * e))
            d2 = d2 + ((d / r) ** 2).reshape([-1 if b == a else 1 for b in range(len(shape))])
        f[k % 3] = torch.maximum(f[k % 3], torch.sigmoid(6.0 * (1.0 - d2)))
    return f / torch.clamp(f.sum(0, keepdim=True), min=1.0)


def _calibration(case, seed):
    """2-D polycrystal with circular precipitates, as gpk.adjoint.calibration_case lays it out."""
    n, grains = case["n"], case["grains"]
    phi, g, mob = gpk.calibration_case(n, grains, case["precipitates"], 1 + seed % (1 << 20), (5, 14))
    rng = np.random.default_rng([seed, 3])
    theta = np.concatenate([[0.01, -0.004, 0.003], [0.05, -0.02, 0.01, 0.005],
                            1.0 + 0.1 * rng.standard_normal(grains)])
    return phi, g, mob, theta


def prepare(case, seed):
    kind = case["kind"]
    s = types.SimpleNamespace(case=case, kind=kind)
    if kind == "growth":
        s.grid = _growth_grid(case, seed)
        s.grid.step_n(SETTLE)
        s.load = {k: _pinned(s.grid.get(k)) for k in ("phi", "alpha", "g")}
    elif kind == "geometry":
        s.grid = _growth_grid(case, seed)
        s.grid.set_geometry_kernel(case["kernel"])
    elif kind == "solidify":
        n = case["n"]
        th = gpk.thermo.solidification(M0=5e-8, sigma0=0.2, eps4=0.04, m_liq=-500.0, k_part=0.14, T_melt=933.0,
                                       L=1e8)
        th.solute_rejection, th.k_partition = True, 0.14
        s.grid = grid = gpk.GPKGrid(n, n, n, 0.5e-6, th, 3e-9, 1.5, precision="f64")
        rng = np.random.default_rng([seed, 4])
        z, y, x = np.indices((n, n, n), dtype=np.float64)
        c0 = n / 2 + rng.uniform(-2, 2, 3)
        r2 = (z - c0[0]) ** 2 + (y - c0[1]) ** 2 + (x - c0[2]) ** 2
        grid.set("phi", (r2 <= case["radius"] ** 2).astype(np.int32))
        grid.set("c", 0.02 + 1e-4 * rng.standard_normal((n, n, n)))
        grid.set("T", 893.0)
        grid.step_graph(2 * SETTLE + 1)
        s.load = {k: _pinned(grid.get(k)) for k in ("phi", "alpha", "c")}
    elif kind == "sweep":
        # instances first, first + 1, ... of the generator, each with its own noise in the composition
        s.grids = []
        for k in range(case["instances"]):
            grid, inst = sweep.lamellar_grid(case["first"] + k)
            grid.set("c", inst["c"] + np.random.default_rng([seed, 6, k]).normal(0.0, 1e-3, inst["c"].shape))
            s.grids.append(grid)
        s.batch = gpk.GPKBatch(s.grids)
        s.batch.step_graph(3)
        s.stream = torch.cuda.ExternalStream(s.batch.graph_stream_ptr())
        # the sweep has no region identity, so its state can be set on the device
        s.state = {k: [_view(g, k) for g in s.grids] for k in ("phi", "alpha", "c")}
        s.load = {k: [t.clone() for t in v] for k, v in s.state.items()}
    elif kind == "elastic":
        s.fractions = _elastic_fractions(case, seed)
        s.solver = gpk.SpectralElasticity(_elastic_shape(case), 1.0, **CUBIC, eig=variant_eigenstrains(0.004, -0.011))
    elif kind == "calibrate":
        phi, g, mob, s.theta = _calibration(case, seed)
        s.grid = gpk.GPKGrid(1, case["n"], case["n"], 1.0, gpk.thermo.isotropic(1.0, 1.0), 0.0, 1.5, precision="f64")
        s.grid.set("phi", phi)
        s.grid.set("g", g)
        s.problem = gpk.AdjointProblem(s.grid, mob, case["grains"], **CALIBRATE)
        s.problem.set_target(s.problem.forward(1.05 * s.theta, want_v=True)[1])
    else:
        rng = np.random.default_rng([seed, 5])
        lab = _plates(case, rng)
        f0 = float(np.mean(lab > 0))
        ctot = np.where(lab > 0, 1.0 / 3.0, (0.0169 - f0 / 3.0) / (1.0 - f0))
        ctot = np.where(lab > 0, ctot, np.abs(ctot) * (1.0 + 0.05 * rng.standard_normal(lab.shape)))
        s.labels, s.alpha = torch.from_numpy(lab).cuda(), torch.from_numpy(rng.uniform(0.05, 1.0, lab.shape)).cuda()
        s.ctot = torch.from_numpy(ctot).cuda()
        s.cross = torch.from_numpy(rng.random(lab.shape) < 0.1).cuda()
        s.growth = torch.from_numpy(rng.uniform(0.0, 0.02, lab.shape)).cuda()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s.kind
    if kind in ("growth", "solidify"):
        for name, value in s.load.items():
            s.grid.set(name, value)
        if kind == "growth":
            s.grid.step_n(s.case["steps"])
            names = ("phi", "alpha", "g", "phi_comp", "mask", "nx_f", "ny_f", "nz_f", "kappa_f", "vn_f")
        else:
            s.grid.step_graph(s.case["steps"])
            names = ("phi", "alpha", "c", "kappa_f", "vn_f")
        return {k: _view(s.grid, k) for k in names}
    if kind == "geometry":
        s.grid.geometry()
        return {k: _view(s.grid, k) for k in ("mask", "phi_comp", "nx_f", "ny_f", "nz_f", "kappa_f")}
    if kind == "sweep":
        with torch.cuda.stream(s.stream):
            for k, v in s.state.items():
                torch._foreach_copy_(v, s.load[k])
        s.batch.step_graph(s.case["steps"])
        with torch.cuda.stream(s.stream):
            return {k: torch.cat([t.reshape(-1) for t in v]) for k, v in s.state.items()}
    if kind == "elastic":
        driving, energy, hydrostatic, _ = s.solver.solve(s.fractions, want_residual=False)
        return {"driving": driving, "energy": energy, "hydrostatic": hydrostatic}
    if kind == "calibrate":
        loss, gradient = s.problem.gradient(s.theta)
        return {"loss": loss, "gradient": gradient}
    # one step of the Al-Cu chain
    labels, alpha = s.labels.clone(), s.alpha.clone()
    mask, competitor = alcu.neighbor_competitor(labels)
    fraction = alcu.precip_fraction(labels, alpha, competitor)
    cm = alcu.matrix_composition(s.ctot, fraction, ALCU)
    trace = alcu.interface_matrix_composition(cm, fraction, ALCU)
    ctot, _, _ = alcu.diffuse_conservative_subcycled(s.ctot, fraction, ALCU, ALCU_DT)
    alcu.conservative_partition_transfer(ctot, fraction, fraction + s.growth * mask, trace, ALCU)
    deferred = alcu.commit_topology_transactions(labels, alpha, competitor, s.cross & mask)
    changed = alcu.conservative_gaussian_remap(labels, alpha, ALCU_REMAP_SIGMA)
    return {"labels": labels, "alpha": alpha, "ctot": ctot, "trace": trace, "fraction": fraction,
            "deferred": deferred, "changed": changed}


# ---------------------------------------------------------------------------
# bytes and operations a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("growth", "geometry"):
        n = case["nz"] * case["ny"] * case["nx"]
        d = 3 if case["nz"] > 1 else 2
        r = 4 if case["precision"] == "f32" else 8
        # interface cells: two layers of each grain's boundary
        per = n / case["grains"]
        iface = n * min(1.0, (4.84 * per ** (-1 / 3) if d == 3 else 3.55 * per ** -0.5))
        width = 2 * math.ceil(3.5 * case["sigma"]) + 1
        # smoothing of the own label's indicator along each axis and the differences, per interface cell
        flops = iface * (2 * d * width + 120)
        if kind == "geometry":
            return {"bytes": n * (4 + 1) + iface * (4 + (d + 1) * r), "flops": flops}
        # labels, alpha and orientation read and written, the interface fields written
        step = n * (2 * (4 + 2 * r) + 1) + iface * (4 + (d + 2) * r)
        return {"bytes": case["steps"] * step, "flops": case["steps"] * flops}
    if kind == "solidify":
        n = case["n"] ** 3
        # labels, alpha and composition read and written, the solid fraction kept between
        return {"bytes": case["steps"] * n * (2 * (4 + 8 + 8) + 8), "flops": case["steps"] * n * 30}
    if kind == "sweep":
        n = case["instances"] * 97000  # mean cells of sides U[64, 512]
        return {"bytes": case["steps"] * n * 2 * (4 + 8 + 8), "flops": case["steps"] * n * 20}
    if kind == "elastic":
        n = math.prod(_elastic_shape(case))
        return {"bytes": n * (24 + 40), "flops": n * (9 * 2.5 * math.log2(n) + 150)}
    if kind == "calibrate":
        n = case["n"] ** 2
        return {"bytes": n * (4 + 4 + 8 * 4), "flops": n * (12 * 2.5 * math.log2(n) + 200)}
    n = case["n0"] * case["n1"] * case["n2"]
    # labels 1 B and alpha, ctot, growth read, labels, alpha, ctot, trace, fraction written
    return {"bytes": n * (1 + 24 + 1 + 1 + 32), "flops": n * 300}


# ---------------------------------------------------------------------------
# the same results in 64 bits with torch alone
# ---------------------------------------------------------------------------
def _taps(sigma):
    """Gaussian of radius ceil(3.5 sigma) and its fourth-order first and second differences."""
    s = max(sigma, 0.5)
    r = math.ceil(3.5 * s)
    g = np.exp(-np.arange(-r, r + 1) ** 2 / (2.0 * s * s))
    g = np.pad(g / g.sum(), 2)
    d1, d2 = np.array([-1.0, 8.0, 0.0, -8.0, 1.0]) / 12.0, np.array([-1.0, 16.0, -30.0, 16.0, -1.0]) / 12.0
    return r + 2, [g, -np.convolve(g, d1, "same"), np.convolve(g, d2, "same")]


def _exact_geometry(phi, sigma):
    """Mask, competitor, normals and curvature of int labels (Nz, Ny, Nx) on the GPU, dx = 1."""
    nz, ny, nx = phi.shape
    is3d = nz > 1
    offs = [(0, 0, -1), (0, 0, 1), (0, -1, 0), (0, 1, 0)] + ([(-1, 0, 0), (1, 0, 0)] if is3d else [])
    mask = torch.zeros_like(phi, dtype=torch.bool)
    for a, b, c in offs:
        mask |= torch.roll(phi, (-a, -b, -c), (0, 1, 2)) != phi
    z, y, x = torch.nonzero(mask, as_tuple=True)
    own, flat = phi[z, y, x], phi.reshape(-1)

    def at(dz, dy, dx):
        return flat[(((z + dz) % nz) * ny + (y + dy) % ny) * nx + (x + dx) % nx]

    rad, w = _taps(sigma)
    w = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in w]
    acc = torch.zeros((3, 3, 3, z.numel()), dtype=torch.float64, device="cuda")  # derivative orders in z, y, x
    wx = torch.stack(w)
    span = torch.arange(-rad, rad + 1, device="cuda")
    orders = [(a, b, c) for a in range(3) for b in range(3) for c in range(3) if 0 < a + b + c <= 2]
    for dz in range(-rad, rad + 1) if is3d else (0,):
        for dy in range(-rad, rad + 1):
            row = flat[((((z + dz) % nz) * ny + (y + dy) % ny) * nx)[:, None] + (x[:, None] + span) % nx]
            sx = wx @ (row == own[:, None]).double().T  # (3, cells)
            for a, b, c in orders:
                if is3d or a == 0:
                    acc[a, b, c] += sx[c] * (w[b][dy + rad] * (w[a][dz + rad] if is3d else 1.0))
    ix, iy, iz = acc[0, 0, 1], acc[0, 1, 0], acc[1, 0, 0]
    ixx, iyy, izz = acc[0, 0, 2], acc[0, 2, 0], acc[2, 0, 0]
    ixy, ixz, iyz = acc[0, 1, 1], acc[1, 0, 1], acc[1, 1, 0]
    g2 = ix * ix + iy * iy + iz * iz
    ok = g2 > 1e-8
    grad = torch.sqrt(torch.where(ok, g2, torch.ones_like(g2)))
    n = [torch.where(ok, -v / grad, torch.zeros_like(v)) for v in (ix, iy, iz)]
    ghg = ix * ix * ixx + iy * iy * iyy + iz * iz * izz + 2 * (ix * iy * ixy + ix * iz * ixz + iy * iz * iyz)
    k = (ghg - g2 * (ixx + iyy + izz)) / (grad ** 3)
    k = torch.where(ok & (k.abs() >= 1e-6), k, torch.zeros_like(k)).clamp(-1.0 / sigma, 1.0 / sigma)
    # competitor: the unlike face neighbour with the most support around the cell, then the best aligned
    score = [-n[0], n[0], -n[1], n[1], -n[2], n[2]]
    comp, best, best_s = own.clone(), torch.full_like(own, -1), torch.full_like(k, -2.0)
    around = [(a, b, c) for a in ((-1, 0, 1) if is3d else (0,)) for b in (-1, 0, 1) for c in (-1, 0, 1) if a or b or c]
    for f, o in enumerate(offs):
        q = at(*o)
        sup = sum((at(*v) == q).to(own.dtype) for v in around)
        take = (q != own) & ((sup > best) | ((sup == best) & (score[f] > best_s)))
        comp, best, best_s = torch.where(take, q, comp), torch.where(take, sup, best), torch.where(take, score[f], best_s)

    def full(v, fill=None):
        out = torch.zeros(phi.shape, dtype=v.dtype, device="cuda") if fill is None else fill.clone()
        out[z, y, x] = v
        return out
    return {"mask": mask, "phi_comp": full(comp, phi), "nx_f": full(n[0]), "ny_f": full(n[1]), "nz_f": full(n[2]),
            "kappa_f": full(k)}


def _exact_elastic(f):
    shape, nd = f.shape[1:], f.dim() - 1
    c11, c12, c44 = CUBIC["c11"], CUBIC["c12"], CUBIC["c44"]
    eig = torch.from_numpy(variant_eigenstrains(0.004, -0.011)).cuda()
    es = torch.einsum("vj,v...->j...", eig, f)
    k = torch.meshgrid(*[2 * math.pi * torch.fft.fftfreq(n, dtype=torch.float64, device="cuda") for n in shape],
                       indexing="ij")
    k = list(k) + [torch.zeros(shape, dtype=torch.float64, device="cuda")] * (3 - nd)
    eh = [torch.fft.fftn(e.to(torch.complex128)) for e in es]
    k2, mean = k[0] ** 2 + k[1] ** 2 + k[2] ** 2, (0,) * nd
    a = torch.zeros(tuple(shape) + (3, 3), dtype=torch.float64, device="cuda")
    for i in range(3):
        for j in range(3):
            a[..., i, j] = c44 * k2 + (c11 - c44) * k[i] ** 2 if i == j else (c12 + c44) * k[i] * k[j]
    a[mean] = torch.eye(3, dtype=torch.float64, device="cuda")
    tr = eh[0] + eh[1] + eh[2]
    b = torch.stack([k[i] * ((c11 - c12) * eh[i] + c12 * tr) for i in range(3)], -1)
    b[mean] = 0
    u = torch.linalg.solve(a.to(torch.complex128), b[..., None])[..., 0]
    pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
    de = []
    for m, (i, j) in enumerate(pairs):
        e = 0.5 * (k[i] * u[..., j] + k[j] * u[..., i])
        if m < 3:
            e[mean] = eh[m][mean]
        e = torch.fft.ifftn(e).real
        de.append(e - es[m] if m < 3 else e)
    t = de[0] + de[1] + de[2]
    sig = [(c11 - c12) * de[m] + c12 * t if m < 3 else 2 * c44 * de[m] for m in range(6)]
    energy = 0.5 * sum(sig[m] * de[m] * (1 if m < 3 else 2) for m in range(6))
    return {"driving": torch.stack([-sum(eig[v, m] * sig[m] for m in range(3)) for v in range(3)]),
            "energy": energy, "hydrostatic": (sig[0] + sig[1] + sig[2]) / 3}


def _calibration_forward(phi, geo, g, mob, theta):
    """Interface velocities and summed elastic energy of the calibration model (differentiable in theta)."""
    n = phi.shape[0]
    c11, c12, c44 = CALIBRATE["c11"], CALIBRATE["c12"], CALIBRATE["c44"]
    q = 2 * math.pi * torch.fft.fftfreq(n, dtype=torch.float64, device="cuda")
    ky, kx = q[:, None].expand(n, n), q[None, :].expand(n, n)
    eta = (mob[phi.long()] < 0).double()
    es = [eta * theta[m] for m in range(3)]
    h = [torch.fft.fft2(e.to(torch.complex128)) for e in es]
    bx = kx * (c11 * h[0] + c12 * h[1]) + ky * 2 * c44 * h[2]
    by = kx * 2 * c44 * h[2] + ky * (c12 * h[0] + c11 * h[1])
    a00, a11, a01 = c11 * kx ** 2 + c44 * ky ** 2, c44 * kx ** 2 + c11 * ky ** 2, (c12 + c44) * kx * ky
    origin = (kx == 0) & (ky == 0)
    det = torch.where(origin, torch.ones_like(kx), a00 * a11 - a01 * a01)
    u0, u1 = (a11 * bx - a01 * by) / det, (a00 * by - a01 * bx) / det
    s = [torch.where(origin, h[0], kx * u0), torch.where(origin, h[1], ky * u1),
         torch.where(origin, torch.zeros_like(h[2]), 0.5 * (kx * u1 + ky * u0))]
    d = [torch.fft.ifft2(s[m]).real - es[m] for m in range(3)]
    en = 0.5 * ((c11 * d[0] + c12 * d[1]) * d[0] + (c12 * d[0] + c11 * d[1]) * d[1] + 4 * c44 * d[2] * d[2])
    y, x = torch.nonzero(geo["mask"][0], as_tuple=True)
    own, comp = phi[y, x], geo["phi_comp"][0][y, x]
    e0 = en[y, x]
    de, found = torch.zeros_like(e0), own == comp
    for dy, dx in ((0, -1), (0, 1), (-1, 0), (1, 0)):
        yy, xx = (y + dy) % n, (x + dx) % n
        hit = ~found & (phi[yy, xx] == comp)
        de, found = torch.where(hit, en[yy, xx] - e0, de), found | hit
    nx_, ny_, kap, ang = (v[0][y, x] for v in (geo["nx_f"], geo["ny_f"], geo["kappa_f"], g))
    cg, sg = torch.cos(ang), torch.sin(ang)
    th = torch.atan2(-nx_ * sg + ny_ * cg, nx_ * cg + ny_ * sg)
    sa = CALIBRATE["sigma0"] * (1 + sum(theta[3 + m] * torch.cos(4 * (m + 1) * th) for m in range(4)))
    p = mob[own.long()].long()
    m_of = torch.where(p >= 0, theta[7:][p.clamp(min=0)], torch.full_like(e0, CALIBRATE["m_fixed"]))
    vr = m_of * (de - sa * kap)
    lo, hi = torch.minimum(own, comp).long(), torch.maximum(own, comp).long()
    pair = torch.where(own == comp, torch.full_like(lo, -1), lo * (1 << 20) + hi)
    sign = torch.where(own.long() == lo, 1.0, -1.0).double()
    slot = torch.full((n, n), -1, dtype=torch.long, device="cuda")
    slot[y, x] = torch.arange(y.numel(), device="cuda")
    num, den = torch.zeros_like(vr), torch.zeros_like(vr)
    for dy in range(-3, 4):
        for dx in range(-3, 4):
            j = slot[(y + dy) % n, (x + dx) % n]
            same = (j >= 0) & (pair[j] == pair) & (pair >= 0)
            wgt = math.exp(-(dy * dy + dx * dx) * 0.5 / 0.85 ** 2) * same.double()
            num, den = num + wgt * (sign * vr)[j], den + wgt
    v = torch.where(pair >= 0, sign * num / torch.where(den > 0, den, torch.ones_like(den)), vr)
    return v, en.sum()


def _exact_calibrate(case, seed):
    phi, g, mob, theta = _calibration(case, seed)
    phi, g = torch.from_numpy(phi).cuda(), torch.from_numpy(np.asarray(g, np.float64)).cuda()
    geo = _exact_geometry(phi, 1.5)
    # competitors are whole numbers; where two are equally good up to rounding, the grid's choice stands
    s = prepare(case, seed)
    geo["phi_comp"] = torch.from_numpy(s.grid.get("phi_comp")).cuda()
    mob = torch.from_numpy(mob).cuda()
    t = torch.from_numpy(theta).cuda()
    target, _ = _calibration_forward(phi[0], geo, g, mob, 1.05 * t)
    t.requires_grad_(True)
    v, energy = _calibration_forward(phi[0], geo, g, mob, t)
    loss = 0.5 * ((v - target) ** 2).sum() + CALIBRATE["energy_weight"] * energy
    loss.backward()
    return {"loss": float(loss.detach()), "gradient": t.grad.cpu().numpy()}


def _smooth(a, sigma):
    r = int(4.0 * sigma + 0.5)
    w = np.exp(-0.5 / sigma ** 2 * np.arange(-r, r + 1) ** 2)
    w = w / w.sum()
    for axis in range(a.dim()):
        a = sum(float(w[j + r]) * torch.roll(a, j, axis) for j in range(-r, r + 1))
    return a


def _exact_alcu(s):
    p, sigma = ALCU, ALCU.composition_extension_sigma_cells
    lab, alpha = s.labels, s.alpha
    # the competitor is whole numbers, its own output: taken from the step
    mask, comp = alcu.neighbor_competitor(lab)
    frac = torch.where(lab > 0, alpha, torch.where(comp > 0, 1.0 - alpha, torch.zeros_like(alpha))).clamp(0.0, 1.0)

    def lever(c):
        m = (1.0 - frac).clamp(min=1e-8)
        cm = torch.where(m > 1e-7, (c - frac * p.c_theta) / m, torch.full_like(c, p.c_matrix_eq))
        return cm.clamp(0.0, p.c_theta), m

    cm, m = lever(s.ctot)
    mf = (1.0 - frac).clamp(0.0, 1.0)
    trace = (_smooth(cm * mf, sigma) / _smooth(mf, sigma).clamp(min=1e-12)).clamp(0.0, p.c_theta)
    n = max(1, math.ceil(ALCU_DT / (0.4 * p.dx * p.dx / (2.0 * lab.dim() * p.diffusivity))))
    c = s.ctot.clone()
    for _ in range(n):
        cm, m = lever(c)
        dc = torch.zeros_like(c)
        for axis in range(c.dim()):
            face = 0.5 * (m + torch.roll(m, -1, axis))
            flux = -p.diffusivity * face * (torch.roll(cm, -1, axis) - cm) / p.dx
            dc -= (flux - torch.roll(flux, 1, axis)) / p.dx
        c = c + ALCU_DT / n * dc
    new = frac + s.growth * mask
    transfer = (new.clamp(0.0, 1.0) - frac) * (p.c_theta - trace)
    total = transfer.sum()
    c = c + transfer
    matrix = (1.0 - new).clamp(0.0, 1.0)
    weight = _smooth(transfer.abs(), sigma) * matrix
    if -total < 0.0:
        weight = weight * (c - p.c_matrix_eq * matrix).clamp(min=0.0)
    c = c - total * weight / weight.sum()
    return {"labels": None, "alpha": None, "ctot": c, "trace": trace, "fraction": frac, "deferred": None,
            "changed": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "geometry":
        s = prepare(case, seed)
        e = _exact_geometry(torch.from_numpy(s.grid.get("phi")).cuda(), case["sigma"])
        return {k: (None if k in ("mask", "phi_comp") else v) for k, v in e.items()}
    if kind == "elastic":
        return _exact_elastic(_elastic_fractions(case, seed))
    if kind == "calibrate":
        return _exact_calibrate(case, seed)
    if kind == "alcu":
        return _exact_alcu(prepare(case, seed))
    return None  # a step's labels are decisions; what follows them has no value of its own in 64 bits
