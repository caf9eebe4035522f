"""The launch counter against the launches that the profiler records."""
import numpy as np
import pytest

from gpk_b200 import GPKGrid, sweep, thermo, voronoi

pytestmark = pytest.mark.gpu


def _profiled(call):
    """Kernels of this library that `call` launches (not the radix sorts'; copies and memsets are no kernels)."""
    torch = pytest.importorskip("torch")
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA, ProfilerActivity.CPU]) as p:
        call()
        torch.cuda.synchronize()
    names = [e.name for e in p.events() if e.device_type.name == "CUDA"]
    if not names:
        pytest.skip("the profiler records no kernels here")
    return [n for n in names if "gpk_dev::" in n and "cub::" not in n]


def _check(g, call, least):
    call()  # (what is made once)
    before = g.launch_count()
    names = _profiled(call)
    assert len(names) >= least
    assert g.launch_count() - before == len(names), sorted(names)
    g.close()


@pytest.mark.parametrize("shape,grains,sigma,precision,kind", [
    ((1, 96, 96), 12, 1.5, "f32", "tiled"), ((1, 400, 400), 900, 1.5, "f32", "tiled"),
    ((64, 72, 80), 200, 1.5, "f32", "tiled"), ((64, 72, 80), 200, 1.5, "f64", "tiled"),
    ((40, 44, 48), 30, 1.5, "f32", "per_cell"), ((40, 44, 48), 30, 1.5, "f64", "separable_tiles"),
    ((40, 44, 48), 12, 5.0, "f32", "tiled"), ((40, 44, 48), 6, 9.0, "f32", "tiled")])
def test_growth(shape, grains, sigma, precision, kind):
    phi, o = voronoi(*shape, grains, 3)
    g = GPKGrid(*shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, sigma, precision=precision)
    g.set_geometry_kernel(kind)
    g.set("phi", phi)
    g.set("g", o)
    g.set("alpha", 0.5)
    _check(g, lambda: g.step_n(9), 60)  # (9 steps: one with the extinction)


def test_solidification_with_transport():
    n = 48
    th = thermo.solidification(M0=5e-8, sigma0=0.2, eps4=0.04, m_liq=-500.0, k_part=0.14, T_melt=933.0, L=1e8)
    th.solute_rejection, th.k_partition = True, 0.14
    g = GPKGrid(n, n, n, 0.5e-6, th, 3e-9, 1.5, precision="f64")
    z, y, x = np.indices((n, n, n)) - n // 2
    g.set("phi", ((x * x + y * y + z * z) <= 36).astype(np.int32))
    g.set("c", 0.02)
    g.set("T", 893.0)
    _check(g, lambda: g.step_n(6), 60)


@pytest.mark.parametrize("call", ["step_n", "step_graph"])
def test_lamellar(call):
    g = sweep.lamellar_grid(5000)[0]
    g.step_n(1)
    _check(g, lambda: getattr(g, call)(6), 48)


@pytest.mark.parametrize("precision,real", [("f32", "float"), ("f64", "double")])
@pytest.mark.parametrize("sigma,radius", [(1.5, 3), (3.0, 4), (4.0, 5), (5.0, 6), (6.0, 7), (7.0, 8), (8.0, 9)])
def test_projection_on_bitmaps(sigma, radius, precision, real):
    """Every projection radius runs on pair bitmaps, in both precisions."""
    g = GPKGrid(30, 34, 41, 1.0, thermo.isotropic(1.0, 1.0), 0.0, sigma, precision=precision)
    g.set("phi", voronoi(30, 34, 41, 14, 8)[0])
    g.set("alpha", 1.0)
    names = [n for n in _profiled(g.step) if "k_projection" in n]
    assert len(names) == 1 and f"k_projection_bits<{real}, true, {radius}>" in names[0], names
    g.close()
