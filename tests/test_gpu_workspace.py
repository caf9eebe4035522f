"""The geometry's workspace comes with the grid: no step, geometry call or
capture of any kernel kind or kernel width adds device memory, and what the geometry leaves in
the shared scratch changes no later step.
"""
import numpy as np
import pytest

from gpk_b200 import GPKGrid, sweep, thermo, voronoi

pytestmark = pytest.mark.gpu
KINDS = ("tiled", "per_cell", "tiled_batched", "tiled_exact_scores")


@pytest.mark.parametrize("precision,per_cell", [("f32", 200), ("f64", 273)])
@pytest.mark.parametrize("shape", [(64, 72, 80), (1, 500, 600)])
def test_no_memory_at_the_first_step(shape, precision, per_cell):
    for kind in KINDS + (("separable_tiles",) if precision == "f64" and shape[0] > 1 else ()):
        g = GPKGrid(*shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, 1.5, precision=precision)
        g.set_geometry_kernel(kind)
        made = g.device_bytes()
        assert made < per_cell * np.prod(shape) + (2 << 20), kind
        g.voronoi(40, 3)
        g.set("alpha", 1.0)
        held = g.device_bytes()
        g.geometry()
        g.step_n(2)
        assert g.device_bytes() == held, kind
        g.close()


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("sigma,labels", [(5.0, 12), (9.0, 12), (5.0, 20000)])  # boxes; radius 32 and many labels: whole grid
def test_no_memory_at_the_first_separable_step(sigma, labels, precision):
    shape = (40, 44, 48)
    g = GPKGrid(*shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, sigma, precision=precision)
    # bytes a cell, and twelve products for every tap of the direct form's table
    cell, real = (200, 4) if precision == "f32" else (273, 8)
    taps = (2 * (int(np.ceil(3.5 * sigma)) + 2) + 1) ** 3
    assert g.device_bytes() < cell * np.prod(shape) + 12 * real * taps + (2 << 20)
    phi = voronoi(*shape, 12, 3)[0]
    g.set("phi", np.where(phi == 12, labels, phi).astype(np.int32))
    g.set("alpha", 0.3)
    held = g.device_bytes()
    g.geometry()
    g.step_n(2)
    assert g.device_bytes() == held
    g.close()


def test_no_memory_at_a_capture():
    g = sweep.lamellar_grid(5000)[0]
    g.step_n(1)
    held = g.device_bytes()
    g.step_graph(4)
    assert g.device_bytes() == held
    g.close()


@pytest.mark.parametrize("shape", [(30, 34, 41), (1, 90, 110)])
def test_geometry_between_steps_changes_nothing(oracle_mod, shape):
    phi, o = oracle_mod.voronoi(*shape, 20, 8)
    out = []
    for extra in (False, True):
        g = GPKGrid(*shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, 1.5)
        g.set("phi", phi)
        g.set("g", o)
        g.set("alpha", 0.3)
        for _ in range(10):
            if extra:
                g.geometry()
            g.step()
            if extra:
                g.geometry()
                g.topology_simple_move(7, int(phi.ravel()[0]))
        out.append({f: g.get(f) for f in ("phi", "alpha", "g")})
        g.close()
    for f in out[0]:
        assert np.array_equal(out[0][f], out[1][f]), f
