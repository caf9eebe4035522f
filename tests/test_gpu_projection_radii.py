"""The pair projection on bitmaps at every radius against the per-cell kernel,
bit for bit (both add the same weights in the same order), with few pairs per
tile, with more than a tile's slots hold, and with velocities that are not
finite on some pairs only.
"""
import numpy as np
import pytest

from _cases import bits_equal
from gpk_b200 import GPKGrid, thermo

pytestmark = pytest.mark.gpu


def _fields(kind, phi, sigma, precision, g=None):
    grid = GPKGrid(*phi.shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, sigma, precision=precision)
    grid.set_geometry_kernel(kind)
    grid.set("phi", phi)
    grid.set("alpha", 1.0)
    if g is not None:
        grid.set("E_el", g)
        grid.set_external_elastic(True)
    grid.step(1e-3)
    return {f: grid.get(f) for f in ("vn_f", "kappa_f", "alpha", "phi")}


def _same(phi, sigma, precision, g=None):
    a, b = (_fields(k, phi, sigma, precision, g) for k in ("tiled", "per_cell"))
    for f in a:
        assert bits_equal(a[f], b[f]), f
    return a


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("sigma", [1.5, 3.0, 4.0, 5.0, 6.0, 7.0, 8.0])  # projection radii 3 to 9
def test_every_radius(oracle_mod, sigma, precision):
    phi = oracle_mod.voronoi(30, 34, 41, 14, 8)[0]
    _same(phi, sigma, precision)


@pytest.mark.parametrize("sigma", [1.5, 3.0])
def test_more_pairs_than_slots(sigma):
    phi = np.random.default_rng(4).integers(0, 40, size=(20, 24, 36)).astype(np.int32)
    _same(phi, sigma, "f32")


@pytest.mark.parametrize("shape", [(24, 20, 40), (1, 40, 60)])
def test_velocities_that_are_not_finite(oracle_mod, shape):
    """An infinite elastic energy on one grain makes the velocities of its
    pairs infinite or NaN; every other pair keeps finite ones."""
    phi = oracle_mod.voronoi(*shape, 9, 3)[0]
    e = np.zeros(shape, dtype=np.float32)
    e[phi == 4] = np.inf
    v = _same(phi, 1.5, "f32", e)["vn_f"]
    assert not np.all(np.isfinite(v)) and np.any(np.isfinite(v) & (v != 0))
