"""The remap's screening by core rows against the per-cell kernel, bit for bit:
fields whose cells the bound settles, cannot settle (thin and one-cell grains:
the resident label holds less than half of its box) and settles only for one
candidate (many labels around a cell: no leader among the candidates).
"""
import numpy as np
import pytest

from _cases import bits_equal
from gpk_b200 import GPKGrid, thermo

pytestmark = pytest.mark.gpu


def _fields(kind, phi, sigma, precision):
    grid = GPKGrid(*phi.shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, sigma, precision=precision)
    grid.set_geometry_kernel(kind)
    grid.set("phi", phi)
    grid.set("alpha", 1.0)
    for _ in range(3):
        grid.step(1e-3)
    return {f: grid.get(f) for f in ("phi", "phi_comp", "alpha", "vn_f")}


def _phi(kind, shape, rng):
    z, y, x = np.indices(shape)
    if kind == "flat":
        return (x // 12).astype(np.int32)
    if kind == "layers":  # one to three cells thick
        return ((2 * x + y) // 4 % 9).astype(np.int32)
    if kind == "corners":  # every interface cell within two cells of a junction
        return (x // 4 % 3 + 3 * (y // 4 % 3) + 9 * (z // 4 % 3)).astype(np.int32)
    if kind == "specks":
        phi = (x // 10).astype(np.int32)
        spots = rng.random(shape) < 0.02
        phi[spots] = 50 + rng.integers(0, 5, int(spots.sum()))
        return phi
    return rng.integers(0, 3, size=shape).astype(np.int32)  # noise: few labels, no box half its own


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("shape", [(20, 23, 53), (1, 70, 60)])
@pytest.mark.parametrize("kind", ["flat", "layers", "corners", "specks", "noise"])
def test_core_screening(kind, shape, precision):
    phi = _phi(kind, shape, np.random.default_rng(11))
    a, b = (_fields(k, phi, 1.5, precision) for k in ("tiled", "per_cell"))
    for f in a:
        assert bits_equal(a[f], b[f]), f
