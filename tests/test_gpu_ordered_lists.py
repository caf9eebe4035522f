"""The interface list and the candidate list, each made in one launch.

Positions in the lists order the crossing sweep, so a step's labels and every
other public field equal the oracle's bit for bit only if the lists are in
increasing cell order.  Sizes: one cell tile, a partial last tile, both tile
sizes (they change at 2^22 cells), rows that are and are not a multiple of
four cells, empty lists.
"""
import numpy as np
import pytest

from _cases import compare_all
from gpk_b200 import GPKGrid, thermo

pytestmark = pytest.mark.gpu


def _run(oracle_mod, phi, sigma, steps, precision="f32"):
    iso = thermo.isotropic(1.0, 1.0)
    gpu = GPKGrid(*phi.shape, 1.0, iso, 0.0, sigma, precision=precision)
    ora = oracle_mod.OracleGrid(*phi.shape, 1.0, iso, 0.0, sigma, precision=precision)
    alpha = np.random.default_rng(1).uniform(0.01, 1.0, phi.shape)
    for g in (gpu, ora):
        g.set("phi", phi)
        g.set("alpha", alpha.astype(np.float32))
    for s in range(steps):
        assert gpu.step() == ora.step(), s
        assert not compare_all(gpu, ora), s
    return gpu


@pytest.mark.parametrize("shape", [(1, 4, 4), (1, 33, 64), (1, 45, 47), (9, 16, 16), (13, 14, 15), (16, 32, 64)])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_small_lists(oracle_mod, shape, precision):
    phi = np.random.default_rng(sum(shape)).integers(0, 6, size=shape).astype(np.int32)
    _run(oracle_mod, phi, 0.5, 3, precision)


@pytest.mark.parametrize("shape", [(1, 2048, 2052), (1, 2049, 2051)])
def test_large_tiles(oracle_mod, shape):
    """Above 2^22 cells, with rows of whole and of partial int4 groups."""
    phi = oracle_mod.voronoi(*shape, 9000, 5)[0]
    _run(oracle_mod, phi, 0.5, 2)


def test_empty_lists(oracle_mod):
    g = _run(oracle_mod, np.full((1, 40, 44), 3, dtype=np.int32), 1.5, 2)
    assert g.interface_fraction() == 0.0


def test_lists_again_after_other_grids(oracle_mod):
    """The lists' tickets start again for every launch, whatever ran between."""
    phi = oracle_mod.voronoi(1, 64, 60, 20, 2)[0]
    for _ in range(3):
        _run(oracle_mod, phi, 1.5, 2)
