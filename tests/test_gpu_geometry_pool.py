"""The pool of the geometry's label bitmaps.

Tiles that ask for very different shares of a pool too small for all of them:
every repetition equals the per-cell kernel, bit for bit, and the tiles without
bitmaps are counted.  A polycrystal of small grains finds room at every radius.
"""
import numpy as np
import pytest

from _cases import bits_equal
from gpk_b200 import GPKGrid, thermo

pytestmark = pytest.mark.gpu
FIELDS = ("phi_comp", "nx_f", "ny_f", "nz_f", "kappa_f")


def uneven_labels(shape, seed):
    """Blocks of 12 x 16 x 16 cells, each with labels of its own: 2 to 1500 of them."""
    rng = np.random.default_rng(seed)
    phi = np.zeros(shape, dtype=np.int32)
    base = 0
    for z in range(0, shape[0], 12):
        for y in range(0, shape[1], 16):
            for x in range(0, shape[2], 16):
                k = int(round(2 * 750 ** rng.random()))
                b = phi[z:z + 12, y:y + 16, x:x + 16]
                b[...] = base + rng.integers(0, k, size=b.shape)
                base += k
    return phi


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("sigma", [1.5, 2.0])
def test_uneven_requests(sigma, precision):
    phi = uneven_labels((84, 96, 110), 5)
    ref = None
    for kind in ("per_cell", "tiled"):
        g = GPKGrid(*phi.shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, sigma, precision=precision)
        g.set_geometry_kernel(kind)
        g.set("phi", phi)
        for rep in range(1 if ref is None else 12):
            g.geometry()
            got = {f: g.get(f) for f in FIELDS}
            ref = ref or got
            for f in FIELDS:
                assert bits_equal(ref[f], got[f]), (kind, rep, f)
            st = g.geometry_stats()
            assert st["words"] <= st["pool_words"] and (st["tiles_without_bitmaps"] > 0) == (kind == "tiled"), st
            assert (st["items"] > 0) == (kind == "tiled"), st
        g.close()


@pytest.mark.parametrize("sigma,cells", [(1.5, 1500), (2.0, 1500), (2.2, 1500)])  # radii 8, 9, 10
def test_small_grains_find_room(sigma, cells):
    """2.4 M cells in grains of 1500: 9 to 11 labels a tile, 4.4 to 6.6 words a cell."""
    shape = (128, 136, 136)
    g = GPKGrid(*shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, sigma)
    g.voronoi(int(np.prod(shape)) // cells, 7)
    g.geometry()
    st = g.geometry_stats()
    assert st["tiles_without_bitmaps"] == 0 and st["words"] > 2 * np.prod(shape), st
    g.set_geometry_kernel("tiled_batched")  # no pool: every tile with interface cells is counted
    g.geometry()
    assert g.geometry_stats()["tiles_without_bitmaps"] > 0
    g.close()
