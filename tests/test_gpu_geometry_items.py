"""The item-based direct geometry against the per-cell kernel, bit for bit.

Both add the same products in the same order, so every field is equal to the
last bit.  The sizes sit where the item kernels change form: grids smaller
than a tile or a kernel radius, every radius, few items (three warps an item
half), half items, whole items, and labels so many that some tiles find the
bitmap pool full.
"""
import numpy as np
import pytest

from _cases import bits_equal
from gpk_b200 import GPKGrid, thermo

pytestmark = pytest.mark.gpu
FIELDS = ("mask", "phi_comp", "nx_f", "ny_f", "nz_f", "kappa_f")


def _agree(phi, sigma, precision, kinds=("tiled", "per_cell")):
    out = []
    for kind in kinds:
        g = GPKGrid(*phi.shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, sigma, precision=precision)
        g.set_geometry_kernel(kind)
        g.set("phi", phi)
        g.geometry()
        g.geometry()  # the items' counters start again
        out.append({f: g.get(f) for f in FIELDS})
        g.close()
    for f in FIELDS:
        assert bits_equal(out[0][f], out[1][f]), f
    return int(out[0]["mask"].sum())


def _blocks(shape, edge, seed):
    """Random labels on blocks of `edge` cells, jittered by a label-free shear."""
    rng = np.random.default_rng(seed)
    z, y, x = np.indices(shape)
    s = [(e + edge - 1) // edge + 1 for e in shape]
    lab = rng.integers(1, 1 + s[0] * s[1] * s[2], size=s).astype(np.int32)
    q = (x + y // 2 + z // 3) % shape[2]
    return np.ascontiguousarray(lab[z // edge, y // edge, q // edge])


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("sigma", [0.5, 0.8, 1.0, 1.4, 1.5, 2.0, 2.2])
@pytest.mark.parametrize("shape", [(19, 21, 37), (1, 45, 53)])
def test_every_radius(shape, sigma, precision):
    _agree(_blocks(shape, 7, 3), sigma, precision)


@pytest.mark.parametrize("shape", [(2, 2, 2), (3, 5, 40), (1, 1, 9), (1, 3, 70), (33, 2, 2), (17, 33, 17)])
def test_grids_smaller_than_a_tile(shape):
    _agree(_blocks(shape, 2, 5), 1.5, "f32")
    _agree(_blocks(shape, 2, 6), 1.5, "f64")


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("shape,edge,lo,hi", [((24, 32, 40), 16, 1, 20000), ((52, 60, 60), 16, 45000, 72000),
                                              ((80, 88, 100), 9, 170000, 10 ** 9)])
def test_item_counts(shape, edge, lo, hi, precision):
    """FP32: three warps per half item up to 592 items of 64 cells, half items
    up to 1776, whole ones beyond (148 SMs); FP64 changes at 370 and 1184."""
    assert lo <= _agree(_blocks(shape, edge, 7), 1.5, precision) <= hi


def test_more_labels_than_the_pool_holds():
    rng = np.random.default_rng(9)
    phi = rng.integers(0, 700, size=(48, 64, 64)).astype(np.int32)
    _agree(phi, 1.0, "f32")
    _agree(phi, 1.0, "f64", kinds=("tiled", "tiled_batched"))
