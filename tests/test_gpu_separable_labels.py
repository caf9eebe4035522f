"""The separable geometry's label boxes, found on the device.

Labels whose boxes and whole-grid passes (taken where the marks of all labels a
grid has had need more than eight bytes a cell) must give the same bits: more
labels than one copy brings back, single cells, labels everywhere, extents that
are no multiple of a warp, boxes across the seam.  And ids far apart, as after
most grains of a run have gone, cost no more than dense ones.
"""
import time

import numpy as np
import pytest

from gpk_b200 import GPKGrid, thermo, voronoi

pytestmark = pytest.mark.gpu
FIELDS = ("mask", "nx_f", "ny_f", "nz_f", "kappa_f")


def _grid(phi, precision="f32"):
    g = GPKGrid(*phi.shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, 5.0, precision=precision)
    g.set("phi", phi)
    return g


def _geometry(phi, precision):
    g = _grid(phi, precision)
    g.geometry()
    out = {f: g.get(f) for f in FIELDS}, g.get("phi_comp"), g.launch_count()
    g.close()
    return out


def _labels(name):
    rng = np.random.default_rng(3)
    if name == "noise":  # 1500 labels all over the grid: each box is the grid
        return rng.integers(0, 1500, size=(40, 38, 45)).astype(np.int32)
    if name == "single cells":  # 1100 labels of one cell each
        phi = np.zeros((41, 39, 50), dtype=np.int32)
        at = rng.choice(phi.size, size=1100, replace=False)
        phi.ravel()[at] = 1 + np.arange(1100)
        return phi
    if name == "seam":
        phi = np.zeros((38, 70, 33), dtype=np.int32)
        phi[-3:, :5, 20:] = 1
        phi[:4, :5, 20:] = 1
        phi[10:20, 60:, :3] = 2
        phi[10:20, :8, :3] = 2
        phi[10:20, 60:, -4:] = 2
        return phi
    return voronoi(40, 64, 96, 30, 4)[0]


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("name", ["noise", "single cells", "seam", "grains"])
def test_boxes_against_whole_grid_passes(name, precision):
    phi = _labels(name)
    span = sum(phi.shape)
    far = 8 * phi.size // span + 2     # an id from which on the marks do not fit
    assert phi.max() + 1 < far
    top = np.where(phi == phi.max(), far, phi).astype(np.int32)
    (a, ca, la), (b, cb, lb) = _geometry(phi, precision), _geometry(top, precision)
    assert la != lb
    for f in FIELDS:
        assert np.array_equal(a[f].view(np.uint8), b[f].view(np.uint8)), f
    assert np.array_equal(np.where(ca == phi.max(), far, ca), cb)


def test_ids_far_apart():
    phi = voronoi(128, 128, 128, 24, 4)[0]
    ms = []
    for mul in (1, 1700):  # 40 801 labels: 7.5 bytes of marks a cell
        g = _grid(phi * mul)
        t = []
        for _ in range(15):
            t0 = time.perf_counter()
            g.geometry()
            t.append(time.perf_counter() - t0)
        ms.append(1e3 * float(np.median(t[3:])))
        g.close()
    assert ms[1] < 3 * ms[0], ms
