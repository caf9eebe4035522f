"""The separable geometry's per-label boxes against the oracle, bit for bit.

Boxes that are a whole period along some or all axes, thin ones, ones that
cross the periodic seam, so many that the workspace takes several batches, and
labels whose cells lie in separate places.  FP32 fields equal the oracle's to
the last bit; FP64 fields too, since every value is formed by the same
operations in the same order.
"""
import numpy as np
import pytest

from _cases import compare_all
from gpk_b200 import GPKGrid, thermo

pytestmark = pytest.mark.gpu


def _slab(shape, axis, lo, hi):
    phi = np.ones(shape, dtype=np.int32)
    sl = [slice(None)] * 3
    sl[axis] = slice(lo, hi)
    phi[tuple(sl)] = 2
    return phi


def _case(name):
    if name == "slab":
        return _slab((38, 42, 40), 2, 5, 12)
    if name == "seam":
        phi = _slab((40, 41, 43), 1, 0, 3)
        phi[:, -4:, :] = 2
        return phi
    if name == "two places":
        phi = np.ones((44, 40, 46), dtype=np.int32)
        phi[2:6, 3:9, 1:8] = 7
        phi[30:36, 25:33, 36:45] = 7
        return phi
    from oracle import voronoi
    shape, n = {"periods": ((38, 40, 36), 24), "small grains": ((64, 72, 80), 60)}[name]
    return voronoi(*shape, n, 4)[0]


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("name,sigma", [("slab", 5.0), ("seam", 4.75), ("two places", 5.0), ("periods", 5.0),
                                        ("small grains", 5.5)])
def test_boxes(oracle_mod, name, sigma, precision):
    phi = _case(name)
    iso = thermo.isotropic(1.0, 1.0)
    gpu = GPKGrid(*phi.shape, 1.0, iso, 0.0, sigma, precision=precision)
    ora = oracle_mod.OracleGrid(*phi.shape, 1.0, iso, 0.0, sigma, precision=precision)
    for g in (gpu, ora):
        g.set("phi", phi)
        g.set("alpha", 0.05)
    for s in range(2):
        assert gpu.step() == ora.step(), s
        assert not compare_all(gpu, ora), s
