"""The crossing sweep's window test of branch connectivity against the oracle.

The window (9^3 cells, 15^2 in 2-D) decides most label-wide tests; the flood
fill decides what leaves the window, and everything where an extent is shorter
than it.  Sizes below, at and above the window's, with labels whose branches
meet inside it, outside it or not at all; every public field is compared bit
for bit after each step.
"""
import numpy as np
import pytest

from _cases import compare_all
from gpk_b200 import GPKGrid, thermo

pytestmark = pytest.mark.gpu


def _lockstep(oracle_mod, phi, steps):
    iso = thermo.isotropic(1.0, 1.0)
    gpu = GPKGrid(*phi.shape, 1.0, iso, 0.0, 0.6)
    ora = oracle_mod.OracleGrid(*phi.shape, 1.0, iso, 0.0, 0.6)
    rng = np.random.default_rng(2)
    alpha = rng.uniform(0.02, 1.0, phi.shape).astype(np.float32)
    for g in (gpu, ora):
        g.set("phi", phi)
        g.set("alpha", alpha)
        g.set("g", (phi * 0.1).astype(np.float32))
    floods = 0
    for s in range(steps):
        assert gpu.step() == ora.step(), s
        assert not compare_all(gpu, ora), s
        floods += gpu.wave_stats()["flood_fills"]
    return floods


@pytest.mark.parametrize("shape", [(8, 12, 11), (9, 9, 9), (10, 9, 21), (16, 18, 20), (1, 14, 40), (1, 15, 15),
                                   (1, 16, 33), (1, 60, 64)])
def test_window_and_flood_fill(oracle_mod, shape):
    """Blocks of two or three cells of few labels: clusters wind through the
    grid, so branches meet near the cell, far from it and nowhere."""
    rng = np.random.default_rng(shape[1] * 100 + shape[2])
    small = [max(1, (e + 2) // 3) for e in shape]
    phi = rng.integers(1, 5, size=small)
    for a in range(3):
        phi = np.repeat(phi, 3, axis=a)
    phi = np.ascontiguousarray(phi[:shape[0], :shape[1], :shape[2]]).astype(np.int32)
    if shape[0] == 1:
        phi = np.ascontiguousarray(phi[:1])
    assert _lockstep(oracle_mod, phi, 12) > 0


def test_long_channel(oracle_mod):
    """A serpentine two cells wide: its ends are connected only far outside
    the window of any cell that a crossing would remove."""
    phi = np.ones((1, 48, 48), dtype=np.int32)
    for k, y in enumerate(range(4, 44, 6)):
        phi[0, y:y + 2, 4:44] = 2
        x = 42 if k % 2 == 0 else 4
        phi[0, y:y + 8 if y + 8 <= 44 else 44, x:x + 2] = 2
    phi[0, 20:28, 20:28] = 3
    assert _lockstep(oracle_mod, phi, 20) > 0
