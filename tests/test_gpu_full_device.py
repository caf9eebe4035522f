"""Geometry workspaces on a device with little memory left.

The direct geometry's items and the separable geometry's boxes take what room
there is: with less than their full workspace (and, for the items, with none)
a step gives the same bits as with all of it.
"""
import numpy as np
import pytest

from gpk_b200 import GPKGrid, thermo, voronoi

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _grid(shape, sigma, phi, kind):
    g = GPKGrid(*shape, 1.0, thermo.isotropic(1.0, 1.0), 0.0, sigma)
    g.set_geometry_kernel(kind)
    g.set("phi", phi)
    g.set("alpha", 0.05)
    return g


# 96^3 FP32: the items take 12 MiB and their pool 32, the boxes 58 (least: 10)
@pytest.mark.parametrize("sigma,grains,leave", [(1.5, 200, 30), (1.5, 200, 8), (5.0, 12, 40)])
def test_little_room(sigma, grains, leave):
    torch = pytest.importorskip("torch")
    shape = (96, 96, 96)
    phi = voronoi(*shape, grains, 5)[0]
    fields = ("phi", "nx_f", "ny_f", "nz_f", "kappa_f", "phi_comp", "vn_f", "alpha")
    want = None
    for kind in ("tiled", "tiled_batched", "per_cell"):  # (every kernel is loaded before the memory is held)
        g = _grid(shape, sigma, phi, kind)
        g.step_n(2)
        got = {f: g.get(f) for f in fields}
        want = want or got
        for f in fields:
            assert np.array_equal(want[f].view(np.uint8), got[f].view(np.uint8)), (kind, f)
        del g
    g = _grid(shape, sigma, phi, "tiled")
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = torch.cuda.mem_get_info()[0] - leave * MIB
    held = torch.empty(room // (2 * MIB) * 2 * MIB, dtype=torch.uint8, device="cuda")
    try:
        g.step_n(2)
    finally:
        del held
        torch.cuda.empty_cache()
    for f in fields:
        assert np.array_equal(want[f].view(np.uint8), g.get(f).view(np.uint8)), f
