"""Grain growth does not depend on how far apart the label ids lie: the same
fields, and crossing sweeps whose time does not follow the largest id.
"""
import numpy as np
import pytest

from gpk_b200 import GPKGrid, thermo, voronoi

pytestmark = pytest.mark.gpu


def _run(mul):
    phi, o = voronoi(1, 256, 256, 100, 4)
    g = GPKGrid(1, 256, 256, 1.0, thermo.isotropic(1.0, 1.0), 0.0, 1.5)
    g.set("phi", phi * mul)
    g.set("g", o)
    g.set("alpha", 1.0)
    g.step_n(4)
    g.profile(True)
    g.step_n(24)
    ms, calls = g.stage_times()["crossings"]
    out = {f: g.get(f) for f in ("phi", "alpha", "g")}
    assert g.counters()[0] > 0
    g.close()
    return out, ms / calls


def test_ids_far_apart():
    (a, near), (b, far) = _run(1), _run(50000)  # 5 M ids: 40 MB of counts copied, some 20 us
    assert np.array_equal(a["phi"] * 50000, b["phi"])
    for f in ("alpha", "g"):
        assert np.array_equal(a[f], b[f]), f
    assert far < 3 * near + 0.1, (near, far)
