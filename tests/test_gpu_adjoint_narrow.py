"""The calibration's projection, whose taps a lane holds in registers, on fields
narrower than, as wide as and little wider than its 7 x 7 box (each tap wraps),
and with rows that no cell's box leaves.

Forward against the oracle: the tolerance is that of the forward pass elsewhere
(1e-10 of the largest value: FFT and summation rounding).  The transpose by the
identity it has to satisfy: the loss is quadratic in the anisotropies, so its
central difference has no truncation error and is off by rounding alone,
eps * loss / h per difference; 1e-7 of the largest component leaves a factor of
some hundred at h = 1e-3.
"""
import numpy as np
import pytest

from gpk_b200 import GPKGrid, thermo
from gpk.adjoint import AdjointProblem, calibration_case
from oracle import adjoint_oracle

pytestmark = pytest.mark.gpu
CONST = dict(m_fixed=1.0, sigma0=1e-3, c11=1.08, c12=0.62, c44=0.28, energy_weight=1e-6)


@pytest.mark.parametrize("n", [5, 7, 9, 16, 48])
def test_projection_on_narrow_fields(n):
    phi, g, mob_index = calibration_case(n, 6, 1, 3, (1, 2))
    grid = GPKGrid(1, n, n, 1.0, thermo.isotropic(1.0, 1.0), 0.0, 1.5, precision="f64")
    grid.set("phi", phi)
    grid.set("g", g)
    prob = AdjointProblem(grid, mob_index, 6, **CONST)
    rng = np.random.default_rng(5)
    theta = np.concatenate([[0.01, -0.004, 0.003], [0.05, -0.02, 0.01, 0.005], 1.0 + 0.1 * rng.standard_normal(6)])
    star = theta.copy()
    star[3:7] += 0.01
    star[7:] *= 1.0 + 0.05 * rng.standard_normal(6)
    _, target = prob.forward(star, want_v=True)
    prob.set_target(target)

    f = {k: grid.get(k)[0] for k in ("phi", "phi_comp", "mask", "nx_f", "ny_f", "kappa_f", "g")}
    inv = 0.5 / (0.85 * 0.85)
    want, v_want = adjoint_oracle.forward(f["phi"], f["phi_comp"], f["mask"], f["nx_f"], f["ny_f"], f["kappa_f"],
                                          f["g"], mob_index, theta, CONST["c11"], CONST["c12"], CONST["c44"],
                                          CONST["sigma0"], CONST["m_fixed"], CONST["energy_weight"], 1.0, target,
                                          3, lambda r2: float(np.exp(-r2 * inv)))
    loss, v = prob.forward(theta, want_v=True)
    assert abs(loss - want) <= 1e-10 * abs(want)
    assert np.max(np.abs(v - v_want)) <= 1e-10 * np.max(np.abs(v_want))

    grad = prob.gradient(theta)[1][3:7]
    h = 1e-3
    for k in range(4):
        hi, lo = theta.copy(), theta.copy()
        hi[3 + k] += h
        lo[3 + k] -= h
        fd = (prob.forward(hi) - prob.forward(lo)) / (2 * h)
        assert abs(grad[k] - fd) <= 1e-7 * np.max(np.abs(grad)) + 4e-16 * loss / h
