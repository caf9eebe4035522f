"""A step that finds no memory for its model's buffers fails before it changes
anything: labels, fields, time and step count are as they were, and the same
step taken later gives the bits of an undisturbed run.
"""
import numpy as np
import pytest

from gpk_b200 import GPKError, GPKGrid, thermo

pytestmark = pytest.mark.gpu
MIB = 1 << 20
N = 128  # FP64: 16 MiB a buffer


def _solute():
    th = thermo.solidification(M0=5e-8, sigma0=0.2, eps4=0.04, m_liq=-500.0, k_part=0.14, T_melt=933.0, L=1e8)
    th.solute_rejection, th.k_partition = True, 0.14
    return th, 3e-9


def _elastic():
    th = thermo.isotropic(5e-8, 0.2)
    th.elastic_enabled, th.elastic_modulus, th.eigenstrain_coeff = True, 1e9, 0.01
    return th, 0.0


def _grid(model):
    th, D = model()
    g = GPKGrid(N, N, N, 0.5e-6, th, D, 1.5, precision="f64")
    z, y, x = np.indices((N, N, N)) - N // 2
    g.set("phi", ((x * x + y * y + z * z) <= 36).astype(np.int32))
    g.set("c", 0.02)
    g.set("T", 893.0)
    return g


# the solute's buffers: none, one or two of them fit (16 MiB each, and 2 for the flags)
@pytest.mark.parametrize("model,leave", [(_solute, 8), (_solute, 26), (_elastic, 8), (_elastic, 42)])
def test_step_without_memory(model, leave):
    torch = pytest.importorskip("torch")
    fields = ("phi", "alpha", "c", "vn_f", "E_el")
    ref = _grid(model)
    for _ in range(3):
        ref.step()
    want, when = {f: ref.get(f) for f in fields}, ref.time
    ref.close()
    g = _grid(model)
    first = {f: g.get(f) for f in fields}
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    room = torch.cuda.mem_get_info()[0] - leave * MIB
    held = torch.empty(room // (2 * MIB) * 2 * MIB, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            with pytest.raises(GPKError) as e:
                g.step()
            assert e.value.code == 4
        assert g.time == 0.0 and g.step_id == 0
        for f in fields:
            assert np.array_equal(first[f], g.get(f)), f
    finally:
        del held
        torch.cuda.empty_cache()
    for _ in range(3):
        g.step()
    assert g.time == when
    for f in fields:
        assert np.array_equal(want[f].view(np.uint8), g.get(f).view(np.uint8)), f
    g.close()
