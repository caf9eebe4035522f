"""The summation tree and the transaction sweep of the Al-Cu chain where they can go wrong.

The tree, bit for bit against np.sum: sizes around a leaf (8, 128 values), a
block's subtree (4096), the levels above it (131072, 4194304) and sizes whose
unequal halves put a node's children at different depths, with zeros of both
signs (an absent split must not add +0).

The transactions against the oracle's serial order: every interface cell
crosses, so that chains of waiting neighbours run through the whole field; and
a label that the sweep can reduce to one cell, which keeps the serial order.
"""
import numpy as np
import pytest

from oracle import alcu_oracle as O

gpu = pytest.mark.gpu

SIZES = [1, 7, 8, 9, 127, 128, 129, 136, 257, 1031, 4095, 4096, 4097, 4111, 8193, 8207, 65551, 131071, 131072, 131073,
         131111, 262159, 1000003, 4194303, 4194304, 4194312, 5000016]


@gpu
@pytest.mark.parametrize("n", SIZES)
def test_pairwise_tree(n):
    import torch

    from gpk.alcu import AlCuTransport

    rng = np.random.default_rng(n)
    rows = next(r for r in range(1, n + 1) if n % r == 0 and n // r <= 1 << 20)
    h = AlCuTransport((rows, n // rows), O.AlCuParams())
    for x in (rng.normal(size=n) * 10.0 ** rng.integers(-8, 9, n), np.full(n, -0.0),
              np.where(rng.random(n) < 0.5, 0.0, -0.0)):
        x = x.reshape(rows, -1)
        for _ in range(2):  # the tickets are zero again after a sum
            got = np.float64(h.sum(torch.from_numpy(x).cuda()))
            assert got.tobytes() == np.float64(np.sum(x)).tobytes()


@gpu
@pytest.mark.parametrize("shape,density,speck", [((40, 37, 33), 1.0, False), ((40, 37, 33), 1.0, True),
                                                 ((130, 121), 1.0, False), ((2, 3, 700), 1.0, False),
                                                 ((60, 56, 50), 0.9, False)])
def test_transaction_chains(shape, density, speck):
    import torch

    from gpk.alcu import AlCuTransport

    rng = np.random.default_rng(7)
    labels = rng.integers(0, 4, size=shape).astype(np.int8)
    labels = np.repeat(np.repeat(labels[..., ::3, ::3], 3, axis=-1), 3, axis=-2)[..., : shape[-2], : shape[-1]].copy()
    if speck:
        labels[tuple(s // 2 for s in shape)] = 9
    mask, comp = O.neighbor_competitor(labels)
    crossing = mask & (rng.random(shape) < density)
    if speck:
        crossing[tuple(s // 2 for s in shape)] = True
    alpha = -rng.uniform(0.0, 0.3, shape)
    lr, ar = labels.copy(), alpha.copy()
    want = O.commit_topology_transactions(lr, ar, comp, crossing)
    h = AlCuTransport(shape, O.AlCuParams())
    dl, da = torch.from_numpy(labels).cuda(), torch.from_numpy(alpha).cuda()
    got = h.commit_transactions(dl, da, torch.from_numpy(comp).cuda(),
                                torch.from_numpy(crossing.astype(np.uint8)).cuda())
    assert got == want
    assert np.array_equal(dl.cpu().numpy(), lr)
    assert np.array_equal(da.cpu().numpy().view(np.uint64), ar.view(np.uint64))
