"""Convolution kernels of the congestion seed at tile sizes where their tiles are
ragged (a tile of 16 x 8 or 16 x 16 pixels at full and half resolution), against
the CPU oracle of the network.  Tolerances as for the gradient checks at even
sizes: both sides round to BF16 at the same points, so only roundings to the
neighbouring BF16 value differ: loss 1e-3, gradients 3e-2 of each layer's norm."""
import numpy as np
import pytest

import instantgr_b200 as ig
from oracle_py import seed_grad, seed_slices

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,halo,T", [(8, 0, 1), (10, 1, 3), (18, 2, 2), (34, 4, 1), (50, 8, 2)])
def test_seed_gradients_at_ragged_tiles(S, halo, T):
    r = np.random.default_rng(S)
    x = r.normal(0, 1, (T, S, S, 16)).astype(np.float32)
    x[..., 14:] = 0
    t = np.abs(r.normal(0, 1, (T, S, S, 16))).astype(np.float32)
    t[..., 10:] = 0
    m = ig.Seed(3)
    m.set_tile(S, halo)
    loss_g, g_g = m.grad(x, t)
    loss_o, g_o = seed_grad(x, t, m.params(), halo, rounded=True)
    m.close()
    assert abs(loss_g - loss_o) <= 1e-3 * loss_o, (loss_g, loss_o)
    for i, slices in enumerate(seed_slices()):
        for sl, what in zip(slices, ("weights", "bias")):
            err = np.linalg.norm(g_g[sl] - g_o[sl]) / max(np.linalg.norm(g_o[sl]), 1e-12)
            assert err <= 3e-2, f"layer {i} {what}: relative error {err:.3g}"
