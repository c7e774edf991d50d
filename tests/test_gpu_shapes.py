"""Conflict shapes kept once per cell, by the size of their hash set: designs of one net, of
fewer and more shapes than a block counts (256), and with trees long enough to sample
more cells than a warp's table takes (682 entries).  The colouring must give the
batches that it gives with every repetition kept; whole numbers, so equal."""
import numpy as np
import pytest

import instantgr_b200 as ig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X,Y,nets,bbox", [(61, 44, 1, 5.0), (61, 44, 255, 5.0), (300, 200, 700, 60.0),
                                           (1500, 1200, 600, 900.0), (9000, 40, 300, 6000.0)])
def test_shapes_kept_once_give_the_same_batches(tmp_path, X, Y, nets, bbox):
    cap, net = str(tmp_path / "d.cap"), str(tmp_path / "d.net")
    ig.generate_custom(X, Y, nets, seed=X + nets, pin_mode=1, cap_mode=1, bbox_median=bbox, bbox_sigma=0.3,
                       hotspots=2, hotspot_frac=0.3, cap=cap, net=net)
    res = []
    for dedupe in (0, 1):
        ig.set_test_hook(ig.HOOK_SHAPE_DEDUPE, dedupe)
        try:
            r = ig.Router(cap, net, rrr_iters=2)
            r.run()
            p = r.plan()
            res.append((p["batch_off"], p["net_ids"], r.demand(), r.stats()["color_rounds"]))
            r.close()
        finally:
            ig.set_test_hook(ig.HOOK_RESET)
    (b0, i0, d0, c0), (b1, i1, d1, c1) = res
    assert np.array_equal(b0, b1)
    for b in range(len(b0) - 1):
        assert np.array_equal(np.sort(i0[b0[b]:b0[b + 1]]), np.sort(i1[b1[b]:b1[b + 1]])), f"batch {b}"
    assert np.array_equal(d0, d1)
    assert c0 == c1
