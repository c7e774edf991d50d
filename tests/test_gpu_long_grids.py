"""Cost refresh and fused batch commit on grids whose two track lengths differ by
far, where a block takes several short tracks: the oracle's costs, the demand of
the separate commits, and a time that follows the cells, not the longer side."""
import time

import numpy as np
import pytest

import instantgr_b200 as ig
import cases
from oracle_py import Oracle
from test_gpu_kernels import RTOL, ctx_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X,Y", [(1025, 31), (31, 1025), (2000, 130), (130, 2000), (4096, 255), (257, 3000), (1024, 2)])
def test_refresh_of_long_grids_matches_oracle(X, Y):
    g = cases.grid_case(X + Y, X=X, Y=Y, dir0=Y & 1, unit_wire=0.3)
    c = ctx_for(g)
    c.cost_refresh()
    v, p = c.costs()
    _, ov, op = Oracle(g).cost_refresh(g["demand"])
    np.testing.assert_allclose(v, ov, rtol=RTOL, atol=0)
    np.testing.assert_allclose(p, op, rtol=RTOL, atol=1e-9)
    c.set_demand(g["demand"][::-1].copy())
    c.cost_refresh()
    full = c.costs()
    c.set_demand(g["demand"])
    c.set_demand(g["demand"][::-1].copy())
    c.cost_refresh(only_dirty=True)
    assert all(np.array_equal(a, b) for a, b in zip(c.costs(), full))
    c.close()


@pytest.mark.parametrize("X,Y", [(1500, 40), (40, 1500), (700, 90), (3000, 257)])
def test_fused_commit_of_long_grids_matches_split_commit(tmp_path, X, Y):
    cap, net = str(tmp_path / "d.cap"), str(tmp_path / "d.net")
    ig.generate_custom(X, Y, 4000, seed=X, cap=cap, net=net, bbox_median=12.0)
    res = []
    for split in (1, 0):
        r = ig.Router(cap, net, rrr_iters=0, split_commit=split)
        r.run()
        s = r.stats()
        res.append((r.demand(), s["wirelength"], s["via_cost"], s["overflow_cost"]))
        r.close()
    assert np.array_equal(res[0][0], res[1][0])
    assert res[0][1:] == res[1][1:]


def test_refresh_time_follows_the_cells():
    """64 x 4096 cells against 512 x 512: the same work, tracks of one to sixteen
    warps.  With a block of the longer track's warps for every track the long grid
    took 16 times as long; the bound is 4, on the least of 20 waits each."""
    best = []
    for X, Y in ((512, 512), (64, 4096)):
        c = ctx_for(cases.grid_case(1, X=X, Y=Y))
        t = []
        for _ in range(23):
            t0 = time.perf_counter()
            c.cost_refresh()
            t.append(time.perf_counter() - t0)
        best.append(min(t[3:]))
        c.close()
    assert best[1] <= 4 * best[0], best
