"""Tree DP on cost maps with NaN and infinite prefix sums, net by net against the CPU
oracle.  Infinite sums leave some nets without a finite range: those are refused
(IGR_ERR_STATE) with the record up to the node concerned, the start of the oracle's.
Every other net has the oracle's record and difference array, and a net that reads
none of the odd sums is never refused."""
import numpy as np
import pytest

import instantgr_b200 as ig
import cases
from oracle_py import Oracle
from test_gpu_kernels import ctx_for
from test_gpu_pattern_edges import _batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dir0,signs", [(0, (1,)), (1, (1,)), (1, (1, -1))])
def test_nets_on_infinite_sums_one_by_one(dir0, signs):
    g = cases.grid_case(71, X=61, Y=47, dir0=dir0)
    c = ctx_for(g)
    c.cost_refresh()
    vc, ps = c.costs()
    c.close()
    X, Y, XY = g["X"], g["Y"], g["X"] * g["Y"]
    r = np.random.default_rng(5)
    at = 5 * XY + r.integers(0, 4 * XY, XY // 10)
    ps[at[::2]] = np.nan
    for i, sign in enumerate(signs):
        ps[at[1 + 2 * i::2 * len(signs)]] = sign * np.inf
    odd = ~np.isfinite(ps.reshape(g["L"], X, Y)).all(axis=0)
    tb, o, refused = _batch(g, "random", 72), Oracle(g), 0
    for k, cap in enumerate(tb["route_cap"]):
        a, b = tb["node_off"][k], tb["node_off"][k + 1]
        nodes, par = tb["nodes"][a:b], tb["par"][a:b]
        r_gpu, r_orc = np.zeros(cap, np.int32), np.zeros(cap, np.int32)
        pre, st = np.zeros(o.N, np.int32), np.zeros(o.N, np.int32)
        args = (np.array([0, b - a]), nodes, par, np.zeros(1, np.int64), np.array([cap]))
        assert o.pattern_route(vc, ps, *args, r_orc, pre, st, 5) == 0
        c = ctx_for(g)
        c.set_costs(vc, ps)
        try:
            c.pattern_route(*args, r_gpu, 5)
            code = ig.IGR_OK
        except ig.IgrError as e:
            code = e.code
        m = int(r_gpu[0])
        if code == ig.IGR_OK:
            assert np.array_equal(r_gpu[:m], r_orc[:r_orc[0]]), f"net {k}"
            assert np.array_equal(c.pre(), pre), f"net {k}"
        else:
            x, y = nodes // Y % X, nodes % Y
            p = np.maximum(par, 0)
            assert odd[x, y].any() or odd[x[p], y].any() or odd[x, y[p]].any(), f"net {k} reads no odd sum"
            assert code == ig.IGR_ERR_STATE and m <= r_orc[0], f"net {k}"
            assert np.array_equal(r_gpu[1:m], r_orc[1:m]), f"net {k}"
            refused += 1
        c.close()
    assert 0 < refused < len(tb["route_cap"])
