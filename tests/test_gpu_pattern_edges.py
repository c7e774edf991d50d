"""Tree DP at the sizes where its kernel changes path, against the CPU oracle on
the GPU's own cost map: nets at the edges of the shared-memory tile (16 nodes)
and of a 32-node block, shapes that keep more tables alive than there are
slots, and cost maps with NaN and infinite prefix sums.  Routes and difference
array are bit-exact.  Infinite sums give wires of cost -infinity whose sums
with the unreachable ranges are NaN: nets left without a finite range are
reported (IGR_ERR_STATE)."""
import numpy as np
import pytest

import instantgr_b200 as ig
import cases
from oracle_py import Oracle

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 15, 16, 17, 31, 32, 33, 63, 64, 65, 130]


def _batch(g, shape, seed, repeat=6):
    """Nets of every size; parents: the previous node (chain), the root (star),
    half a net earlier (comb: half of the nodes collect children at once), or a
    random earlier node.  Some nodes share a GCell with their parent."""
    r = np.random.default_rng(seed)
    X, Y = g["X"], g["Y"]
    off, nodes, par = [0], [], []
    for m in SIZES * repeat:
        i = np.arange(m)
        p = {"chain": i - 1, "star": 0 * i, "comb": np.maximum(0, i - max(1, m // 2)),
             "random": np.array([0] + [int(r.integers(0, j)) for j in range(1, m)])}[shape]
        p[0] = -1
        x, y = r.integers(0, X, m), r.integers(0, Y, m)
        for j in range(1, m):
            u = r.random()
            if u < 0.3:
                x[j] = x[p[j]]
            elif u < 0.6:
                y[j] = y[p[j]]
            elif u < 0.65:
                x[j], y[j] = x[p[j]], y[p[j]]
        layer = np.where((r.random(m) < 0.4) & (i > 0), 9, r.integers(0, 3, m))
        nodes += (layer * X * Y + x * Y + y).tolist()
        par += p.tolist()
        off.append(len(nodes))
    off = np.array(off, np.int32)
    cap = (8 * np.diff(off) + 1).astype(np.int32)
    return dict(node_off=off, nodes=np.array(nodes, np.int32), par=np.array(par, np.int32), route_cap=cap,
                route_off=np.concatenate([[0], np.cumsum(cap)[:-1]]).astype(np.int64))


@pytest.mark.parametrize("shape,dir0,odd", [("chain", 0, ""), ("star", 1, ""), ("comb", 0, ""), ("random", 1, ""),
                                            ("random", 0, "nan inf"), ("random", 0, "nan")])
def test_tree_dp_at_its_size_limits(shape, dir0, odd):
    g = cases.grid_case(71, X=61, Y=47, dir0=dir0)
    c = ig.Ctx(g["L"], g["X"], g["Y"], g["DIR"], g["xlen"], g["ylen"], g["unit_wire"], g["unit_via"], g["short"],
               g["cap"])
    c.set_demand(g["demand"])
    c.cost_refresh()
    vc, ps = c.costs()
    if odd:  # NaN and infinite sums on upper layers: those ranges drop out
        r = np.random.default_rng(5)
        XY = g["X"] * g["Y"]
        at = 5 * XY + r.integers(0, 4 * XY, XY // 10)
        ps[at[::2]] = np.nan
        if "inf" in odd:
            ps[at[1::2]] = np.inf
        c.set_costs(vc, ps)
    tb = _batch(g, shape, 72)
    total, stamp = int(tb["route_off"][-1] + tb["route_cap"][-1]), 9
    r_gpu, r_orc = np.zeros(total, np.int32), np.zeros(total, np.int32)
    args = (tb["node_off"], tb["nodes"], tb["par"], tb["route_off"], tb["route_cap"], r_gpu, stamp)
    if "inf" in odd:
        with pytest.raises(ig.IgrError) as e:
            c.pattern_route(*args)
        assert e.value.code == ig.IGR_ERR_STATE
        c.close()
        return
    c.pattern_route(*args)
    o = Oracle(g)
    pre, st = np.zeros(o.N, np.int32), np.zeros(o.N, np.int32)
    assert o.pattern_route(vc, ps, tb["node_off"], tb["nodes"], tb["par"], tb["route_off"], tb["route_cap"], r_orc,
                           pre, st, stamp) == 0
    for k, a in enumerate(tb["route_off"]):
        m = int(r_orc[a])
        assert np.array_equal(r_gpu[a:a + m], r_orc[a:a + m]), f"net {k} of {np.diff(tb['node_off'])[k]} nodes"
    assert np.array_equal(c.pre(), pre)
    c.close()
