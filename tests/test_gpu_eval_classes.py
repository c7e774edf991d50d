"""Device evaluator on nets of each of its size classes (up to 64, 1,024 and
8,192 guide lines, and more), against a plain restatement of the evaluator's
rules on the guide file the same run writes.  Wire length and via cost are
whole numbers times the unit costs and must be equal; the overflow is a sum of
X * Y exponentials per layer in another order: 1e-12 relative."""
import collections
import math

import numpy as np
import pytest

import instantgr_b200 as ig

pytestmark = pytest.mark.gpu


def _score(grid, out):
    """Totals of a guide file by the rules of run/evaluator.cpp:462-672."""
    X, Y, L = grid["X"], grid["Y"], grid["L"]
    wire, stacked = np.zeros((L + 1, X, Y), np.int64), np.zeros((L + 1, X, Y), np.int64)
    vias = wl = 0
    lines = []
    most = 0
    for text in open(out):
        f = text.split()
        if f and f[0] == ")":
            most = max(most, len(lines))
            marks, places = set(), collections.OrderedDict()
            for xl, yl, zl, xh, yh, zh in lines:
                if zl != zh:
                    vias += zh - zl
                    for z in range(zl, zh):
                        places[z, xl, yl] = 1
                    continue
                for x in range(xl, xh + 1):
                    for y in range(yl, yh + 1):
                        marks.add((zl, x, y))
                        if (x, y) != (xh, yh):
                            wire[zl, x, y] += 1
                            wl += int(grid["xlen"][x]) if yl == yh else int(grid["ylen"][y])
            for z, x, y in places:
                if z < 1 or (z, x, y) in marks:
                    continue
                hor = ((z - 1) & 1) ^ grid["DIR"] == 0
                c, last = (x, X - 1) if hor else (y, Y - 1)
                before = (z, x - 1, y) if hor else (z, x, y - 1)
                if 0 < c < last:
                    stacked[before] += 1
                    stacked[z, x, y] += 1
                elif c > 0:
                    stacked[before] += 2
                elif c < last:
                    stacked[z, x, y] += 2
            lines = []
        elif len(f) == 6:
            lines.append([int(v) for v in f])
    cap = grid["cap"].reshape(L, X, Y).astype(np.float64)
    overflow = 0.0
    for z in range(1, L + 1):
        dem = ((2 * wire[z] + stacked[z]) & 0xffff).astype(np.float64)
        c = cap[z - 1]
        t = np.where(c > 0.001, np.exp((dem - 2 * c) / 2 * 0.5), np.where(dem > 0, np.exp(1.5 * dem * 0.5), 0.0))
        overflow += math.fsum(t.ravel()) * grid["short"][z - 1]
    return wl * grid["unit_wire"], vias * grid["unit_via"], overflow, most


@pytest.mark.parametrize("pins,lines", [(40, 65), (700, 1025), (5200, 8193)])
def test_evaluation_of_a_net_of_each_class(tmp_path, pins, lines):
    cap, net, out = (str(tmp_path / f"d.{e}") for e in ("cap", "net", "out"))
    ig.generate_custom(150, 140, 300, seed=5, cap=cap, net=net)
    r = np.random.default_rng(pins)
    at = r.permutation(150 * 140)[:pins]
    with open(net, "a") as f:  # one net of many pins beside the small ones
        f.write("big\n(\n")
        for a in at:
            f.write(f"[({r.integers(0, 2)}, {a // 140}, {a % 140})]\n")
        f.write(")\n")
    router = ig.Router(cap, net, rrr_iters=1)
    router.run()
    got = router.evaluate()
    again = router.evaluate()
    router.write(out)
    wl, via, of, most = _score(router.grid(), out)
    router.close()
    assert most >= lines, "the big net belongs to the class"
    assert got["wirelength"] == wl and got["via"] == via
    assert abs(got["overflow"] - of) <= 1e-12 * of
    assert again["total"] == got["total"]
