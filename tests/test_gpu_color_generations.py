"""The colouring where its map values run out of batch generations (16,385 nets
take 15 bits of a value and leave 1,024 generations) and where the lists of nets
left over are longer than those that claim while they are listed: the oracle's
batches, number by number."""
import numpy as np
import pytest

import instantgr_b200 as ig
import cases
from oracle_py import color as orc_color

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,X,Y,n,least", [(41, 12, 12, 16385, 1025), (42, 400, 400, 80000, 2)])
def test_batches_across_generations_match_oracle(seed, X, Y, n, least):
    args = cases.color_case(seed, X, Y, n)
    g = cases.grid_case(1, X=X, Y=Y)
    c = ig.Ctx(g["L"], X, Y, g["DIR"], g["xlen"], g["ylen"], g["unit_wire"], g["unit_via"], g["short"], g["cap"])
    ig.set_test_hook(ig.HOOK_COLOR_KEEP_MAP, 0)
    try:
        got, batches = c.color_batches(*args, sparsity=3)
    finally:
        ig.set_test_hook(ig.HOOK_RESET)
    want, n_want = orc_color(X, Y, *args, sparsity=3)
    assert n_want >= least  # the case is what it is meant to be
    assert batches == n_want
    assert np.array_equal(got, want)
