"""What Seed.predict returns beyond the channels that the model writes."""
import numpy as np
import pytest

import instantgr_b200 as ig

pytestmark = pytest.mark.gpu


def test_values_the_model_does_not_write_are_zero():
    """Features of 20 values a GCell: the model reads and writes 16 for each, end to
    end, and the rest of the result is zero, whatever the memory held before."""
    m = ig.Seed.load()
    f = np.random.default_rng(1).random((30, 30, 20), np.float32)
    for _ in range(4):
        old = [np.full_like(f, np.nan) for _ in range(8)]
        del old
        got = m.predict(f).reshape(-1)
        assert np.isfinite(got[:30 * 30 * 16]).all()
        assert not got[30 * 30 * 16:].any()
    m.close()
