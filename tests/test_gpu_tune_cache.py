"""The autotuner's file: what is taken from it and what is measured anew."""
import pytest

import instantgr_b200 as ig

pytestmark = pytest.mark.gpu


def test_lines_of_an_earlier_kernel_are_measured_anew(tmp_path, monkeypatch):
    """A line that names its kernel is taken by the next router of the design; one
    timed with an earlier tree DP (grid, nets, batches, classes, split, lanes per net
    of three classes, no name) is not, and the design gets a line of its own."""
    tune = tmp_path / "tune.txt"
    monkeypatch.setenv("IGR_TUNE_CACHE", str(tune))
    cap, net = str(tmp_path / "d.cap"), str(tmp_path / "d.net")
    ig.generate_custom(96, 80, 3000, seed=4, cap=cap, net=net)

    def route():
        r = ig.Router(cap, net, rrr_iters=0, batched=1)
        r.run()
        r.close()
        return tune.read_text().splitlines()

    first = route()
    assert len(first) == 1 and first[0].split()[1:3] == ["96", "80"]
    assert route() == first
    key = first[0].split()[1:5]
    old = " ".join(key + ["3", "6", "32", "16", "16"])
    tune.write_text(old + "\n")
    lines = route()
    assert lines[0] == old and len(lines) == 2 and lines[1].split()[:5] == first[0].split()[:5]
    assert route() == lines
