"""An ensemble whose first context takes the staged steps passes their form on, but
leaves the lanes of the others to their own size: the staged lanes (16 up to
8,192 beads, 8 above) are no choice of the tuner's."""
import pytest

from sop_gb300 import engine


@pytest.mark.parametrize("kind,lanes", [("tiles", 16), ("tiles", 8), ("pair list and step", 8)])
def test_staged_lanes_are_not_passed_on(kind, lanes):
    p = engine.default_params(h=0.03)
    tuned = {"lanes_per_bead": lanes, "form": 1, "window": 0, "buckets": {"tiled": False}, "staged": kind}
    q = engine.matched_params(p, tuned)
    assert (q.lanes_per_bead, q.step_split, q.step_buckets) == (0, 1, -1)
    q = engine.matched_params(p, dict(tuned, staged=None))
    assert (q.lanes_per_bead, q.step_split, q.step_buckets) == (lanes, 1, -1)
