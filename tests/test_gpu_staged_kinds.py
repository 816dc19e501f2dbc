"""Which contexts the staged steps take (Engine.staged): the comparisons of
test_gpu_staged.py and test_gpu_pair_rows.py are of the kernels they name, both
kinds of tile among them, and the edges of the ranges lie where they are said to."""
import numpy as np
import pytest

from sop_gb300 import engine, system
from test_gpu_staged import CASES, build

pytestmark = pytest.mark.gpu

_MOLS = {}


def one(n, **kw):
    """A context of one molecule at the factor cut-offs (short rows)."""
    if n not in _MOLS:
        _MOLS[n] = system.generate(n, 11)
    return engine.plain(_MOLS[n], params=engine.default_params(h=0.05, zeta=0.05, **kw))


@pytest.mark.parametrize("case", list(CASES))
def test_compared_contexts_are_staged(case):
    beads = sum(n for n, *_ in CASES[case][0])
    for lanes in (0, 8):
        with build(case, nplup=10, lanes_per_bead=lanes) as e:
            e.step(13)
            s = e.staged()
            per = 32 if lanes == 8 or beads > 8192 else 16
            assert (s["kind"], s["lanes"]) == ("tiles", 256 // per)
            assert s["tiles"] == -(-beads // per)
            # rows of up to 192 entries and 32 native contacts fit a tile: all but
            # the dense globule's (about 340) and the two types' (about 60)
            assert (s["gathered"] > 0) == (case in ("dense", "two types"))
        with build(case, nplup=1, lanes_per_bead=lanes) as e:
            s = e.staged()
            assert (s["kind"], s["tiles"], s["gathered"]) == ("pair list and step", 0, 0)
            assert s["lanes"] == (lanes or 16)
    with build(case, nplup=10, lanes_per_bead=4, step_split=2) as e:
        assert e.staged()["kind"] is None


@pytest.mark.parametrize("n,nplup,kind,lanes", [
    (8192, 10, "tiles", 16), (8193, 10, "tiles", 8), (16384, 10, "tiles", 8), (16385, 10, None, 0),
    (8192, 1, "pair list and step", 16), (8193, 1, "pair list and step", 8),
    (19456, 1, "pair list and step", 8), (19457, 1, None, 0)])
def test_edges_of_the_ranges(n, nplup, kind, lanes):
    with one(n, nplup=nplup) as e:
        s = e.staged()
        assert (s["kind"], s["lanes"]) == (kind, lanes)


@pytest.mark.parametrize("kw", [dict(step_split=2), dict(step_split=3), dict(step_split=4),
                                dict(lanes_per_bead=2), dict(lanes_per_bead=4), dict(step_window=512),
                                dict(step_buckets=1)])
@pytest.mark.parametrize("nplup", [1, 10])
def test_what_the_parameters_ask_for_instead(kw, nplup):
    with one(500, nplup=nplup, **kw) as e:
        assert e.staged()["kind"] is None


@pytest.mark.parametrize("count,n,lanes,window", [
    (1, 1344, 16, 1600), (1, 1600, 16, 1600), (1, 1601, 16, 0), (10, 400, 16, 656),
    # 304 blocks at three an SM, then more blocks than are resident with a window
    (6, 800, 16, 1056), (5, 1600, 16, 0), (20, 800, 8, 0), (13, 1495, 8, 0), (41, 450, 8, 0)])
def test_window_while_the_blocks_are_resident(count, n, lanes, window):
    """Launches of one wave with their window (152 SMs) take it; where it keeps
    blocks from being resident they gather.  The steps are the same bits."""
    states = []
    for kw in ({}, dict(step_split=2, lanes_per_bead=4)):
        if (n, 0) not in _MOLS:
            _MOLS[n, 0] = system.generate(n, 3)
        m = _MOLS[n, 0]
        e = engine.Engine(engine.default_params(h=0.02, zeta=0.05, **kw))
        for k in range(count):
            e.add(m, m.xyz, T=0.6, traj=k)
        e.commit()
        if not kw:
            s = e.staged()
            assert (s["kind"], s["lanes"], s["window"]) == ("pair list and step", lanes, window)
        e.step(53)
        states.append([e.download_all()] + [e.download(count - 1)[k] for k in ("vel", "force")])
        e.close()
    for a, b in zip(*states):
        assert np.array_equal(a, b)


def test_form_that_is_reported():
    """A default context of 128 beads, where the one-block form was once chosen:
    staged, one kernel per step, 16 lanes; nothing is timed for its steps but the
    plain kernel's force evaluations are."""
    with engine.plain(system.generate(128, 0), params=engine.baseline_params()) as e:
        t = e.tuning()
        assert (t["staged"], t["form"], t["lanes_per_bead"]) == ("tiles", 1, 16)
        assert all(v > 0 for v in t["ms"].values())
