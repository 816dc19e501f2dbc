"""Beads that move far between two neighbour lists: the minimum image, left out
while no listed pair can reach half the box, is back before one does.  Four beads
without bonds, of which the first and the last repel each other, fly apart past
half the box while they stay listed; their force is the one of the nearest image,
by the formula in 64 bits.  T = 0: no noise, velocities stay."""
import numpy as np
import pytest

from sop_gb300 import engine, system

pytestmark = pytest.mark.gpu

FORMS = [{}, dict(nplup=1), dict(nplup=1, lanes_per_bead=8), dict(lanes_per_bead=4, step_split=1),
         dict(lanes_per_bead=4, step_split=2), dict(step_split=3), dict(step_split=4)]


def fly(sep, y, speed, **kw):
    """A context of the four beads, the outer two `sep` (along x) and `y` apart,
    each moving at `speed` A a step."""
    x = np.zeros((4, 3), np.float32)
    x[:, 0] = [-0.5 * sep, -1.0, 1.0, 0.5 * sep]
    x[:, 1] = [-0.5 * y, 0.0, 0.0, 0.5 * y]
    v = np.zeros((4, 3), np.float32)
    v[[0, 3], 0] = [-speed / 0.05, speed / 0.05]
    no_i, no_f = np.zeros(0, np.int32), np.zeros(0, np.float32)
    m = system.Molecule(4, x, no_i, no_i, no_f, no_i, no_i, no_i, no_f, no_i, no_i, no_f, no_f)
    e = engine.Engine(engine.baseline_params(**kw))
    e.add(m, x, T=0.0, vel=v)
    e.commit()
    return e


def exact_force(x, boxl):
    """On the last bead: eps ((s/r)^12 + (s/r)^6), s = 3.8, of the nearest image."""
    d = x[0].astype(np.float64) - x[3]
    d -= boxl * np.rint(d / boxl)
    r2 = (d ** 2).sum()
    u3 = (3.8 ** 2 / r2) ** 3
    return -6.0 / r2 * (2.0 * u3 * u3 + u3) * d


def check(e, boxl, beyond):
    """The forces of the current step; beyond: whether the pair is past half the
    box.  FP32 separations are exact to 1e-7 of the box and enter to the 14th
    power at most: 1e-4 covers boxes up to a few times the separation."""
    d = e.download(0)
    assert (abs(d["unc_pos"][3, 0] - d["unc_pos"][0, 0]) > 0.5 * boxl) == beyond
    i, j, _ = e.list_pairs(0, 3)
    assert list(zip(i, j)) == [(0, 3)]
    want = exact_force(d["unc_pos"], boxl)
    np.testing.assert_allclose(d["force"][3], want, rtol=1e-4, atol=1e-4 * np.abs(want).max())
    np.testing.assert_allclose(d["force"][0], -want, rtol=1e-4, atol=1e-4 * np.abs(want).max())
    assert e.status(0)[0] == 0


@pytest.mark.parametrize("kw", FORMS)
def test_past_half_the_box_before_the_next_list(kw):
    boxl = 40.0
    with fly(6.0, 1.0, 0.25, boxl=boxl, nnlup=200, nl_rep_abs=8.0, pl_rep_abs=30.0, **kw) as e:
        check(e, boxl, False)
        for n, beyond in ((10, False), (20, True), (15, True), (12, True)):
            e.step(n)
            check(e, boxl, beyond)


@pytest.mark.parametrize("kw", FORMS)
def test_past_half_the_box_in_the_step_after_a_list(kw):
    """The list before step 2 is built from coordinates within half the box, the
    step itself is at ones beyond it."""
    boxl = 60.0
    with fly(-3.0, 5.0, 8.3, boxl=boxl, nnlup=2, nl_rep_abs=15.0, pl_rep_abs=40.0,
             **{**dict(nplup=2), **kw}) as e:
        e.step(1)
        check(e, boxl, False)
        e.step(1)
        check(e, boxl, True)


@pytest.mark.parametrize("kw", FORMS)
def test_fast_upload(kw):
    """The same by velocities that a running context is given."""
    boxl = 40.0
    with fly(6.0, 1.0, 0.0, boxl=boxl, nnlup=200, nl_rep_abs=8.0, pl_rep_abs=30.0, **kw) as e:
        e.step(7)
        d = e.download(0)
        v = np.zeros((4, 3), np.float32)
        v[[0, 3], 0] = [-20.0, 20.0]
        e.upload_state(0, d["unc_pos"], vel=v)
        for n, beyond in ((5, False), (5, True), (2, True)):
            e.step(n)
            check(e, boxl, beyond)
