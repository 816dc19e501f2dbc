"""Where the minimum image is left out of a molecule's force and list terms, it
has to be the identity for every pair the molecule's lists hold, and those may be
older than the extent the flag is taken from.  Here a straight chain whose ends are
listed through its image (extent + cut-off just past the box) contracts until
they are further apart than the cut-off, still listed.  Whatever looks at its
extent in between -- a restore of it or of another molecule of the context -- must
not change its steps."""
import numpy as np
import pytest

from sop_gb300 import engine, system

pytestmark = pytest.mark.gpu

N, CUT = 120, 8.0
FORMS = [{}, dict(nplup=1), dict(lanes_per_bead=4, step_split=2), dict(step_split=4)]


def chain():
    m = system.generate(N, 21)
    x = m.extended_xyz()
    ext = float(np.ptp(x[:, 0]))
    v = np.zeros_like(x)
    mid = 0.5 * (x[:, 0].min() + x[:, 0].max())
    # the ends come nearer by 0.1 A a step each
    v[:, 0] = (-2.0 * (x[:, 0] - mid) / (0.5 * ext)).astype(np.float32)
    return m, x, v, ext + CUT - 0.5


def params(boxl, **kw):
    base = dict(boxl=boxl, nl_rep_abs=CUT, pl_rep_abs=2.0 * CUT, nl_att_abs=CUT, pl_att_abs=CUT)
    return engine.baseline_params(**{**base, **kw})


def context(**kw):
    m, x, v, boxl = chain()
    e = engine.Engine(params(boxl, **kw))
    e.add(m, x, T=0.6, traj=3, vel=v)
    other = system.generate(60, 5)
    e.add(other, other.xyz, T=0.6, traj=4)
    e.commit()
    return e, boxl


def extent(e):
    return float(np.ptp(e.download(0)["unc_pos"], axis=0).max())


def state(e):
    out = []
    for k in range(2):
        d = e.download(k)
        out += [d[q] for q in ("unc_pos", "pos", "vel", "force")] + [e.energy(k)]
        out += list(e.list_pairs(k, 3))
    return out


def ends_listed(e):
    i, j, _ = e.list_pairs(0, 3)
    return (0, N - 1) in set(zip(i.tolist(), j.tolist()))


def uninterrupted(**kw):
    """States at steps 6, 9 and 40; the ends listed through the image at 0 and 6,
    the extent past the line of the flag at 0 and below it at 6."""
    e, boxl = context(**kw)
    assert extent(e) + CUT >= boxl and ends_listed(e)
    out = []
    for n in (6, 3, 31):
        e.step(n)
        if not out:
            assert extent(e) + CUT < boxl - 0.25 and ends_listed(e)
            blobs = [e.checkpoint(k) for k in range(2)]
        out.append(state(e))
    e.close()
    return out, blobs


def same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("kw", FORMS)
def test_restored_context_continues_as_uninterrupted(kw):
    want, blobs = uninterrupted(**kw)
    e, _ = context(**kw)
    for k, b in enumerate(blobs):
        e.restore(k, b)
    got = [state(e)]
    for n in (3, 31):
        e.step(n)
        got.append(state(e))
    e.close()
    for a, b in zip(got, want):
        same(a, b)


@pytest.mark.parametrize("kw", FORMS)
def test_restore_of_one_molecule_leaves_the_other(kw):
    want, _ = uninterrupted(**kw)
    e, _ = context(**kw)
    e.step(6)
    e.restore(1, e.checkpoint(1))
    got = [state(e)]
    for n in (3, 31):
        e.step(n)
        got.append(state(e))
    e.close()
    for a, b in zip(got, want):
        same(a, b)


@pytest.mark.parametrize("kw", [FORMS[0], FORMS[2], FORMS[3]])
@pytest.mark.parametrize("how", ["update", "stage"])
def test_neighbour_list_by_the_caller_keeps_the_pair_list_s_image(how, kw):
    """The caller's own neighbour-list rebuild between two pair-list rebuilds:
    the steps until the next one sum the same pairs, so the same bits."""
    want, _ = uninterrupted(**kw)
    e, _ = context(**kw)
    e.step(6)
    if how == "update":
        e.update_neighbor_list()
    else:
        e.launch_stage(2, 0)
    got = state(e)
    same(got, want[0])
    e.step(3)
    same(state(e), want[1])
    e.close()
