"""The repulsive pair-list rows as the force sum reads them (chunks of 16 entries,
four words each, the last chunk filled up with the bead itself): forces at every
lane count against the oracle and as the same bits, rows of every length modulo 16
among them, freshly built and restored into a context that holds another molecule."""
import numpy as np
import pytest

from oracle import pyoracle as O
from sop_gb300 import engine, system

pytestmark = pytest.mark.gpu

_X = {}


def start(n):
    if n not in _X:
        m = system.generate(n, 11)
        x = m.xyz + np.random.default_rng(n).normal(0, 0.1, m.xyz.shape)
        _X[n] = (m, x.astype(np.float32))
    return _X[n]


def context(n, extra=0, **kw):
    """A plain context, and with `extra` a second molecule of that size."""
    m, x = start(n)
    e = engine.Engine(engine.baseline_params(**kw))
    e.add(m, x, T=0.6)
    if extra:
        e.add(*start(extra), T=0.6)
    e.commit()
    return e


def forces(e):
    e.set_noise(np.zeros((sum(m.n for m in e.mols), 3), np.float32))
    e.force_eval()
    return e.download(0)["force"]


@pytest.mark.parametrize("n", [3, 19, 700])
@pytest.mark.parametrize("lanes", [2, 4, 8, 16])
@pytest.mark.parametrize("split", [1, 2])
def test_forces_of_rows(n, lanes, split):
    m, x = start(n)
    # the two-kernel form gathers from the rows whatever the lanes
    with context(n, lanes_per_bead=lanes, step_split=2) as e:
        want = forces(e)
        blob = e.checkpoint(0)
        ai, aj, _ = e.list_pairs(0, 2)
        ri, rj, _ = e.list_pairs(0, 3)
    lengths = np.bincount(np.concatenate([ri, rj]).astype(np.int64), minlength=n)
    if n == 700:
        assert set(lengths % 16) == set(range(16))
    with context(n, lanes_per_bead=lanes, step_split=split) as e:
        got = forces(e)
    assert np.array_equal(got, want)
    key = {(int(a), int(b)): k for k, (a, b) in enumerate(zip(m.nat_i, m.nat_j))}
    sel = np.array([key[(int(a), int(b))] for a, b in zip(ai, aj)], np.int64)
    exact, _ = O.forces_f64(m, x, sel, ri, rj)
    # the package's bound on a force: 1e-5 of the largest
    assert np.abs(got.astype(np.float64) - exact).max() <= 1.0e-5 * max(np.abs(exact).max(), 1e-12)
    # restored rows
    with context(n, extra=1500, lanes_per_bead=lanes, step_split=split) as e:
        e.restore(0, blob)
        r2, s2, _ = e.list_pairs(0, 3)
        assert np.array_equal(r2, ri) and np.array_equal(s2, rj)
        assert np.array_equal(forces(e), want)


@pytest.mark.parametrize("n", [16385, 19456, 19457])
def test_list_and_step_in_one_launch_of_large_contexts(n):
    """The edges of the range where short rows keep the staged form, against the
    two-kernel form: the same bits."""
    m, x = start(n)
    got = []
    for split in (1, 2):
        e = engine.Engine(engine.default_params(h=0.05, zeta=0.05, step_split=split))
        e.add(m, x, T=0.6)
        e.commit()
        e.step(13)
        got.append([*(e.download(0)[k] for k in ("unc_pos", "vel", "force")), e.energy(0),
                    *e.list_pairs(0, 3)])
        e.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
