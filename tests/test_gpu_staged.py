"""The staged steps of small contexts (tiles of 16 or 32 beads; pair-list
rebuild and step in one launch) against the two-kernel form, which gathers
everything from global memory: coordinates (both), velocities, forces, energies
and lists are the same bits, whatever the contexts hold -- two bead types, molecules
that finish mid-run, T = 0, the overdamped integrator, a box that wraps, rows
past what a block keeps in shared memory, tiles whose lists do not fit, sizes
about the tiles' and the window's edges -- and after uploads, restores and
injected noise.  The lists themselves are checked against the oracle."""
import numpy as np
import pytest

from helpers import oracle_lists, pairset
from sop_gb300 import engine, system

pytestmark = pytest.mark.gpu

_MOLS = {}


def mol_of(n, seed, two_types=False):
    key = (n, seed, two_types)
    if key not in _MOLS:
        m = system.generate(n, seed, (0.7, 1.3))
        if two_types:
            # natives by type, as the reference's files hold them: up to about
            # 60 of one bead
            rng = np.random.default_rng(seed)
            ty = np.where(rng.random(n) < 0.3, 2, 1).astype(np.int32)
            ii, jj = np.triu_indices(n, 3)
            d = np.linalg.norm(m.xyz[jj].astype(np.float64) - m.xyz[ii], axis=1).astype(np.float32)
            nat = d < system.RCUT_NAT.astype(np.float32)[ty[ii], ty[jj]]
            ni, nj = ii[nat].astype(np.int32), jj[nat].astype(np.int32)
            m = system.Molecule(n, m.xyz, m.bond_i, m.bond_j, m.bond_r0, m.ang_i, m.ang_j, m.ang_k,
                                m.ang_r, ni, nj, d[nat], np.ones(len(ni), np.float32), types=ty)
        _MOLS[key] = m
    return _MOLS[key]


CASES = {  # molecules (n, two types, start, T, nsteps), parameters
    "one bead past a tile": ([(17, 0, "native", 0.6, -1)], {}),
    "three beads": ([(3, 0, "native", 0.6, -1)], {}),
    "many small, one finishing": ([(60, 0, "native", 0.6, -1), (33, 0, "native", 0.0, -1),
                                   (150, 0, "native", 0.7, 23), (97, 0, "extended", 0.5, -1)],
                                  dict(boxl=2000.0)),
    "two types": ([(700, 1, "native", 0.6, -1)], dict(h=0.0025)),
    "wraps": ([(300, 0, "extended", 0.6, -1), (128, 0, "native", 0.6, -1)], dict(boxl=500.0)),
    "dense": ([(1200, 0, "dense", 0.6, -1)], dict(h=1.0e-5)),
    "window edge": ([(1344, 0, "native", 0.6, -1), (300, 0, "native", 0.6, -1)], {}),
    "past the window": ([(1601, 0, "native", 0.6, -1)], {}),
    "overdamped, 6-power": ([(400, 0, "native", 0.6, -1), (90, 0, "native", 0.6, 31)],
                            dict(integrator=1, h=5.0e-4, rep6=1)),
    "no budgets": ([(60, 0, "native", 0.6, -1), (33, 0, "native", 0.0, -1),
                    (150, 0, "native", 0.7, -1), (97, 0, "extended", 0.5, -1)], dict(boxl=2000.0)),
    "32-bead tiles": ([(9000, 0, "native", 0.6, -1)], {}),
}


def build(case, **kw):
    mols, prm = CASES[case]
    e = engine.Engine(engine.baseline_params(**{**prm, **kw}))
    for k, (n, two, start, T, nsteps) in enumerate(mols):
        m = mol_of(n, 400 + n, bool(two))
        x = m.extended_xyz() if start == "extended" else m.xyz
        if start == "dense":   # eight times as dense: rows of several hundred entries
            x = ((x - x.mean(0)) * 0.5 + x.mean(0)).astype(np.float32)
        e.add(m, x, T=T, traj=k, nsteps=nsteps, vel=np.full((m.n, 3), 0.1, np.float32))
    e.commit()
    return e


def state(e):
    out = []
    for k in range(len(e.mols)):
        d = e.download(k)
        out += [d["unc_pos"], d["pos"], d["vel"], d["force"], e.energy(k), np.array(e.status(k))]
        for which in range(4):
            out += list(e.list_pairs(k, which))
    return out


def same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("case", list(CASES))
@pytest.mark.parametrize("nplup,lanes", [(10, 0), (10, 8), (1, 0), (1, 8)])
def test_staged_equals_two_kernel_form(case, nplup, lanes):
    outs = []
    for kw in (dict(lanes_per_bead=lanes), dict(lanes_per_bead=4, step_split=2)):
        with build(case, nplup=nplup, **kw) as e:
            got = []
            for n in (1, 9, 13, 60):   # before and at a pair-list rebuild, across a neighbour list's
                e.step(n)
                got += state(e)
            outs.append(got)
    same(*outs)


@pytest.mark.parametrize("nplup", [1, 10])
def test_staged_after_upload_restore_and_noise(nplup):
    """State that comes from outside the steps: an upload mid-run, a restore
    into a fresh context (odd and even steps), injected normals; and the lists
    of the last step against the oracle."""
    outs = []
    for kw in ({}, dict(lanes_per_bead=4, step_split=2)):
        got = []
        with build("no budgets", nplup=nplup, **kw) as e:
            e.step(27)
            d = e.download(3)
            e.upload_state(3, d["unc_pos"] + np.float32(0.25), vel=d["vel"])
            e.step(36)
            rng = np.random.default_rng(1)
            e.set_noise(rng.normal(size=(sum(m.n for m in e.mols), 3)))
            e.step(12)
            e.set_noise(None)
            e.step(8)
            got += state(e)
            blobs = [e.checkpoint(k) for k in range(len(e.mols))]
        with build("no budgets", nplup=nplup, **kw) as e:
            for k, b in enumerate(blobs):
                e.restore(k, b)
            e.step(19)
            got += state(e)
            x1 = e.download(0)["unc_pos"]
            e.update_neighbor_list()
            e.update_pair_list()
            m = e.mols[0]
            _, (nri, nrj), _, (opi, opj) = oracle_lists(m, x1, e.params, 2000.0)
            assert pairset(*e.list_pairs(0, 1)[:2]) == pairset(nri, nrj)
            assert pairset(*e.list_pairs(0, 3)[:2]) == pairset(opi, opj)
            e.step(11)
            got += state(e)
        outs.append(got)
    same(*outs)


@pytest.mark.parametrize("n,boxl", [(300, 90.0), (300, 130.0), (1500, 160.0), (4000, 190.0), (4000, 260.0),
                                    (4000, 360.0)])
@pytest.mark.parametrize("kw", [{}, dict(lanes_per_bead=4, step_split=2), dict(nplup=1)])
def test_left_out_minimum_image(n, boxl, kw):
    """Where the molecule's extent shows that the minimum image is the identity,
    for every pair or for the listed ones, it is left out.  Contexts that rebuild
    their lists rarely (nnlup > 200) keep it to a quarter of the box: over the
    steps before either rebuilds them the results are the same bits, and the
    lists equal the oracle's.  Boxes below, about and above twice the extent,
    and ones the molecule reaches across."""
    m = mol_of(n, 500 + n)
    outs = []
    for nnlup in (50, 1000):
        p = engine.baseline_params(**{**dict(boxl=boxl, nnlup=nnlup), **kw})
        with engine.plain(m, m.xyz, p, T=0.6) as e:
            _, (nri, nrj), _, (opi, opj) = oracle_lists(m, m.xyz, p, boxl)
            assert pairset(*e.list_pairs(0, 1)[:2]) == pairset(nri, nrj)
            assert pairset(*e.list_pairs(0, 3)[:2]) == pairset(opi, opj)
            e.step(45)
            outs.append(state(e))
    same(*outs)
