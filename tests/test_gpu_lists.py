"""The cell binning's two paths -- one block per molecule in shared memory, and
the chain of kernels for molecules past 8,192 beads -- at the sizes where they
change: the all-pairs grid of up to 96 beads, 256 and 1,024 threads, the
largest molecule of a block, both paths in one context, contexts on either
side of 16,384 bead slots (a warp or 8 lanes per bead, the attractive list in
the build or by itself).  Lists equal the oracle's as sets."""
import numpy as np
import pytest

from helpers import oracle_lists, pairset
from sop_gb300 import engine, system

pytestmark = pytest.mark.gpu


def perturbed(n, seed, two_types):
    mol = system.generate(n, seed)
    rng = np.random.default_rng(seed)
    if two_types:
        mol.types = rng.integers(1, 3, n).astype(np.int32)
    return mol, (mol.xyz + rng.normal(0.0, 0.3, mol.xyz.shape)).astype(np.float32)


def keys(i, j, n):
    a, b = np.minimum(i, j).astype(np.int64), np.maximum(i, j).astype(np.int64)
    return np.sort(a * n + b)


@pytest.mark.parametrize("sizes,two_types", [
    ((3, 96, 97), False), ((33, 2048, 100), True), ((2049,), False), ((8192, 65), False),
    ((8193, 64), True), ((300, 9000, 128, 7500, 97), False), ((1200,) * 14, False)])
def test_binning_paths(sizes, two_types):
    p = engine.baseline_params()
    made = [perturbed(n, 100 + 7 * k + n % 50, two_types) for k, n in enumerate(sizes)]
    with engine.Engine(p) as e:
        for k, (mol, x) in enumerate(made):
            e.add(mol, x, T=0.6, traj=k)
        e.commit()
        for k, (mol, x) in enumerate(made[:6]):
            nl_att, (nri, nrj), pl_att, (opi, opj) = oracle_lists(mol, x, p)
            ai, aj, _ = e.list_pairs(k, 0)
            ri, rj, _ = e.list_pairs(k, 1)
            pri, prj, _ = e.list_pairs(k, 3)
            assert pairset(ai, aj) == pairset(mol.nat_i[nl_att], mol.nat_j[nl_att])
            np.testing.assert_array_equal(keys(ri, rj, mol.n), keys(nri, nrj, mol.n))
            np.testing.assert_array_equal(keys(pri, prj, mol.n), keys(opi, opj, mol.n))


def test_far_apart_beads_without_bonds():
    """Beads scattered on a line far longer than a chain of them could be: the
    grid's rounds have to coarsen the cells to the molecule's cap (a fixed
    number of them stops short on one axis)."""
    n = 200
    base = system.generate(n, 5)
    e0, f0 = np.empty(0, np.int32), np.empty(0, np.float32)
    mol = system.Molecule(n, base.xyz, e0, e0, f0, e0, e0, e0, f0, e0, e0, f0, f0)
    x = np.zeros((n, 3), np.float32)
    x[:, 0] = np.sort(np.random.default_rng(3).uniform(0.0, 9.0e5, n)).astype(np.float32)
    x[1::2, 0] = x[::2, 0] + 20.0
    x[:, 1] = np.arange(n) % 3
    p = engine.baseline_params(boxl=1.0e6)
    with engine.plain(mol, x, p) as e:
        ri, rj, _ = e.list_pairs(0, 1)
    _, (nri, nrj), _, _ = oracle_lists(mol, x, p, 1.0e6)
    assert pairset(ri, rj) == pairset(nri, nrj)


def test_served_molecules_in_other_slots():
    """Jobs submitted twice to one server: the second time molecule slots and
    bead ranges pair up in another order (free slots come last in, first out,
    bead ranges first fit), so the molecules' cells have to lie apart whatever
    slot and range they have.  Same results both times."""
    p = engine.baseline_params(boxl=12000.0)
    sizes = (400, 60, 1200, 97, 700, 33, 2500, 150)
    mols = [system.generate(n, 300 + n) for n in sizes]
    with engine.Server(p, 256 << 20, 2500) as srv:
        runs = []
        for _ in range(3):
            ids = [srv.submit(m, m.extended_xyz() if k % 2 else m.xyz, nsteps=55 + 10 * k, T=0.6,
                              traj=k) for k, m in enumerate(mols)]
            srv.run_until_idle()
            runs.append([srv.result(i) for i in ids])
    for again in runs[1:]:
        for a, b in zip(runs[0], again):
            assert a["status"] == b["status"] == engine.MOL_DONE
            for key in ("unc_pos", "vel", "energy"):
                np.testing.assert_array_equal(a[key], b[key])
