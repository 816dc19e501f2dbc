"""Block-wide FP64 sums of the energies and observables at the edges of their
blocks: one partly filled block, exactly full blocks, one bead or entry more,
and more partial sums than the final block has threads.  Against FP64 on the
same coordinates and lists, with the tolerances of the energy and observables
parity tests (FP32 terms, FP64 sums)."""
import numpy as np
import pytest

from helpers import att_sel
from oracle import pyoracle as O
from sop_gb300 import engine, system

pytestmark = pytest.mark.gpu

ENERGY_RTOL = 2e-5


@pytest.mark.parametrize("n", [3, 127, 128, 129, 257, 33000])   # 128 beads a block, 256 partials
def test_energy_and_observables_at_block_edges(n):
    mol = system.generate(n, 70 + n % 100, (0.7, 1.3))
    rng = np.random.default_rng(n)
    x = (mol.xyz + rng.normal(0.0, 0.2, mol.xyz.shape)).astype(np.float32)
    v = rng.normal(0.0, 0.8, x.shape).astype(np.float32)
    with engine.plain(mol, x, engine.baseline_params(), vel=v) as e:
        t, ob = e.energy(), e.observables()
        pai, paj, _ = e.list_pairs(0, 2)
        pri, prj, _ = e.list_pairs(0, 3)
    _, eo = O.forces_f64(mol, x, att_sel(mol, pai, paj), pri, prj)
    np.testing.assert_allclose(t[:4], eo, rtol=ENERGY_RTOL, atol=1e-6)
    oo = O.observables(mol, x, v)
    assert ob["contct_nat"] == oo["contct_nat"]
    # Rg^2 from the moments of the unwrapped coordinates (the oracle's pair sum
    # takes the minimum image, which differs past half the box: 33,000 beads)
    x64 = x.astype(np.float64)
    oo["rgsq"] = (x64 ** 2).sum(1).mean() - (x64.mean(0) ** 2).sum()
    for k in ("Q", "rgsq", "kinT"):
        assert ob[k] == pytest.approx(oo[k], rel=1e-9, abs=1e-12)


@pytest.mark.parametrize("pairs", [0, 1, 1023, 1024, 1025, 300001])   # 1,024 entries a block
def test_noalloc_energy_at_block_edges(pairs):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(pairs)
    n = 1500
    x = rng.uniform(0.0, 60.0, (n, 3)).astype(np.float32)
    i = rng.integers(0, n, pairs).astype(np.int32)
    j = ((i + rng.integers(1, n, pairs)) % n).astype(np.int32)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (x, i, j)]
    px, pi, pj = (d.data_ptr() for d in dev)
    lists = engine.EnergyLists(n, px, None, 0, None, None, None, 0, None, None, 0, None, None,
                               None, None, pairs, pi if pairs else None, pj if pairs else None)
    out = torch.full((5,), float("nan"), dtype=torch.float64, device="cuda")
    engine.energy_noalloc(engine.baseline_params(), lists, out.data_ptr(), 0)
    torch.cuda.synchronize()
    u3 = (3.8 ** 2 / ((x[j].astype(np.float64) - x[i]) ** 2).sum(1)) ** 3
    want = np.array([0.0, 0.0, 0.0, (u3 * u3 + u3).sum()])
    got = out.cpu().numpy()
    np.testing.assert_allclose(got[:4], want, rtol=ENERGY_RTOL, atol=1e-12)
    assert got[4] == got[:4].sum()
