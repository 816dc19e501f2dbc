"""The work a user of sop_gb300 has it do, as cases that can be timed and checked.

Every case goes through the package's public entry points (sop_gb300.engine):

  steps     Langevin steps of the molecules a context holds and a read of the
            new state: one molecule (Engine), a batch in one context (Engine)
            or an ensemble in two contexts (Ensemble)
  evaluate  forces, energies and observables of given coordinates
  serve     a round of jobs through the served engine (Server)
  energy    the energy of caller-owned device lists (energy_noalloc)

Structures come from the package's synthetic generator, seeded by the case's
seed, with the force field, list cut-offs and cadences of bench.py and of the
tests.  exact() restates the method in 64 bits with plain torch: forces,
Langevin steps, the Philox noise stream and the list cut-offs.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from sop_gb300 import engine, system

# ------------------------------------------------------------------ the cases


def listed() -> list[dict]:
    return [
        # the smallest call: one conformation of a short chain rescored
        # (upload, lists, forces, energies), all launches and latency
        dict(name="evaluate 60", kind="evaluate", beads=60, types=1, cutoffs="absolute"),
        # the 128-bead plain workload of bench.py, a frame every 100 steps
        dict(name="steps 128", kind="steps", beads=128, steps=100, start="native", types=1,
             cutoffs="absolute", eps=0),
        # two bead types in the reference's own settings: cut-offs by factor,
        # pair list before every step, its time step (an odd size)
        dict(name="steps 1531 reference settings", kind="steps", beads=1531, steps=50,
             start="native", types=2, cutoffs="factor", eps=0),
        # the 4,000-bead plain workload of bench.py
        dict(name="steps 4000", kind="steps", beads=4000, steps=100, start="native", types=1,
             cutoffs="absolute", eps=0),
        # unfolding: the same from the fully extended chain (short rows, a long
        # row of cells, a box that holds 15,200 A)
        dict(name="steps 4000 extended", kind="steps", beads=4000, steps=100, start="extended",
             types=1, cutoffs="absolute", eps=0),
        # the 50,000-bead plain workload of bench.py (an epsilon per contact)
        dict(name="steps 50000", kind="steps", beads=50000, steps=50, start="native", types=1,
             cutoffs="absolute", eps=1),
        # a small overdamped batch in one context, 6-power repulsion
        dict(name="batch 37 overdamped", kind="batch", molecules=37, low=50, high=1200, steps=50,
             contexts=1, overdamped=1),
        # bench.py's headline: 512 trajectories of 60-1,500 beads, two contexts
        dict(name="ensemble 512", kind="batch", molecules=512, low=60, high=1500, steps=50,
             contexts=2, overdamped=0),
        # one large conformation rescored: list rebuild, forces, energies
        dict(name="evaluate 50000", kind="evaluate", beads=50000, types=1, cutoffs="absolute"),
        # a round of folding and unfolding jobs through the served engine
        dict(name="serve 64", kind="serve", jobs=64, low=50, high=3000, steps_low=50,
             steps_high=400),
        # energy of the caller's own lists, in a loop that may not allocate
        dict(name="energy lists 20000", kind="energy", beads=20000, types=1),
    ]


def _log_int(rng, low: float, high: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng) -> dict:
    kind = rng.choice(["steps", "steps", "steps", "batch", "batch", "evaluate", "serve", "energy"])
    if kind == "steps":
        types = rng.choice([1, 1, 1, 2])
        extended = types == 1 and rng.random() < 0.25
        n = _log_int(rng, 20, 2500 if types == 2 else 20000 if extended else 50000)
        steps = rng.randint(11, 100) if n < 20000 else rng.randint(11, 50)
        return dict(kind=kind, beads=n, steps=steps, start="extended" if extended else "native",
                    types=types, cutoffs="factor" if types == 2 or rng.random() < 0.25 else "absolute",
                    eps=rng.randint(0, 1))
    if kind == "batch":
        low, overdamped = rng.randint(20, 200), rng.choice([0, 0, 1])
        return dict(kind=kind, molecules=_log_int(rng, 2, 80 if overdamped else 300), low=low,
                    high=low + _log_int(rng, 10, 1300), steps=rng.randint(11, 50),
                    contexts=rng.randint(1, 2), overdamped=overdamped)
    if kind == "evaluate":
        types = rng.choice([1, 1, 2])
        return dict(kind=kind, beads=_log_int(rng, 20, 2500 if types == 2 else 50000), types=types,
                    cutoffs=rng.choice(["absolute", "factor"]))
    if kind == "serve":
        low = rng.randint(50, 200)
        return dict(kind=kind, jobs=_log_int(rng, 4, 64), low=low,
                    high=low + _log_int(rng, 50, 2800), steps_low=50, steps_high=rng.randint(60, 400))
    types = rng.choice([1, 1, 2])
    return dict(kind=kind, beads=_log_int(rng, 50, 2500 if types == 2 else 40000), types=types)


# --------------------------------------------------------- structures, settings

_SIGMA = {(1, 1): 3.8, (1, 2): 5.4, (2, 1): 5.4, (2, 2): 7.0}


def _molecule(n: int, seed: int, types: int = 1, eps: int = 0) -> system.Molecule:
    """A synthetic structure; with two types, natives are the pairs below the
    reference's native cut-off of their types (system.RCUT_NAT)."""
    mol = system.generate(n, seed, (0.7, 1.3) if eps else None)
    if types == 1:
        return mol
    rng = np.random.default_rng(seed + 77)
    ty = np.where(rng.random(mol.n) < 0.3, 2, 1).astype(np.int32)
    ii, jj = np.triu_indices(mol.n, 3)
    d = np.linalg.norm(mol.xyz[jj].astype(np.float64) - mol.xyz[ii], axis=1).astype(np.float32)
    nat = d < system.RCUT_NAT.astype(np.float32)[ty[ii], ty[jj]]
    ni, nj, nr = ii[nat].astype(np.int32), jj[nat].astype(np.int32), d[nat]
    ne = rng.uniform(0.7, 1.3, len(ni)).astype(np.float32) if eps else np.ones(len(ni), np.float32)
    return system.Molecule(mol.n, mol.xyz, mol.bond_i, mol.bond_j, mol.bond_r0, mol.ang_i,
                           mol.ang_j, mol.ang_k, mol.ang_r, ni, nj, nr, ne, types=ty, seed=seed)


def _around(xyz: np.ndarray, sigma: float, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    return (xyz + rng.normal(0.0, sigma, xyz.shape)).astype(np.float32)


def _settings(case: dict) -> dict:
    """The parameters of a case as engine.default_params keywords."""
    if case["kind"] == "batch" and case["overdamped"]:
        return dict(_ABSOLUTE, integrator=1, h=5.0e-4, nplup=1, rep6=1)
    if case["kind"] == "serve":
        return dict(_ABSOLUTE, boxl=12000.0)
    if case.get("start") == "extended":
        return dict(_ABSOLUTE, boxl=max(40000.0, 8.0 * case["beads"]))
    if case.get("cutoffs") == "factor":
        return {}
    return dict(_ABSOLUTE)


# engine.baseline_params: 32 / 16 A lists every 50 / 10 steps, h = zeta = 0.05
_ABSOLUTE = dict(h=0.05, zeta=0.05, nl_att_fac=0.0, nl_att_abs=32.0, nl_rep_fac=0.0,
                 nl_rep_abs=32.0, pl_att_fac=0.0, pl_att_abs=16.0, pl_rep_fac=0.0,
                 pl_rep_abs=16.0, nnlup=50, nplup=10)


def _trajectories(case: dict, seed: int) -> list[dict]:
    """The molecules of a steps / batch / serve case: structure, start,
    temperature, Philox stream and (serve) step budget.  Sizes depend on the
    case alone, structures on the seed too."""
    if case["kind"] == "steps":
        m = _molecule(case["beads"], seed, case["types"], case["eps"])
        x = m.extended_xyz() if case["start"] == "extended" else _around(m.xyz, 0.05, seed)
        return [dict(mol=m, x=x, T=0.6, traj=seed % 1000003, nsteps=-1)]
    count = case["molecules"] if case["kind"] == "batch" else case["jobs"]
    ns, ts = system.ensemble_spec(count, case["low"], case["high"], 0.5, 0.8, 4)
    out = []
    for k, (n, t) in enumerate(zip(ns, ts)):
        m = _molecule(int(n), seed + 7919 * k)
        x, nsteps = _around(m.xyz, 0.05, seed + 7919 * k), -1
        if case["kind"] == "serve":
            lo, hi = math.log(case["steps_low"]), math.log(case["steps_high"])
            nsteps = int(round(math.exp(lo + (hi - lo) * (k * 0.618034 % 1.0))))
            if k % 2:
                x = m.extended_xyz()
        out.append(dict(mol=m, x=x, T=float(t), traj=(seed + k) % 1000003, nsteps=nsteps))
    return out


def prepare(case: dict, seed: int):
    kind, params = case["kind"], engine.default_params(**_settings(case))
    if kind == "steps" or kind == "batch":
        trajs = _trajectories(case, seed)
        two = kind == "batch" and case["contexts"] > 1
        e = engine.Ensemble(params, parts=2) if two else engine.Engine(params)
        for t in trajs:
            e.add(t["mol"], t["x"], T=t["T"], traj=t["traj"])
        e.commit()
        return dict(case=case, e=e)
    if kind == "serve":
        # pools for about 200,000 beads
        srv = engine.Server(params, 1 << 30, int(case["high"]))
        return dict(case=case, srv=srv, jobs=_trajectories(case, seed))
    m = _molecule(case["beads"], seed, case["types"], 1)
    x = _around(m.xyz, 0.2, seed + 1)
    if kind == "evaluate":
        v = np.random.default_rng(seed + 2).normal(0.0, 0.77, x.shape).astype(np.float32)
        # T = 0: no noise force, so the force read back is the conservative one
        return dict(case=case, e=engine.plain(m, m.xyz, params, T=0.0), x=x, v=v)
    s = _System([dict(mol=m, x=x)], _settings(dict(case, cutoffs="absolute")))
    s.rebuild(s.x)
    dev = s.x.device
    types = torch.as_tensor(m.types, device=dev)
    t = dict(x=torch.as_tensor(x, device=dev), ty=types,
             bi=s.bi.int(), bj=s.bj.int(), br=s.br.float(), ai=s.ai.int(), ak=s.ak.int(),
             ni=s.pni.int(), nj=s.pnj.int(), nr=s.pnr.float(), ne=s.pne.float(),
             ri=s.pri.int(), rj=s.prj.int())
    lists = engine.EnergyLists(m.n, t["x"].data_ptr(), t["ty"].data_ptr(), len(t["bi"]),
                               t["bi"].data_ptr(), t["bj"].data_ptr(), t["br"].data_ptr(),
                               len(t["ai"]), t["ai"].data_ptr(), t["ak"].data_ptr(), len(t["ni"]),
                               t["ni"].data_ptr(), t["nj"].data_ptr(), t["nr"].data_ptr(),
                               t["ne"].data_ptr(), len(t["ri"]), t["ri"].data_ptr(),
                               t["rj"].data_ptr())
    return dict(case=case, params=params, lists=lists, keep=t,
                out=torch.empty(5, dtype=torch.float64, device=dev))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "steps":
        state["e"].step(case["steps"])
        d = state["e"].download(0)
        status, step = state["e"].status(0)
        return [d["unc_pos"], d["pos"], d["vel"], d["force"], status, step]
    if kind == "batch":
        state["e"].step(case["steps"])
        return [state["e"].download_all()]
    if kind == "evaluate":
        e = state["e"]
        e.upload_state(0, state["x"], vel=state["v"])
        energy, obs, d = e.energy(0), e.observables(0), e.download(0)
        return [energy, d["force"], obs["Q"], obs["rgsq"], obs["kinT"], obs["contct_nat"]]
    if kind == "serve":
        srv = state["srv"]
        ids = [srv.submit(j["mol"], j["x"], nsteps=j["nsteps"], T=j["T"], traj=j["traj"])
               for j in state["jobs"]]
        srv.run_until_idle()
        srv.finished()
        res = [srv.result(i) for i in ids]
        return [np.concatenate([r["unc_pos"] for r in res]), np.concatenate([r["vel"] for r in res]),
                np.stack([r["energy"] for r in res]),
                np.array([[r["status"], r["steps"]] for r in res], np.int64)]
    stream = torch.cuda.current_stream().cuda_stream
    engine.energy_noalloc(state["params"], state["lists"], state["out"].data_ptr(), stream)
    return [state["out"]]


# ----------------------------------------------------------- what it takes

# Pairs of a bead in a folded synthetic structure (each counted once): within
# the 16 A pair list, within the 32 A neighbour list, natives; in the factor
# settings (2.5 sigma = 9.5 A) and on the extended chain far fewer.
_PAIRS = {"absolute": 20.0, "factor": 3.0, "extended": 2.0}
_NL_PAIRS, _NATIVES = 90.0, 2.8


def _per_step_flops(n: float, pairs: float) -> float:
    # 24 a repulsive pair, 60 a native, 45 a bond and a soft-sphere pair
    # together; noise, velocity and position update 130 a bead
    return n * (24.0 * pairs + 60.0 * _NATIVES + 45.0 + 130.0)


def work(case: dict) -> dict:
    """Coordinates, increments and topology read once, the new state written
    once, and the arithmetic of every step's pairs and of the list rebuilds'
    distances (each pair once)."""
    kind = case["kind"]
    if kind == "energy":
        n = case["beads"]
        items = n * (2.0 + _NATIVES + _PAIRS["absolute"])
        return dict(bytes=16.0 * n + 10.0 * items, flops=22.0 * items)
    if kind == "evaluate":
        n = case["beads"]
        near = case["cutoffs"] == "absolute"
        p = min(n / 2.0, _PAIRS[case["cutoffs"]])
        nl = min(n / 2.0, _NL_PAIRS if near else 8.0)
        return dict(bytes=n * (24.0 + 12.0 + 24.0 + 16.0 * _NATIVES),
                    flops=n * (16.0 * nl + 50.0 * p + 260.0))
    if kind == "steps":
        groups = [(case["beads"], case["steps"])]
        where = "extended" if case["start"] == "extended" else case["cutoffs"]
        every = 1 if case["cutoffs"] == "factor" else 10
        out = 48.0
    else:
        count = case["molecules"] if kind == "batch" else case["jobs"]
        ns, _ = system.ensemble_spec(count, case["low"], case["high"], 0.5, 0.8, 4)
        if kind == "serve":
            lo, hi = math.log(case["steps_low"]), math.log(case["steps_high"])
            groups = [(int(n), math.exp(lo + (hi - lo) * (k * 0.618034 % 1.0)))
                      for k, n in enumerate(ns)]
        else:
            groups = [(int(n), case["steps"]) for n in ns]
        where, out = "absolute", 24.0 if kind == "serve" else 12.0
        every = 1 if kind == "batch" and case["overdamped"] else 10
    byts = flops = 0.0
    for n, steps in groups:
        p = min(n / 2.0, _PAIRS[where])
        nl = min(n / 2.0, _NL_PAIRS * _PAIRS[where] / _PAIRS["absolute"])
        byts += n * (36.0 + 20.0 + 12.0 * _NATIVES + out)
        flops += steps * (_per_step_flops(n, p) + 8.0 * n * nl / every)
    return dict(bytes=byts, flops=flops)


# --------------------------------------------------------------- in 64 bits


def _mulhi(a: torch.Tensor, b: int):
    """High and low words of a 32 x 32-bit product (int64 tensors)."""
    low = a * (b & 0xffff)
    hi = (a * (b >> 16) + (low >> 16)) >> 16
    return hi, (a * b) & 0xffffffff


def _normals(bead: torch.Tensor, step: torch.Tensor, traj: torch.Tensor, seed: int) -> torch.Tensor:
    """Philox4x32-10 (Salmon et al., SC'11) keyed by the seed, counter (bead,
    step, trajectory); uniforms (float)r 2^-32 + 2^-33, Box-Muller."""
    c = [bead, step & 0xffffffff, step >> 32, traj]
    k0, k1 = seed & 0xffffffff, seed >> 32
    for _ in range(10):
        h0, l0 = _mulhi(c[0], 0xD2511F53)
        h1, l1 = _mulhi(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
    u = [(r.float() * 2.3283064365386963e-10 + 1.1641532182693481e-10).double() for r in c]
    m0, m1 = torch.sqrt(-2.0 * torch.log(u[0])), torch.sqrt(-2.0 * torch.log(u[2]))
    a0, a1 = 2.0 * math.pi * u[1], 2.0 * math.pi * u[3]
    return torch.stack([m0 * torch.cos(a0), m0 * torch.sin(a0), m1 * torch.cos(a1)], 1)


class _System:
    """Molecules side by side, in 64 bits.  No molecule here comes within a
    cut-off of its own periodic image, so separations need no minimum image."""

    def __init__(self, trajs: list[dict], settings: dict):
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.p = dict(k_bnd=20.0, R0=2.0, eps_ss=1.0, sigma_ss=3.5, eps_rep=1.0, boxl=500.0,
                      h=2.5e-3, zeta=5.0e-2, nl_att_fac=3.2, nl_att_abs=0.0, nl_rep_fac=3.2,
                      nl_rep_abs=0.0, pl_att_fac=2.5, pl_att_abs=0.0, pl_rep_fac=2.5,
                      pl_rep_abs=0.0, nnlup=50, nplup=1, rep6=0, integrator=0, seed=1234)
        self.p.update(settings)
        sizes = [t["mol"].n for t in trajs]
        self.starts = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
        self.n = int(self.starts[-1])

        def join(name, shift, dtype):
            parts = [getattr(t["mol"], name) + (o if shift else 0) for t, o in zip(trajs, self.starts)]
            return torch.as_tensor(np.concatenate(parts).astype(dtype), device=dev)

        self.x = torch.as_tensor(np.concatenate([t["x"] for t in trajs]).astype(np.float64), device=dev)
        self.types = join("types", False, np.int64)
        self.bi, self.bj = join("bond_i", True, np.int64), join("bond_j", True, np.int64)
        self.br = join("bond_r0", False, np.float64)
        self.ai, self.ak = join("ang_i", True, np.int64), join("ang_k", True, np.int64)
        self.ni, self.nj = join("nat_i", True, np.int64), join("nat_j", True, np.int64)
        self.nr, self.ne = join("nat_r0", False, np.float64), join("nat_eps", False, np.float64)
        self.bead = torch.cat([torch.arange(n, device=dev) for n in sizes])
        self.mol = torch.repeat_interleave(torch.arange(len(sizes), device=dev),
                                           torch.as_tensor(sizes, device=dev))
        self.sig = torch.zeros((3, 3), dtype=torch.float64, device=dev)
        for (a, b), v in _SIGMA.items():
            self.sig[a, b] = v
        self.nat_key = torch.sort(self.ni * self.n + self.nj).values

    def _cut(self, which: str, r):
        fac = self.p[which + "_fac"]
        return fac * r if fac > 0 else torch.full_like(r, self.p[which + "_abs"])

    def _d2(self, x, i, j):
        return ((x[j] - x[i]) ** 2).sum(1)

    def neighbours(self, x):
        """The neighbour lists: non-native pairs with |i - j| > 2 (i < j)."""
        rc = float(self._cut("nl_rep", self.sig.max().reshape(1))[0])
        got_i, got_j = [], []
        for a, b in zip(self.starts[:-1], self.starts[1:]):
            rows = max(1, int(5e7 // max(1, b - a)))
            xm = x[a:b].float() - x[a].float()
            for r in range(0, int(b - a), rows):
                xa = xm[r:r + rows]
                d2 = sum((xa[:, None, q] - xm[None, :, q]) ** 2 for q in range(3))
                i, j = torch.nonzero(d2 < (rc + 0.01) ** 2, as_tuple=True)
                i = i + r
                keep = j > i + 2
                got_i.append(i[keep] + a)
                got_j.append(j[keep] + a)
        i, j = torch.cat(got_i), torch.cat(got_j)
        if len(self.nat_key):
            key = i * self.n + j
            at = torch.searchsorted(self.nat_key, key).clamp(max=len(self.nat_key) - 1)
            keep = self.nat_key[at] != key
            i, j = i[keep], j[keep]
        cut = self._cut("nl_rep", self.sig[self.types[i], self.types[j]])
        keep = self._d2(x, i, j) < cut ** 2
        self.nri, self.nrj = i[keep], j[keep]
        keep = self._d2(x, self.ni, self.nj) < self._cut("nl_att", self.nr) ** 2
        self.natt = torch.nonzero(keep).reshape(-1)

    def pairs(self, x):
        i, j = self.nri, self.nrj
        sg = self.sig[self.types[i], self.types[j]]
        keep = self._d2(x, i, j) < self._cut("pl_rep", sg) ** 2
        self.pri, self.prj, self.psg2 = i[keep], j[keep], sg[keep] ** 2
        s = self.natt
        s = s[self._d2(x, self.ni[s], self.nj[s]) < self._cut("pl_att", self.nr[s]) ** 2]
        self.pni, self.pnj, self.pnr, self.pne = self.ni[s], self.nj[s], self.nr[s], self.ne[s]

    def rebuild(self, x):
        self.neighbours(x)
        self.pairs(x)

    def forces(self, x):
        p, f = self.p, torch.zeros_like(x)

        def add(i, j, d, c):
            g = c[:, None] * d
            f.index_add_(0, i, g)
            f.index_add_(0, j, -g)

        d = x[self.bj] - x[self.bi]
        r = d.norm(dim=1)
        dev = r - self.br
        add(self.bi, self.bj, d, p["k_bnd"] * dev / (r * (1.0 - (dev / p["R0"]) ** 2)))
        d = x[self.ak] - x[self.ai]
        add(self.ai, self.ak, d, -6.0 * p["eps_ss"] * p["sigma_ss"] ** 6 / (d ** 2).sum(1) ** 4)
        d = x[self.pnj] - x[self.pni]
        d2 = (d ** 2).sum(1)
        s3 = (self.pnr ** 2 / d2) ** 3
        add(self.pni, self.pnj, d, -12.0 * self.pne / d2 * (s3 * s3 - s3))
        d = x[self.prj] - x[self.pri]
        d2 = (d ** 2).sum(1)
        u3 = (self.psg2 / d2) ** 3
        add(self.pri, self.prj, d,
            -6.0 * p["eps_rep"] / d2 * (u3 if p["rep6"] else 2.0 * u3 * u3 + u3))
        return f

    def energies(self, x):
        """The four terms and their sum, of every molecule: (molecules, 5)."""
        p = self.p
        out = torch.zeros((len(self.starts) - 1, 5), dtype=torch.float64, device=x.device)

        def put(k, i, e):
            out[:, k].index_add_(0, self.mol[i], e)

        dev = (x[self.bj] - x[self.bi]).norm(dim=1) - self.br
        put(0, self.bi, -0.5 * p["k_bnd"] * p["R0"] ** 2 * torch.log1p(-(dev / p["R0"]) ** 2))
        put(1, self.ai, p["eps_ss"] * p["sigma_ss"] ** 6 / self._d2(x, self.ai, self.ak) ** 3)
        s3 = (self.pnr ** 2 / self._d2(x, self.pni, self.pnj)) ** 3
        put(2, self.pni, self.pne * (s3 * s3 - 2.0 * s3))
        u3 = (self.psg2 / self._d2(x, self.pri, self.prj)) ** 3
        put(3, self.pri, p["eps_rep"] * (u3 if p["rep6"] else u3 * u3 + u3))
        out[:, 4] = out[:, :4].sum(1)
        return out

    def run(self, trajs: list[dict], stops: list[int]):
        """Steps every molecule from rest to its own step count; returns
        coordinates, velocities, forces and energies there."""
        p, dev = self.p, self.x.device
        h, z = p["h"], p["zeta"]
        a1, a2 = h * (1.0 - z * h / 2.0), h * h / 2.0
        a3, a4 = (1.0 - h * z / 2.0 + (h * z) ** 2 / 4.0) / h, h / 2.0 * (1.0 - h * z / 2.0)
        if p["integrator"] == 1:
            a1, a2, a3, a4 = 0.0, h / z, 0.0, 0.0
        T = torch.tensor([t["T"] for t in trajs], dtype=torch.float64, device=dev)[self.mol]
        sigma = torch.sqrt(2.0 * T * z / h)[:, None]
        traj = torch.tensor([t["traj"] for t in trajs], device=dev)[self.mol]
        stop = torch.tensor(stops, device=dev)
        x, v = self.x.clone(), torch.zeros_like(self.x)
        out = [torch.zeros_like(x) for _ in range(3)]
        energy = torch.zeros((len(stops), 5), dtype=torch.float64, device=dev)
        incr = None
        ends = set(stops)
        for n in range(max(stops) + 1):
            if n == 0 or n % p["nnlup"] == 0:
                self.rebuild(x)
            elif p["nplup"] <= 1 or n % p["nplup"] == 0:
                self.pairs(x)
            if n:
                x = x + incr
            f = self.forces(x) + sigma * _normals(self.bead, torch.full_like(self.bead, n), traj,
                                                  p["seed"])
            if n:
                v = a3 * incr + a4 * f
            if n in ends:
                here = stop == n
                mask = here[self.mol][:, None]
                out = [torch.where(mask, new, old) for new, old in zip((x, v, f), out)]
                energy = torch.where(here[:, None], self.energies(x), energy)
            incr = a1 * v + a2 * f
        return out[0], out[1], out[2], energy


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("steps", "batch", "serve"):
        trajs = _trajectories(case, seed)
        s = _System(trajs, _settings(case))
        stops = [t["nsteps"] if kind == "serve" else case["steps"] for t in trajs]
        x, v, f, energy = s.run(trajs, stops)
        if kind == "steps":
            box = s.p["boxl"]
            return [x, x - box * torch.round(x / box), v, f, None, None]
        if kind == "batch":
            return [x]
        return [x, v, energy, None]
    m = _molecule(case["beads"], seed, case["types"], 1)
    x = _around(m.xyz, 0.2, seed + 1)
    s = _System([dict(mol=m, x=x)], _settings(case if kind == "evaluate" else
                                              dict(case, cutoffs="absolute")))
    s.rebuild(s.x)
    if kind == "energy":
        return [s.energies(s.x)[0]]
    v = np.random.default_rng(seed + 2).normal(0.0, 0.77, x.shape).astype(np.float32)
    near = torch.sqrt(s._d2(s.x, s.ni, s.nj)) / s.nr < 1.25
    contacts = float(near.sum())
    mean = s.x.mean(0)
    return [s.energies(s.x)[0], s.forces(s.x), contacts / max(1, len(s.ni)),
            float((s.x ** 2).sum(1).mean() - (mean ** 2).sum()),
            float((v.astype(np.float64) ** 2).sum() / (3.0 * m.n)), None]
