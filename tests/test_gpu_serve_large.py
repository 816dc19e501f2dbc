"""A served context that holds more than 65,536 bead slots (4 lanes a bead, two
kernels) and, as its jobs finish, fewer (8 lanes, then 16, one kernel): every
job's result is the bits of its run alone and of a context that never holds that
many."""
import ctypes

import numpy as np
import pytest

from sop_gb300 import engine, system

pytestmark = pytest.mark.gpu

N, JOBS = 1500, 48     # 72,000 beads together


def form(srv):
    lanes, f = ctypes.c_int(), ctypes.c_int()
    assert engine.lib().sop_step_form(srv.h, ctypes.byref(lanes), ctypes.byref(f)) == engine.SOP_OK
    return lanes.value, f.value


def test_above_and_below_65536_slots():
    p = engine.baseline_params(boxl=12000.0)
    mols = [system.generate(N, 50 + k) for k in range(4)]

    def job(k):
        """Molecule, start and steps of job k: the first jobs, in the lowest slots,
        go on longest."""
        m = mols[k % 4]
        return m, m.extended_xyz() if k % 3 == 1 else m.xyz, 260 if k < 8 else 160 if k < 40 else 60

    with engine.Server(p, 600 << 20, N) as srv:
        assert srv.stats()["bead_capacity"] > N * JOBS
        ids = []
        for k in range(JOBS):
            m, x, steps = job(k)
            ids.append(srv.submit(m, x, steps, 0.6, traj=k))
        forms = []
        while True:
            s = srv.stats()
            if not s["queued"] and not s["active"]:
                break
            srv.advance(1)
            forms.append(form(srv))
        assert set(forms) == {(4, 2), (8, 1), (16, 1)} and forms[0] == (4, 2)
        many = [srv.result(i) for i in ids]
    for k in (0, 7, 8, 25, 39, 40, 47):
        m, x, steps = job(k)
        with engine.Server(p, 64 << 20, N) as srv:
            i = srv.submit(m, x, steps, 0.6, traj=k)
            srv.advance(1)
            assert form(srv) == (16, 1)
            srv.run_until_idle()
            few = srv.result(i)
        with engine.plain(m, x, p, T=0.6, traj=k, nsteps=steps) as e:
            e.step(steps)
            d = e.download()
            alone = dict(unc_pos=d["unc_pos"], vel=d["vel"], energy=e.energy())
        assert many[k]["steps"] == few["steps"] == steps
        assert many[k]["status"] == few["status"] == engine.MOL_DONE
        for q in ("unc_pos", "vel", "energy"):
            np.testing.assert_array_equal(many[k][q], few[q])
            np.testing.assert_array_equal(many[k][q], alone[q])
