"""States to and from the host: what is uploaded is read back bit for bit at
the sizes where the way through pinned memory ends, the other molecules'
states stay, an upload whose lists overflow their rows grows them, and jobs
whose rows and results exceed the served engine's transfer buffer come out as
they do alone."""
import numpy as np
import pytest

from sop_gb300 import engine, system

pytestmark = pytest.mark.gpu


def state(n, seed):
    rng = np.random.default_rng(seed)
    return [rng.normal(0.0, s, (n, 3)).astype(np.float32) for s in (1.0, 5.0, 0.7)]


@pytest.mark.parametrize("n", [3, 257, 8192, 8193])
def test_states_come_back(n):
    m, other = system.generate(n, 5), system.generate(40, 6)
    d, vel, vel2 = state(n, 7)
    unc, pos = m.xyz + d, m.xyz - d
    with engine.Engine(engine.baseline_params()) as e:
        e.add(other, other.xyz)
        e.add(m, m.xyz)
        e.add(other, other.xyz)
        e.commit()
        e.step(3)  # an odd step: the second coordinate buffer
        before = [e.download(k) for k in (0, 2)]
        e.upload_state(1, unc, pos=pos, vel=vel)
        got = e.download(1)
        for k, want in (("unc_pos", unc), ("pos", pos), ("vel", vel)):
            assert np.array_equal(got[k], want)
        e.upload_state(1, m.xyz)  # positions alone: the velocities stay
        got = e.download(1)
        for k, want in (("unc_pos", m.xyz), ("pos", m.xyz), ("vel", vel)):
            assert np.array_equal(got[k], want)
        assert e.status(1)[1] == 3
        e.upload_state(1, m.xyz, vel=vel2)
        assert np.array_equal(e.download(1)["vel"], vel2)
        for k, want in zip((0, 2), before):
            got = e.download(k)
            assert all(np.array_equal(got[a], want[a]) for a in want)
        assert np.array_equal(e.download_all()[40:40 + n], m.xyz)


def test_upload_grows_the_rows():
    m = system.generate(1500, 9)
    got = []
    for rows in (0, 64):
        p = engine.baseline_params(boxl=12000.0, nl_rows=rows)
        with engine.plain(m, m.extended_xyz(), p) as e:
            e.step(20)
            e.upload_state(0, m.xyz)
            got.append((e.download(0)["force"], e.energy(0), e.list_sizes()))
            e.step(60)
            got[-1] += (e.download(0)["unc_pos"],)
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert got[0][2] == got[1][2] and np.array_equal(got[0][3], got[1][3])


def test_jobs_past_the_buffer():
    """60 jobs of 700 beads: about 11 MB of rows that arrive in one round and
    leave in another; the buffer holds 8 MB."""
    m = system.generate(700, 11)
    p = engine.baseline_params(boxl=12000.0)

    def serve(trajs):
        with engine.Server(p, 1 << 29, 1000) as srv:
            ids = [srv.submit(m, m.xyz, nsteps=50, T=0.6, traj=t) for t in trajs]
            srv.run_until_idle()
            return [srv.result(i) for i in ids]

    together = serve(range(60))
    for t in (0, 23, 59):
        one, = serve([t])
        for k in ("unc_pos", "vel", "energy", "status", "steps"):
            assert np.array_equal(together[t][k], one[k])


@pytest.mark.parametrize("extra", [{}, dict(nplup=1), dict(nnlup=30, lanes_per_bead=4)])
def test_period_graphs(extra):
    """A context that goes on stepping takes graphs of a whole list period: the
    same bits as blocks of 10, from any phase."""
    ms = [system.generate(n, 13 + n) for n in (90, 300)]
    got = []
    for gs in (0, 10):
        p = engine.baseline_params(graph_steps=gs, **extra)
        with engine.Engine(p) as e:
            for k, m in enumerate(ms):
                e.add(m, m.xyz, traj=k, nsteps=640 if k else -1)
            e.commit()
            for n in (405, 5, 100, 49, 161):
                e.step(n)
            got.append([e.download(0), e.download(1), e.status(0), e.status(1), e.list_sizes()])
    for a, b in zip(got[0][:2], got[1][:2]):
        assert all(np.array_equal(a[k], b[k]) for k in a)
    assert got[0][2:] == got[1][2:]
