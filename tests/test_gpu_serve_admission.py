"""A served round that fails while it admits (a resumed job whose checkpoint does
not hold): the error is reported, the jobs admitted before it in the same round are
in their slots with their own state, and the failing job takes no slot or range."""
import numpy as np
import pytest

from sop_gb300 import engine, system

pytestmark = pytest.mark.gpu


def corrupt(blob):
    """The checkpoint with its last list entry past the molecule's beads."""
    return blob[:-4] + np.int32(1 << 20).tobytes()


def start_of(blob, n):
    """The step and the coordinates of a checkpoint."""
    return np.frombuffer(blob, np.int64, 1, 16)[0], np.frombuffer(blob, np.float32, 4 * n, 64).reshape(n, 4)[:, :3]


def test_jobs_admitted_before_a_failure_keep_their_state():
    p = engine.baseline_params(boxl=12000.0)
    m1, m2 = system.generate(700, 32), system.generate(250, 33)
    with engine.Server(p, 64 << 20, 4000) as srv:
        # a first job leaves its slot's old step and state behind
        srv.submit(m1, m1.xyz, 100, 0.6, traj=1)
        srv.advance(3)
        j = srv.submit(m1, m1.xyz, 400, 0.6, traj=1)
        srv.advance(3)
        blob = srv.checkpoint(j)
        srv.run_until_idle()
    with engine.Server(p, 64 << 20, 4000) as srv:
        first = srv.submit(m1, m1.extended_xyz(), 50, 0.6, traj=3)
        srv.run_until_idle()
        assert srv.finished() == [first]
        ok = srv.submit(m2, m2.xyz, 50, 0.5, traj=2)
        srv.resume(m1, corrupt(blob), 400, 0.6, traj=1)
        # more rounds than the pools hold ranges of the failing job
        assert 40 * m1.n > srv.stats()["bead_capacity"]
        for _ in range(40):
            with pytest.raises(engine.SopError, match="corrupt checkpoint"):
                srv.advance(1)
            s = srv.stats()
            assert (s["active"], s["queued"]) == (1, 1) and srv.finished() == []
            step, x = start_of(srv.checkpoint(ok), m2.n)
            assert step == -p.nnlup
            np.testing.assert_array_equal(x, m2.xyz)
