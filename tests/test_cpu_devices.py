"""Contexts on a device that is not the calling thread's current one, on a stand-in
for the CUDA runtime (fake_cudart.c: two devices, launches into a foreign stream
refused): every entry point works from any current device, leaves it as it was and
allocates on the context's own."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

PROGRAM = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, %r)
from sop_gb300 import engine, system
fake = ctypes.CDLL(None)

def current(d=None):
    c = ctypes.c_int(-1)
    if d is None:
        fake.cudaGetDevice(ctypes.byref(c))
        return c.value
    fake.cudaSetDevice(d)

m = system.generate(60, 0)
big = system.generate(9000, 1)
p = engine.baseline_params(device=1, **%r)
fake.fake_expect(1)
e = engine.Engine(p)
e.add(m, m.xyz, nsteps=5)
e.add(big, big.xyz)
e.commit()
srv = engine.Server(p, 64 << 20, 500)
total = m.n + big.n
out = np.empty((total, 3), np.float32)

def restore():
    e.restore(0, e.checkpoint(0))

def copy_all():
    e.download_wait(e.download_all_async(out))

def serve():
    srv.submit(m, m.xyz, 100)
    srv.advance(2)

calls = dict(
    staged=e.staged, restore=restore, download=lambda: [e.download(k) for k in (0, 1)], status=lambda: e.status(0),
    energy=lambda: e.energy(1), observables=lambda: e.observables(0),
    upload=lambda: [e.upload_state(k, q.xyz, vel=np.zeros_like(q.xyz)) for k, q in ((0, m), (1, big))],
    step=lambda: e.step(73), step_async=lambda: e.step_async(20), sync=e.sync,
    stages=lambda: [e.launch_stage(k, 0) for k in range(4)], neighbour_list=e.update_neighbor_list,
    pair_list=e.update_pair_list, force=e.force_eval,
    noise=lambda: [e.set_noise(np.zeros((total, 3), np.float32)), e.step(3), e.set_noise(None)],
    lists=lambda: [e.list_pairs(0, k) for k in range(4)], sizes=e.list_sizes,
    download_all=lambda: e.download_all(out), copy_all=copy_all, serve=serve,
    barrier=lambda: e.check_step_barrier(0, 0.1))
for name, call in calls.items():
    current(0)
    n = fake.fake_launches()
    call()
    assert current() == 0, name
    assert fake.fake_foreign_mallocs() == 0, name
e.close()
print("ok", fake.fake_launches())
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fake") / "fake_cudart.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-w", "-o", so, os.path.join(HERE, "fake_cudart.c")], check=True)
    return so


@pytest.mark.parametrize("kw", [{}, dict(nplup=1), dict(step_split=2, lanes_per_bead=4)])
def test_entry_points_from_another_current_device(fake, kw):
    r = subprocess.run([sys.executable, "-c", PROGRAM % (ROOT, kw)], capture_output=True, text=True,
                       env={**os.environ, "LD_PRELOAD": fake}, timeout=120)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stderr[-2000:]
