"""Rules of programmatic dependent launch that the compiler does not check, read
from the kernels' source: a kernel that waits for its predecessor
(griddepcontrol.wait, pdl_wait()) takes no data as const __restrict__, and no
thread of it returns before it has waited."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sop_gb300", "csrc")


def source(name):
    txt = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", txt)


def kernels(txt):
    """(name, parameters, body) of every __global__ function."""
    out = []
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\s*\([^{;]*?\)\s*)?(\w+)\s*\(", txt):
        k, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(txt[k], 0)
            k += 1
        params = txt[m.end():k - 1]
        b = txt.index("{", k)
        e, depth = b + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(txt[e], 0)
            e += 1
        out.append((m.group(1), params, txt[b:e]))
    return out


FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu"))
WAITING = [(f, name, params, body) for f in FILES for name, params, body in kernels(source(f))
           if "pdl_wait()" in body]


def test_kernels_are_found():
    names = {name for _, name, _, _ in WAITING}
    assert {"k_step", "k_finish", "k_pl", "k_step_tile", "k_pl_tile", "k_pair_step", "k_advance",
            "k_energy_final", "k_observables_final", "k_energy_lists_final"} <= names


@pytest.mark.parametrize("f,name,params", [w[:3] for w in WAITING], ids=[w[1] for w in WAITING])
def test_waiting_kernels_take_nothing_as_const_restrict(f, name, params):
    for p in params.split(","):
        assert not ("const" in p and "__restrict__" in p), (f, name, p)


@pytest.mark.parametrize("f", ["step_force.cuh", "step_dev.cuh", "lists_dev.cuh", "kernels_tile.cu"])
def test_code_of_waiting_kernels_reads_nothing_as_const_restrict(f):
    assert not re.search(r"const[\w\s]*\*\s*__restrict__", source(f))


@pytest.mark.parametrize("f,name,body", [(w[0], w[1], w[3]) for w in WAITING],
                         ids=[w[1] for w in WAITING])
def test_no_thread_returns_before_the_wait(f, name, body):
    """A grid all of whose threads returned first would complete before the
    kernel it follows, and the kernels after it would not wait for that one."""
    assert not re.search(r"\breturn\b", body[:body.index("pdl_wait()")]), (f, name)
