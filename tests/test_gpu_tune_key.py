"""Tuned lane counts are reused for meshes like the one they were timed on, and
not for one with work items of another length or for a batch.  In a process of its
own, so that no other test has tuned anything."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = """
import sys
sys.path.insert(0, %r)
from nextgen_b200 import cases, cgx
from nextgen_b200.meshgen import PeriodicBoxMesh

prm = cases.tgv_params()

def launches(dims):
    m = PeriodicBoxMesh(*dims, L=tuple(float(n) for n in dims), jitter=0.25, seed=3)
    s = cgx.Solver(cgx.Mesh(m, device=0), prm)
    s.set_state_primitive(*cases.tgv_state(m.x_cv[: m.ncv], prm))
    n = s.launch_count()
    s.initComplete()
    return s.launch_count() - n

# 32768 and 33792 cells in items of 64, 38304 and 38400 in items of 128: one power of two
print([launches(d) for d in ((32, 32, 32), (33, 32, 32), (38, 36, 28), (20, 40, 48))])

def batch(edges):
    b = cgx.Batch(0)
    for k, n in enumerate(edges):
        m = PeriodicBoxMesh(n, jitter=0.25, seed=k)
        b.add(cgx.Mesh(m, device=0), prm, *cases.tgv_state(m.x_cv[: m.ncv], prm), nsteps=5)
    n = b.launch_count()
    b.step(1)
    return b.launch_count() - n

print([batch((24, 24, 20)), batch((25, 23, 20))])  # about 35700 cells in items of 32, then again
"""


def test_each_kind_is_tuned_once(built):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", CODE % root], capture_output=True, text=True, check=True).stdout
    single, batch = (eval(line) for line in out.split("\n")[:2])
    tuning = 4 * 17  # a warm-up and three timed launches of 17 candidates
    assert single[0] == single[2] == single[1] + tuning
    assert single[1] == single[3]
    assert batch[0] >= batch[1] + tuning
