"""cgx_set_scalars with another number of scalars between steps: every step form
takes the new arrays up, whichever form ran before."""
import numpy as np
import pytest

from nextgen_b200 import cases, cgx
from nextgen_b200.meshgen import PeriodicBoxMesh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def box(built):
    m = PeriodicBoxMesh(13, jitter=0.25, seed=7)
    prm = cases.tgv_params()
    return m, prm, cases.tgv_state(m.x_cv[: m.ncv], prm), cgx.Mesh(m, device=0)


def solver(box):
    m, prm, st, gm = box
    s = cgx.Solver(gm, prm)
    s.set_state_primitive(*st)
    s.initComplete()
    return s


def step_out(s):
    out = [np.empty(s.ncv), np.empty((s.ncv, 3)), np.empty(s.ncv)]
    assert s.step_out_ptr(1, *(a.ctypes.data for a in out)) == 0


def test_step_out_takes_new_scalars(box):
    n = box[0].ncv
    sc = [np.random.default_rng(k).random((n, k)) for k in (1, 3)]
    a, b = solver(box), solver(box)
    step_out(a)
    assert b.step(1) == 0
    for c in sc:
        a.set_scalars(c)
        b.set_scalars(c)
        step_out(a)
        assert b.step(1) == 0
        assert np.array_equal(a.get_scalars(), b.get_scalars())
        assert not np.array_equal(a.get_scalars(), c)
    a.close()
    b.close()
