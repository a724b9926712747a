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


def test_scalars_that_do_not_fit(built):
    """Out of device memory the call fails, and the solver goes on without scalars."""
    torch = pytest.importorskip("torch")
    m = PeriodicBoxMesh(40, jitter=0.25, seed=7)  # 64000 cells: the arrays of 8 scalars take 59 MB
    prm = cases.tgv_params()
    gm = cgx.Mesh(m, device=0)
    a, b = (solver((m, prm, cases.tgv_state(m.x_cv[: m.ncv], prm), gm)) for _ in range(2))
    a.set_scalars(np.ones((m.ncv, 1)))
    assert a.step(1) == 0 and b.step(1) == 0
    held, size = [], 1 << 33
    while size >= 1 << 23:
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda:0"))
        except torch.OutOfMemoryError:
            size >>= 1
    try:
        with pytest.raises(cgx.CgxError) as e:
            a.set_scalars(np.ones((m.ncv, 8)))
    finally:
        held.clear()
        torch.cuda.empty_cache()
    assert e.value.code == -2
    assert a.step(2) == 0 and b.step(2) == 0
    assert all(np.array_equal(x, y) for x, y in zip(a.get_state(), b.get_state()))
    sc = np.random.default_rng(0).random((m.ncv, 8))
    a.set_scalars(sc)
    assert a.step(1) == 0 and np.isfinite(a.get_scalars()).all()
    a.close()
    b.close()
