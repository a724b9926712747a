"""One device mesh under several solvers: what a solver adds to it (the FP32
copies of the first mixed one, the neighbour list of the first with scalars) is
added once, whichever host threads ask for it, and a batch gives back for a mesh
what it took for it."""
import threading

import numpy as np
import pytest

from nextgen_b200 import cases, cgx
from nextgen_b200.meshgen import PeriodicBoxMesh

pytestmark = pytest.mark.gpu


def solver(gm, prm, st, prec=cgx.CGX_FP64):
    s = cgx.Solver(gm, prm, prec)
    s.set_state_primitive(*st)
    s.initComplete()
    return s


@pytest.fixture(scope="module")
def box(built):
    m = PeriodicBoxMesh(12, jitter=0.25, seed=7)
    prm = cases.tgv_params()
    return m, prm, cases.tgv_state(m.x_cv[: m.ncv], prm)


def test_batch_gives_back_what_it_took(box):
    m, prm, st = box
    gm = cgx.Mesh(m, device=0)
    b = cgx.Batch(0, max_cases=4)
    ids = [b.add(gm, prm, *st, nsteps=2) for _ in range(2)]
    before = gm.stats().device_bytes
    lone = [solver(gm, prm, st), solver(gm, prm, st, cgx.CGX_MIXED)]
    lone[0].set_scalars(np.ones((m.ncv, 1)))
    assert gm.stats().device_bytes > before
    b.step(2)
    for i in ids:
        b.remove(i)
    assert b.bytes()[0] == 0
    for s in lone:
        s.close()
    b.close()


def test_threads_extend_the_mesh_once(box):
    m, prm, st = box
    gm = cgx.Mesh(m, device=0)
    a, c = solver(gm, prm, st), solver(gm, prm, st, cgx.CGX_MIXED)
    a.set_scalars(np.ones((m.ncv, 1)))
    want = gm.stats().device_bytes
    assert a.step(2) == 0 and c.step(2) == 0
    ref = [a.get_scalars(), c.get_state()[2]]
    bad = []
    for _ in range(5):
        gm = cgx.Mesh(m, device=0)
        gate = threading.Barrier(6)

        def work(k, gm=gm):
            gate.wait()
            s = solver(gm, prm, st, cgx.CGX_MIXED if k % 2 else cgx.CGX_FP64)
            if k % 2 == 0:
                s.set_scalars(np.ones((m.ncv, 1)))
            if s.step(2) != 0 or not np.array_equal(s.get_state()[2] if k % 2 else s.get_scalars(), ref[k % 2]):
                bad.append(k)
            s.close()
        ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
        for t in ts:
            t.start()
        for t in ts:
            t.join()
        assert gm.stats().device_bytes == want
    assert not bad
