"""The pinned chunks behind pageable copies are shared by a process's solvers:
solvers on several host threads at once, more of them than the pairs that are
kept, each get their own arrays back bit for bit, over several calls and after
another solver's chunks came back."""
import threading

import numpy as np
import pytest

from nextgen_b200 import cases, cgx
from nextgen_b200.meshgen import DeviceOperatorMesh, PeriodicBoxMesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [1, 4])
def test_threads_share_the_chunks(built, threads):
    m = DeviceOperatorMesh(PeriodicBoxMesh(58, jitter=0.25, compact_only=True))  # u is 4.7 MB: staged
    gm = cgx.Mesh(m, device=0)
    prm = cases.tgv_params()
    wrong = []

    def work(k):
        s = cgx.Solver(gm, prm)
        rng = np.random.default_rng(k)
        for _ in range(3):
            rho, u, e = rng.random(m.ncv) + 1.0, rng.random((m.ncv, 3)), rng.random(m.ncv) + 200.0
            s.set_state(rho, u, e)
            for a, b in zip(s.get_state(), (rho, u, e)):
                if not np.array_equal(a, b):
                    wrong.append(k)
        s.close()
    ts = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong
