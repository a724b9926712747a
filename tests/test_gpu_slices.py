"""The row layout of the face kernels at its edges, against the oracle: cell
counts that leave the last slice of 32 cells (and the last work item) partly
empty, on both sides of each change of the item length (32, 64 and 128 cells,
which follows from the cell count), and the smallest boxes.

calcRhs and the properties are compared per cell to 1e-12 of the face-sum scale
(FP64 sums of about 100 terms: 100 x 1.1e-16, and as much in the oracle), the
mixed form to its FP32 flux arithmetic, and a step's state to 1e-12."""
import numpy as np
import pytest

from nextgen_b200 import cases, cgx
from nextgen_b200.meshgen import PeriodicBoxMesh
from oracle import Oracle

pytestmark = pytest.mark.gpu

# cells: 512 (whole slices), 1287 = 40 x 32 + 7, then 18941 and 19008, 37758 and
# 38125 around the changes to 64 and 128 cells an item (18944 and 37888 cells)
DIMS = [(8, 8, 8), (11, 13, 9), (13, 31, 47), (11, 18, 96), (29, 31, 42), (25, 25, 61)]


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "%dx%dx%d" % d)
def test_rows_match_oracle(built, dims):
    m = PeriodicBoxMesh(*dims, L=tuple(2.0 * np.pi * n / max(dims) for n in dims), jitter=0.25, seed=3)
    prm = cases.tgv_params()
    rho, u, p = cases.tgv_state(m.x_cv[: m.ncv], prm)
    o = Oracle(m, prm)
    o.set_state_primitive(rho, u, p)
    o.init_complete()
    ref, scale = o.calc_rhs(1)
    co = o.calc_cfl(1.0)[0]
    gm = cgx.Mesh(m, device=0)
    for prec, tol in ((cgx.CGX_FP64, 1e-12), (cgx.CGX_MIXED, 2e-5)):
        s = cgx.Solver(gm, prm, prec)
        s.set_state_primitive(rho, u, p)
        s.initComplete()
        r = s.calcRhs(1)
        assert (np.abs(r - ref) / np.maximum(np.abs(ref), scale)).max() <= tol
        assert abs(s.calcCfl(1.0) - co) <= (1e-12 if prec == cgx.CGX_FP64 else 1e-6) * co
        if prec == cgx.CGX_FP64:
            assert s.step(1) == 0
            o.step(1)
            for a, b in zip(s.get_state(), o.get_state()):
                assert np.abs(a - b).max() <= 1e-12 * np.abs(b).max()
        s.close()
