"""The two cells of a face see exactly opposite fluxes: on a mesh of pairs of
cells, each joined by one face that is both extended and compact, calcRhs of one
cell is minus the other's bit for bit in every component (FP64; the mixed form's
closures are FP32 differences of squares, opposite to their rounding)."""
import numpy as np
import pytest

from list_mesh import list_mesh, state
from nextgen_b200 import cases, cgx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tune", ["1,1,1,1", "4,2,1,2"])
def test_pairs(built, tune, monkeypatch):
    monkeypatch.setenv("CGX_TUNE", tune)
    n = 40000  # items of 128 cells
    rng = np.random.default_rng(1)
    pairs = rng.permutation(n).reshape(-1, 2)
    m = list_mesh(n, pairs, np.arange(len(pairs)), 2)
    prm = cases.hit_params()
    s = cgx.Solver(cgx.Mesh(m, device=0), prm)
    s.set_state_primitive(*state(n, 3, prm))
    s.initComplete()
    r = s.calcRhs(1)
    s.close()
    assert np.abs(r).min() > 0.0
    for q in range(5):
        assert np.array_equal(r[pairs[:, 0], q], -r[pairs[:, 1], q]), q
