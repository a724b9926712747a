"""The face kernels' rows where they are most delicate, against the oracle: every
lane count on items of several slices, with the scalars that read the entries'
mass fluxes by row; items split because their neighbours would not fit in shared
memory, some inside a slice of 32 cells; the largest compact union; a batch of
128-cell items.

Tolerances as in the tests of the plain cases: face sums to 1e-12 of their scale in
FP64 (about 100 terms in two orders), 2e-5 with FP32 fluxes."""
import numpy as np
import pytest

from list_mesh import list_mesh, state
from nextgen_b200 import cases, cgx
from nextgen_b200.meshgen import PeriodicBoxMesh
from oracle import Oracle

pytestmark = pytest.mark.gpu

TOL = {cgx.CGX_FP64: 1e-12, cgx.CGX_MIXED: 2e-5}
PRECS = pytest.mark.parametrize("prec", [cgx.CGX_FP64, cgx.CGX_MIXED], ids=["fp64", "mixed"])


def worst(a, ref, scale):
    return (np.abs(a - ref) / np.maximum(np.maximum(np.abs(ref), scale), 1e-300)).max()


class Case:
    """A mesh, its state and scalars, and the oracle's rhs of them.  `closed`: the
    extended faces' normals of a cell sum to zero; where they do not, as in a mesh
    of random normals, the mixed form (which sums p - p_ref) lacks p_ref times
    their sum."""

    def __init__(self, m, prm, st, closed=True):
        self.m, self.prm, self.st = m, prm, st
        self.sc = np.random.default_rng(5).random((m.ncv, 3))
        o = Oracle(m, prm)
        o.set_state_primitive(*st)
        o.set_scalars(self.sc)
        o.init_complete()
        self.rhs, self.rhs_sc, self.cfl = o.calc_rhs(1), o.rhs_sc(1), o.calc_cfl(1.0)[0]
        self.gm = cgx.Mesh(m, device=0)
        self.defect = np.zeros((m.ncv, 5))
        if not closed:
            for k in range(3):
                np.add.at(self.defect[:, 1 + k], m.cvoef[:, 0], prm.p_ref * m.n_ef[:, k])
                np.add.at(self.defect[:, 1 + k], m.cvoef[:, 1], -prm.p_ref * m.n_ef[:, k])

    def check(self, prec, tune, monkeypatch):
        monkeypatch.setenv("CGX_TUNE", tune)
        s = cgx.Solver(self.gm, self.prm, prec)
        s.set_state_primitive(*self.st)
        s.set_scalars(self.sc)
        s.initComplete()
        assert ",".join(str(v) for v in s.tuning().values()) == tune
        rhs = s.calcRhs(1) - (self.defect if prec == cgx.CGX_MIXED else 0.0)
        assert worst(rhs, *self.rhs) <= TOL[prec]
        assert worst(s.rhs_sc(1), *self.rhs_sc) <= TOL[prec]
        assert abs(s.calcCfl(1.0) - self.cfl) <= (1e-12 if prec == cgx.CGX_FP64 else 1e-6) * self.cfl
        s.close()


# ---- every lane count: items of 64 and of 128 cells, partly empty last slices ----

@pytest.fixture(scope="module", params=[(29, 31, 42), (25, 25, 61)], ids=["items64", "items128"])
def box(request, built):
    dims = request.param
    m = PeriodicBoxMesh(*dims, L=tuple(2.0 * np.pi * n / max(dims) for n in dims), jitter=0.25, seed=3)
    prm = cases.tgv_params()
    return Case(m, prm, cases.tgv_state(m.x_cv[: m.ncv], prm))


@PRECS
@pytest.mark.parametrize("tune", ["1,1,1,1", "2,2,2,2", "4,4,4,4", "8,8,8,8", "16,16,16,16", "32,1,2,1"])
def test_lane_counts(box, prec, tune, monkeypatch):
    box.check(prec, tune, monkeypatch)


# ---- items split for their unions ------------------------------------------------

def random_faces(n, degree, rng):
    """`degree[i]` faces from cell i to other cells, each pair once."""
    a = np.repeat(np.arange(n), degree)
    b = rng.integers(0, n, len(a))
    e = np.unique(np.sort(np.stack([a, b], 1)[a != b], 1), axis=0)
    return e[rng.permutation(len(e))]


@pytest.fixture(scope="module")
def split(built):
    n = 6005
    rng = np.random.default_rng(2)
    degree = np.full(n, 100)
    degree[rng.permutation(n)[:40]] = 1200  # some cells split their items further
    e = random_faces(n, degree, rng)
    m = list_mesh(n, e, np.arange(0, len(e), 6), 3)
    # as the centroids say nothing about the faces, an item is a random run of cells
    adj = [[] for _ in range(n)]
    for a, b in e:
        adj[a].append(b)
        adj[b].append(a)
    perm = rng.permutation(n)
    reach = [len(set(perm[k:k + 32]).union(*(adj[c] for c in perm[k:k + 32]))) for k in range(0, n - 32, 320)]
    assert min(reach) > 3000  # the largest extended union an item may have
    prm = cases.hit_params()
    return Case(m, prm, state(n, 4, prm), closed=False)


@PRECS
@pytest.mark.parametrize("tune", ["1,1,1,1", "2,2,2,2", "4,8,4,8", "16,4,8,4"])
def test_split_items(split, prec, tune, monkeypatch):
    split.check(prec, tune, monkeypatch)


# ---- the largest compact union ---------------------------------------------------

@pytest.fixture(scope="module")
def star(built):
    """1100 cells in a row; the first 32, one item, have every other cell as a
    compact neighbour: 1100 staged records, with which 16 warps' sums do not fit."""
    n = 1100
    leaf = np.arange(32, n)
    e = np.stack([leaf % 32, leaf], 1)
    # (and some extended faces more, for sums of more than one entry)
    more = [np.stack([leaf[:-k], leaf[k:]], 1) for k in (1, 7, 40, 90, 200)]
    m = list_mesh(n, np.concatenate([e] + more), np.arange(len(e)), 6)
    m.x_cv = np.zeros((n, 3))
    m.x_cv[:, 0] = np.arange(n)
    prm = cases.hit_params()
    prm.sgs_model = 0  # one neighbour's gradient has rank one: Vreman's B is the rounding of zero
    return Case(m, prm, state(n, 7, prm), closed=False)


@PRECS
@pytest.mark.parametrize("tune", ["2,8,2,2", "32,16,16,16"])
def test_largest_compact_union(star, prec, tune, monkeypatch):
    star.check(prec, tune, monkeypatch)


# ---- a batch of 128-cell items ---------------------------------------------------

@PRECS
@pytest.mark.parametrize("tune", ["1,1,1,1", "4,2,2,4"])
def test_batch_of_long_items(box, prec, tune, monkeypatch):
    if box.m.ncv < 37888:
        pytest.skip("items of 64 cells")
    monkeypatch.setenv("CGX_TUNE", tune)
    o = Oracle(box.m, box.prm)
    o.set_state_primitive(*box.st)
    o.init_complete()
    assert o.step(2) == 0
    b = cgx.Batch(0, prec, max_cases=2)
    cid = b.add(box.gm, box.prm, *box.st, nsteps=2)
    b.step(2)
    for a, ref in zip(b.get_state(cid), o.get_state()):
        assert np.abs(a - ref).max() <= (1e-12 if prec == cgx.CGX_FP64 else 1e-6) * np.abs(ref).max()
    b.close()
