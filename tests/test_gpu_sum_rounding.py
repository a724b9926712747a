"""The rounding of calcRhs's FP64 face sums: on a state whose cell values and
enthalpies are exact in FP64, with the closures switched off, the rhs differs
from an 80-bit sum of the same fluxes by the rounding of the fluxes and of the
sums alone.

The bound: a rounding is 0.42 u of its value in the mean square (u = 2^-53, the
value's fraction spread over a binade).  A momentum flux carries three roundings
at its own size; its addition, within a block of eight of about 80 entries, one at
4.5/80 of the cell's sum F^2 in the mean, and the ten blocks and the parts as
much again: 0.42 u sqrt((3 + 4.5 + 5.5) sum F^2) at most, whatever way a cell's
list is split.  Adding each of a flux's four terms to one running sum by itself
makes it 0.42 u sqrt(4 x 40 sum F^2)."""
import os

import numpy as np
import pytest

from nextgen_b200 import cgx
from nextgen_b200.meshgen import PeriodicBoxMesh

pytestmark = pytest.mark.gpu


def exact_state(m, rng):
    """Powers of two for rho, few-bit u and p: 1/rho, rhoE, p and K p / rho are exact."""
    n = m.ncv
    rho = rng.choice([0.5, 1.0, 1.0, 2.0], n)
    u = rng.integers(-256, 257, (n, 3)) / 1024.0
    p = 1.0 + rng.integers(-64, 65, n) / 1024.0
    return rho, u, p


def params():
    prm = cgx.Params()
    prm.gamma = 1.5
    prm.p_ref = prm.rho_ref = prm.T_ref = 1.0
    prm.mu_ref = 0.0
    prm.sgs_model = 0
    prm.coeff_p = prm.coeff_h = 0.0
    prm.diss_mode = 1  # none
    return prm


def wide_rhs(m, rho, u, p, K):
    """-sum of the extended faces' fluxes in 80 bits, and the root of sum F^2"""
    L = np.longdouble
    a, b = np.asarray(m.cvoef).reshape(-1, 2).T
    own = np.concatenate([np.arange(m.ncv), np.asarray(m.icv_owner_g)[: m.ncv_g2 - m.ncv]])
    n = np.asarray(m.n_ef).reshape(-1, 3).astype(L)
    c = 0.5 * np.asarray(m.c_ef).reshape(-1, 3).astype(L)
    j = own[b]
    r, v, w, h = rho.astype(L), 1 / rho.astype(L), u.astype(L), K * p.astype(L) / rho.astype(L)
    pl = p.astype(L)
    rf = 2 / (v[a] + v[j])
    uf, du = (w[a] + w[j]) / 2, w[j] - w[a]
    un, uc, duc = (uf * n).sum(1), (uf * c).sum(1), (du * c).sum(1)
    mc = uc * rf
    M = un * rf + uc * (r[j] - r[a]) + rf * duc
    pf, dp = (pl[a] + pl[j]) / 2, pl[j] - pl[a]
    F = np.empty((len(a), 5), L)
    F[:, 0] = M
    F[:, 1:4] = pf[:, None] * n + dp[:, None] * c + M[:, None] * uf + mc[:, None] * du
    F[:, 4] = M * (h[a] + h[j] + (w[a] * w[j]).sum(1)) / 2 + mc * (h[j] - h[a] + (uf * du).sum(1))
    rhs, sq = np.zeros((m.ncv, 5), L), np.zeros((m.ncv, 5), L)
    mine = b < m.ncv
    for q in range(5):
        np.add.at(rhs[:, q], a, -F[:, q])
        np.add.at(rhs[:, q], b[mine], F[mine, q])
        np.add.at(sq[:, q], a, F[:, q] ** 2)
        np.add.at(sq[:, q], b[mine], F[mine, q] ** 2)
    return rhs, np.sqrt(sq)


@pytest.mark.parametrize("tune", [None, "1,1,1,1", "4,2,1,2", "16,8,1,4"])
@pytest.mark.parametrize("n", [20, 34], ids=["items32", "items128"])
def test_sums_round_once_an_entry(built, n, tune, monkeypatch):
    if tune:
        monkeypatch.setenv("CGX_TUNE", tune)
    m = PeriodicBoxMesh(n, jitter=0.25, seed=5)
    prm = params()
    rho, u, p = exact_state(m, np.random.default_rng(n))
    s = cgx.Solver(cgx.Mesh(m, device=0), prm)
    s.set_state(rho, u, p / (prm.gamma - 1.0) + 0.5 * rho * (u * u).sum(1))
    s.initComplete()
    rhs = s.calcRhs(1)
    s.close()
    ref, root = wide_rhs(m, rho, u, p, prm.gamma / (prm.gamma - 1.0))
    err = np.sqrt(np.mean(((rhs - ref) / root).astype(np.float64)[:, 1:4] ** 2))
    assert err <= 0.42 * 2.0 ** -53 * np.sqrt(3 + 4.5 + 5.5), err
