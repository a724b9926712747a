"""Meshes given by their face lists alone (no geometry behind them): random
unit-cube cells whose faces join the listed pairs of cells."""
from types import SimpleNamespace

import numpy as np


def list_mesh(ncv, extended, compact, seed):
    """`extended`: pairs of cells; `compact`: indices of those that are compact
    faces too.  Normals, areas and gradient coefficients are random."""
    rng = np.random.default_rng(seed)
    ef = np.asarray(extended, np.int32).reshape(-1, 2)
    fa = ef[np.asarray(compact)]
    fa = np.where(rng.random(len(fa))[:, None] < 0.5, fa, fa[:, ::-1]).astype(np.int32)  # either way round
    m = SimpleNamespace(ncv=ncv, ncv_g2=ncv, nfa=len(fa), nef=len(ef), cvofa=fa, cvoef=ef)
    m.n_ef, m.c_ef = rng.normal(size=(len(ef), 3)), 0.2 * rng.normal(size=(len(ef), 3))
    m.n_fa, m.area_over_delta_fa = rng.normal(size=(len(fa), 3)), rng.uniform(0.5, 2.0, len(fa))
    a = np.concatenate([fa[:, 0], fa[:, 1], np.arange(ncv)])
    b = np.concatenate([fa[:, 1], fa[:, 0], np.full(ncv, -1)])  # the cell itself stands first
    order = np.lexsort((b, a))
    m.cvocv_i = np.concatenate([[0], np.cumsum(np.bincount(a, minlength=ncv))]).astype(np.int32)
    m.cvocv_v = np.where(b < 0, a, b)[order].astype(np.int32)
    m.cvocv_grad_coeff = 0.1 * rng.normal(size=(len(a), 3))
    m.vol_cv, m.dcmag_hat_cv = rng.uniform(0.5, 2.0, ncv), rng.uniform(0.1, 0.5, ncv)
    m.sa_to_vol_ratio, m.icv_owner_g = rng.uniform(3.0, 9.0, ncv), np.zeros(1, np.int32)
    m.x_cv = rng.random((ncv, 3))
    return m


def state(ncv, seed, prm):
    rng = np.random.default_rng(seed)
    return (prm.rho_ref * rng.uniform(0.8, 1.25, ncv), 0.3 * rng.normal(size=(ncv, 3)),
            prm.p_ref * rng.uniform(0.8, 1.25, ncv))
