"""The FP64 A(f) kernel at the edges of its tiles (64 rows, 32 columns, modes padded to fours),
through the second moments of the force: m2mf = sum_f w_f L^T A(f), A(f) = s (c^|f|) s L restated in
numpy.  Coherences of 0 and 1 and the range where c^f underflows are among the inputs.  Tolerance:
sums of at most 130 x 9 terms in FP64, 1e-12 of the largest moment."""
import numpy as np
import pytest

from bsalib_gb300 import api
from bsalib_gb300.problem import random_structure

pytestmark = pytest.mark.gpu


def _reference(p, f):
    n, nm = p.nn, p.nm
    lin = p.wfc[0, 0, :][:, None] * p.phi
    c = np.zeros((n, n))
    iu = np.triu_indices(n)
    c[iu] = p.nod_corr[:, 0]
    c.T[iu] = p.nod_corr[:, 0]
    ls, u, sg = p.L[0, 0, p.wz_node - 1], p.u_node, p.sigma[0, p.wz_node - 1]
    out = []
    for x in np.abs(f):
        r = ls / u
        s = np.sqrt((2.0 / 3.0) * x * r * r * sg ** 2 / (1.0 + (x * r) ** 2) ** (4.0 / 3.0) / (4.0 * np.pi))
        out.append(lin.T @ (s[:, None] * (c ** x @ (s[:, None] * lin))))
    return np.array(out)  # [f, o, n]


@pytest.mark.parametrize("nodes,modes", [(2, 1), (31, 4), (32, 5), (33, 8), (63, 9), (64, 12), (65, 13), (66, 16), (40, 17),
                                         (40, 21), (40, 25), (40, 33), (40, 41), (40, 49), (130, 57), (70, 64),
                                         (79, 3), (80, 3), (128, 12), (129, 32), (200, 33), (192, 8), (513, 5), (600, 40)])
def test_atable_through_force_moments(bsalib, nodes, modes):
    p = random_structure(nodes + modes, nodes=(nodes, nodes), modes=(modes, modes), nfreq_grid=(17, 17))
    p.settings.ibisp = 0
    p.nod_corr[0, 0] = 1.0
    p.nod_corr[1, 0] = 0.0
    if p.nod_corr.shape[0] > 4:
        p.nod_corr[3, 0], p.nod_corr[4, 0] = 1e-300, 1e-120
    s = api.BsaSession(p)
    try:
        m2 = s.run()["m2mf_cls"]
    finally:
        s.close()
    h = p.settings.nfreqs - 1
    f = np.arange(-h, h + 1) * p.settings.df
    w = np.full(f.size, 2 * np.pi * p.settings.df)
    w[[0, -1]] /= 2
    ref = np.einsum("f,fon->on", w, _reference(p, f)).ravel()
    assert np.max(np.abs(m2 - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("where,value", [(0, 0.5), (3, 1.5), (0, 0.0)])
def test_coherences_outside_the_usual(bsalib, where, value):
    """A node's own coherence below 1, a coherence above 1: the general kernel forms the table."""
    p = random_structure(7, nodes=(90, 90), modes=(5, 5), nfreq_grid=(17, 17))
    p.settings.ibisp = 0
    p.nod_corr[where, 0] = value
    s = api.BsaSession(p)
    try:
        m2 = s.run()["m2mf_cls"]
    finally:
        s.close()
    h = p.settings.nfreqs - 1
    f = np.arange(-h, h + 1) * p.settings.df
    w = np.full(f.size, 2 * np.pi * p.settings.df)
    w[[0, -1]] /= 2
    ref = np.einsum("f,fon->on", w, _reference(p, f)).ravel()
    assert np.max(np.abs(m2 - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("nodes,loaded", [(9, (9, 2, 5)), (7, (7, 1, 4, 6)), (6, (2, 4, 6, 1, 3, 5)), (40, (40, 1))])
def test_loaded_nodes_in_any_order(bsalib, nodes, loaded):
    """Few of many nodes loaded, and out of order: the coherences are those of the loaded nodes."""
    import dataclasses
    p = random_structure(nodes, nodes=(nodes, nodes), modes=(3, 3), nfreq_grid=(9, 9))
    p.settings.ibisp = 0
    ix = np.array(loaded) - 1
    q = dataclasses.replace(p, n_load=np.array(loaded, dtype=np.int32), wfc=np.asfortranarray(p.wfc[:, :, ix]))
    s = api.BsaSession(q)
    try:
        m2 = s.run()["m2mf_cls"]
    finally:
        s.close()
    # the same with zero forces on the other nodes
    w = np.zeros_like(p.wfc)
    w[:, :, ix] = p.wfc[:, :, ix]
    s = api.BsaSession(dataclasses.replace(p, wfc=np.asfortranarray(w)))
    try:
        ref = s.run()["m2mf_cls"]
    finally:
        s.close()
    assert np.max(np.abs(m2 - ref)) <= 1e-12 * np.max(np.abs(ref))
