"""Every element of the FP64 results keeps FP64's own precision, also those far below the largest.

Two groups of nodes a gap apart, modes that move one group only, every factor positive: an element that
couples the groups is smaller than the others by the coherence over the gap, and nothing cancels, so FP64
gives each element to a few roundings of itself.  Term by term K FMAs are within K 2^-53 of a sum of
positive products; both sides together within 2 (K + 4) 2^-53 of the element (the row product, the three
terms' sum and the last rounding besides)."""
import numpy as np
import pytest

from bsalib_gb300 import api
from bsalib_gb300.problem import packed_coherence, random_structure, tall_building

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _groups(nodes, modes, gap, nfreqs=20, df=0.1, comps=(1, 3)):
    """gap in metres between two halves of the nodes; None: no coherence between them."""
    p = tall_building(nodes=nodes, modes=modes, nfreqs=nfreqs, df=df, seed=nodes)
    p.settings.tc = comps
    h, rng = nodes // 2, np.random.default_rng(modes)
    first = np.arange(nodes) < h
    z = 0.5 * np.arange(nodes) + np.where(first, 0.0, gap or 0.0)
    phi = rng.uniform(0.3, 1.0, (nodes, modes)) * np.where(np.arange(modes) < modes // 2, first[:, None], ~first[:, None])
    p.phi[:] = phi / phi.max(0)
    i, j = np.triu_indices(nodes)
    for c in range(3):
        p.nod_corr[:, c] = packed_coherence(z, np.full(nodes, 40.0), 10.0)
        if gap is None:
            p.nod_corr[first[i] != first[j], c] = 0.0
    return p


def _within(got, want, K):
    assert np.all(np.abs(got - want) <= 2 * (K + 4) * U * np.abs(want))


@pytest.mark.parametrize("nodes,modes", [(60, 8), (30, 12), (70, 17)])
@pytest.mark.parametrize("gap", [0.0, 10.0, 40.0, 150.0, None])
def test_bispectra_elements(bsalib, nodes, modes, gap):
    p = _groups(nodes, modes, gap)
    s = api.BsaSession(p)
    try:
        f, bf, _ = s.classic_bispectra()
        n = f.size
        i1, i2 = (v.ravel() for v in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
        want = np.concatenate([s.classic_points(i1[k:k + 15], i2[k:k + 15])[0] for k in range(0, n * n, 15)])
    finally:
        s.close()
    _within(bf.reshape(want.shape), want, 2 * nodes)


@pytest.mark.parametrize("nodes,modes", [(60, 12), (60, 17), (20, 40)])
@pytest.mark.parametrize("gap", [0.0, 10.0, 40.0, 150.0, None])
def test_listed_elements(bsalib, nodes, modes, gap):
    p = _groups(nodes, modes, gap)
    rng = np.random.default_rng(3)
    f1, f2 = rng.uniform(-2, 2, 300), rng.uniform(-2, 2, 300)
    s = api.BsaSession(p)
    try:
        bf, _ = s.msh_bispectra(f1, f2)
        want = np.concatenate([s.msh_bispectra(f1[k:k + 2], f2[k:k + 2])[0] for k in range(0, 300, 2)])
    finally:
        s.close()
    _within(bf, want, 2 * nodes)


def _force_psd(p, f):
    """L^T A(f), A = s (c^|f|) s L, in extended precision (Davenport-Uliege spectra, one component)."""
    X = np.longdouble
    n = p.nn
    lin = (p.wfc[0, 0, :][:, None] * p.phi).astype(X)
    c = np.zeros((n, n), X)
    iu = np.triu_indices(n)
    c[iu] = p.nod_corr[:, 0]
    c.T[iu] = p.nod_corr[:, 0]
    r, sg = (p.L[0, 0, p.wz_node - 1] / p.u_node).astype(X), p.sigma[0, p.wz_node - 1].astype(X)
    s = np.sqrt(X(2) / 3 * f * r * r * sg ** 2 / (1 + (f * r) ** 2) ** (X(4) / 3) / (4 * X(np.pi)))
    return lin.T @ (s[:, None] * (c ** X(f) @ (s[:, None] * lin)))


@pytest.mark.parametrize("nodes,modes", [(80, 8), (129, 12), (200, 33), (100, 64), (600, 5)])
@pytest.mark.parametrize("gap", [0.0, 20.0, 60.0, 150.0])
def test_force_spectra_elements(bsalib, nodes, modes, gap):
    """The A table, one frequency at a time.  Tolerance: sums over the nodes in A and in L^T A, the exponent's
    two roundings of x = |f log c|, and 60 roundings for the spectrum and the weights."""
    p = random_structure(nodes, nodes=(nodes, nodes), modes=(modes, modes), nfreq_grid=(9, 9))
    q = _groups(nodes, modes, gap)
    p.phi[:], p.nod_corr[:] = q.phi, q.nod_corr
    p.settings.ibisp, p.settings.df, h = 0, 0.4, p.settings.nfreqs - 1
    for k in range(1, h):
        s = api.BsaSession(p)
        try:
            s.set_rows(h + k, h + k + 1)
            got = s.run()["m2mf_cls"].reshape(modes, modes)
        finally:
            s.close()
        f = k * p.settings.df
        want = (_force_psd(p, f) * 2 * np.pi * p.settings.df).astype(float)
        x = -f * np.log(p.nod_corr[:, 0].min())
        assert np.all(np.abs(got - want) <= (2 * nodes + 2 * x + 60) * U * want)
