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


# factors of the quadratic and linear coefficients, and node 7's quadratic one for the mode that moves it:
# products Q A over the largest number, Q and A near its root, denormal Q, results among the denormals.  Grid
# points whose sum is on the grid: the point kernel multiplies a sum that reads zero by Q A
@pytest.mark.parametrize("quad,lin,at7", [(1.0, 1e120, 1e200), (1e200, 1e100, 1e7), (1e155, 1e70, 1e84), (1e-313, 1e145, 1e2),
                                          (1e-200, 1e-40, 1.0), (1e-160, 1e-74, 1e9)])
def test_ends_of_the_range(bsalib, quad, lin, at7):
    p = _groups(60, 8, 10.0)
    p.phi[7, :] = np.where(np.arange(8) == 3, 0.5, 0.0)
    p.wfc[0, :3] *= lin
    p.wfc[0, 3:] *= quad
    p.wfc[0, 3:, 7] *= at7
    rng = np.random.default_rng(4)
    f1, f2 = rng.uniform(-2, 2, 400), rng.uniform(-2, 2, 400)
    s = api.BsaSession(p)
    try:
        f, bf, _ = s.classic_bispectra()
        n = f.size
        i1, i2 = (v.ravel() for v in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
        on = np.abs(i1 + i2 - (n - 1)) <= (n - 1) // 2
        i1, i2 = i1[on], i2[on]
        want = np.concatenate([s.classic_points(i1[k:k + 15], i2[k:k + 15])[0] for k in range(0, i1.size, 15)])
        lst, _ = s.msh_bispectra(f1, f2)
        pieces = np.concatenate([s.msh_bispectra(f1[k:k + 2], f2[k:k + 2])[0] for k in range(0, 400, 2)])
    finally:
        s.close()
    for a, b in ((bf.reshape(n * n, -1)[on], want.reshape(on.sum(), -1)), (lst, pieces)):
        ok = np.isfinite(b)
        assert np.array_equal(a[~ok], b[~ok], equal_nan=True)
        # a denormal's rounding is 2^-1075 at every term
        assert np.all(np.abs(a[ok] - b[ok]) <= 2 * (120 + 4) * (U * np.abs(b[ok]) + 2.0 ** -1074))


@pytest.mark.parametrize("at7", [1e306, 1e308, np.inf, 1e-320])
def test_force_spectra_ends_of_the_range(bsalib, at7):
    """Against the same table formed by the general kernel, which a node's own coherence one rounding below 1
    selects (that moves an element by a rounding at most)."""
    got = []
    for own in (1.0, 1.0 - 2.0 ** -53):
        p = random_structure(90, nodes=(90, 90), modes=(6, 6), nfreq_grid=(9, 9))
        q = _groups(90, 6, 20.0)
        p.phi[:], p.nod_corr[:] = q.phi, q.nod_corr
        p.phi[7, :] = np.where(np.arange(6) == 1, 0.5, 0.0)
        p.wfc[0, 0, 7] *= at7 / 1e3 if np.isfinite(at7) else at7
        p.nod_corr[0, 0] = own
        p.settings.ibisp = 0
        s = api.BsaSession(p)
        try:
            got.append(s.run()["m2mf_cls"])
        finally:
            s.close()
    a, b = got
    ok = np.isfinite(b)
    assert np.array_equal(a[~ok], b[~ok], equal_nan=True)
    assert np.all(np.abs(a[ok] - b[ok]) <= 4 * (90 + 20) * U * np.abs(b[ok]))


# K at the edges of a 16-wide step, of a 64-wide block and of the 128-wide exact pass
@pytest.mark.parametrize("nodes", [24, 31, 32, 33, 63, 64, 65, 128, 129])
@pytest.mark.parametrize("modes", [11, 12])
def test_elements_around_a_pass(bsalib, nodes, modes):
    test_bispectra_elements(bsalib, nodes, modes, 10.0)
    test_listed_elements(bsalib, nodes, modes, 10.0)


def test_elements_over_a_wide_range(bsalib):
    """Forces over twelve decades along the height, and a mode that is 1e-60 of the others but at one node."""
    p = _groups(64, 8, 0.0, nfreqs=40, df=0.05)
    p.wfc[0, :3, :] *= np.logspace(0, -12, p.nn)
    p.phi[:, 3] *= np.where(p.phi[:, 3] == 1.0, 1.0, 1e-60)
    s = api.BsaSession(p)
    try:
        f, bf, _ = s.classic_bispectra()
        n = f.size
        i1, i2 = (v.ravel() for v in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
        i1, i2 = i1[::7], i2[::7]
        want = np.concatenate([s.classic_points(i1[k:k + 15], i2[k:k + 15])[0] for k in range(0, i1.size, 15)])
    finally:
        s.close()
    _within(bf.reshape(n * n, -1)[::7], want.reshape(i1.size, -1), 128)


@pytest.mark.parametrize("gap", [0.0, 40.0, None])
@pytest.mark.parametrize("trunc", [True, False])
def test_moment_elements(bsalib, gap, trunc):
    """Third moments of the force: sums of positive products over the grid (but for its four corners), within
    the products' bound and one rounding a grid point, twice for the corners' sign."""
    p = _groups(60, 8, gap)
    nf = p.classic_nf()

    def run(rows=None):
        s = api.BsaSession(p, classic_truncation=trunc)
        try:
            if rows:
                s.set_rows(*rows)
            return s.run()["m3mf_cls"]
        finally:
            s.close()

    a, b = run(), run((0, nf // 2)) + run((nf // 2, nf))
    assert np.all(np.abs(a - b) <= 4 * (120 + nf * nf) * U * np.abs(b))


def test_factors_below_every_high_word(bsalib):
    """Quadratic coefficients whose high word is zero (below 2^-1042) at one node, whose products with large
    linear forces are the largest of their rows, and for one mode the only ones."""
    p = _groups(60, 8, 10.0)
    i, j = np.triu_indices(p.nn)
    p.nod_corr[i != j] = 0.0
    p.phi[:, 1] = np.arange(p.nn) == 7
    p.wfc[0, :3] *= 1e-10
    p.wfc[0, 3:] *= 1e-220
    p.wfc[0, :3, 7] *= 1e157
    p.wfc[0, 3:, 7] = 3e-320
    rng = np.random.default_rng(4)
    f1, f2 = rng.uniform(-2, 2, (2, 400))
    s = api.BsaSession(p)
    try:
        lst, _ = s.msh_bispectra(f1, f2)
        pieces = np.concatenate([s.msh_bispectra(f1[k:k + 2], f2[k:k + 2])[0] for k in range(0, 400, 2)])
    finally:
        s.close()
    ok = np.isfinite(pieces)
    assert np.array_equal(lst[~ok], pieces[~ok], equal_nan=True)
    assert np.all(np.abs(lst[ok] - pieces[ok]) <= 2 * (120 + 4) * U * np.abs(pieces[ok]))
