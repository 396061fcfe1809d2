"""The FP64 Classic analysis over distinct frequency pairs (bsa_pair64.cu) against the point kernel.

A row range that leaves nothing out but is set explicitly in two shards keeps the point kernel, so
the sum of two row shards is the point kernel's whole grid.  Both evaluate the same sums in FP64 in
another order: 1e-12 of the largest moment (about 1e4 roundings of 1e-16)."""
import numpy as np
import pytest

from bsalib_gb300 import api
from bsalib_gb300.problem import random_structure, tall_building

pytestmark = pytest.mark.gpu


def _run(prob, rows=None, trunc=True, sym=False):
    s = api.BsaSession(prob, classic_truncation=trunc)
    try:
        if rows:
            s.set_rows(*rows)
        if sym:
            s.set_symmetry(True)
        return s.run()
    finally:
        s.close()


def _close(a, b, tol=1e-12):
    for k in ("m2mf_cls", "m2mr_cls", "m2o2mr_cls", "m3mf_cls", "m3mr_cls"):
        assert np.max(np.abs(a[k] - b[k])) <= tol * np.max(np.abs(b[k])), k


# modes at and around the tiles of the moment kernel (rows per block, pair lanes) and of the products
@pytest.mark.parametrize("modes,nodes,nfreqs", [(1, 3, 2), (2, 5, 3), (3, 17, 9), (5, 16, 12), (7, 33, 10), (16, 9, 8),
                                                (17, 40, 6), (33, 12, 5), (64, 70, 3)])
@pytest.mark.parametrize("trunc,scalar", [(True, 0), (False, 0), (True, 1), (False, 1)])
def test_pairs_against_points(bsalib, modes, nodes, nfreqs, trunc, scalar):
    p = tall_building(nodes=nodes, modes=modes, nfreqs=nfreqs, df=2.0 / nfreqs, seed=modes)
    p.settings.scalar = scalar
    nf = p.classic_nf()
    whole = _run(p, trunc=trunc)
    a, b = _run(p, (0, 1), trunc), _run(p, (1, nf), trunc)
    _close(whole, {k: a[k] + b[k] for k in a})
    _close(_run(p, trunc=trunc, sym=True), whole)


def test_pairs_one_component(bsalib):
    p = random_structure(11, nodes=(37, 37), modes=(9, 9), nfreq_grid=(41, 41))
    a, b = _run(p, (0, 20)), _run(p, (20, 41))
    _close(_run(p), {k: a[k] + b[k] for k in a})


# tensor-core products: K around a 16-wide step, a 64-wide block and the 512-wide exact pass; rows that
# share a tile and rows that span several
@pytest.mark.parametrize("nodes,modes,nfreqs", [(12, 33, 9), (32, 9, 33), (33, 7, 40), (256, 5, 40), (257, 5, 40),
                                                (550, 3, 34), (20, 64, 4)])
@pytest.mark.parametrize("trunc", [True, False])
def test_tensor_pairs_against_points(bsalib, nodes, modes, nfreqs, trunc):
    p = tall_building(nodes=nodes, modes=modes, nfreqs=nfreqs, df=2.0 / nfreqs, seed=modes)
    nf = p.classic_nf()
    whole = _run(p, trunc=trunc)
    a, b = _run(p, (0, nf // 2), trunc), _run(p, (nf // 2, nf), trunc)
    _close(whole, {k: a[k] + b[k] for k in a})


def test_tensor_pairs_wide_range(bsalib):
    """Mode shapes over twelve decades along the height and modes scaled apart by 1e60: a row's small
    entries lie far below its scale, whole rows far apart from each other."""
    p = tall_building(nodes=64, modes=8, nfreqs=40, df=0.05, seed=5)
    p.wfc[0, :3, :] *= np.logspace(0, -12, p.nn)
    p.phi[:, 3] *= np.where(np.abs(p.phi[:, 3]) == 1.0, 1.0, 1e-60)
    nf = p.classic_nf()
    a, b = _run(p, (0, 20)), _run(p, (20, nf))
    _close(_run(p), {k: a[k] + b[k] for k in a})


def test_tensor_pairs_not_finite(bsalib):
    p = tall_building(nodes=64, modes=8, nfreqs=40, df=0.05, seed=5)
    p.wfc[0, 0, 7] = np.inf
    nf = p.classic_nf()
    whole, a, b = _run(p), _run(p, (0, 20)), _run(p, (20, nf))
    for k in ("m3mf_cls", "m3mr_cls"):
        assert np.array_equal(np.isfinite(whole[k]), np.isfinite(a[k] + b[k]))


# diagonal-only spectra: both product kernels, several row tiles and y lanes past a warp
@pytest.mark.parametrize("modes,nodes,nfreqs", [(1, 3, 2), (3, 17, 9), (5, 16, 40), (24, 33, 20), (33, 130, 70), (64, 20, 34)])
@pytest.mark.parametrize("trunc,scalar", [(True, 0), (False, 0), (True, 1)])
def test_diagonal_pairs_against_points(bsalib, modes, nodes, nfreqs, trunc, scalar):
    p = tall_building(nodes=nodes, modes=modes, nfreqs=nfreqs, df=2.0 / nfreqs, seed=modes)
    p.settings.scalar, p.settings.onlyd = scalar, 1
    nf = p.classic_nf()
    whole = _run(p, trunc=trunc)
    a, b = _run(p, (0, 1), trunc), _run(p, (1, nf), trunc)
    _close(whole, {k: a[k] + b[k] for k in a})
    _close(_run(p, trunc=trunc, sym=True), whole)


@pytest.mark.parametrize("modes,nodes,nfreqs", [(1, 3, 2), (5, 16, 6), (9, 40, 12), (17, 33, 4), (64, 12, 3)])
@pytest.mark.parametrize("trunc", [True, False])
def test_bispectra_against_listed_points(bsalib, modes, nodes, nfreqs, trunc):
    p = tall_building(nodes=nodes, modes=modes, nfreqs=nfreqs, df=2.0 / nfreqs, seed=modes)
    s = api.BsaSession(p, classic_truncation=trunc)
    try:
        f, bf, br = s.classic_bispectra()
        n = f.size
        i1, i2 = (v.ravel() for v in np.meshgrid(np.arange(n), np.arange(n), indexing="ij"))
        pieces = [s.classic_points(i1[k:k + 3], i2[k:k + 3]) for k in range(0, n * n, 3)]
    finally:
        s.close()
    for a, k in ((bf, 0), (br, 1)):
        b = np.concatenate([x[k] for x in pieces]).reshape(a.shape)
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
