"""The FP64 pair products in several parts: chunks of first rows (4 GB of products each) on the Classic grid,
batches of a point list, and a list whose later batch finds no room.

Same sums in another order as the point kernel's: 1e-12 of the largest moment."""
import numpy as np
import pytest

from bsalib_gb300 import api
from bsalib_gb300.problem import tall_building

pytestmark = pytest.mark.gpu


def _close(a, b):
    for x, y in zip(a, b):
        assert np.max(np.abs(x - y)) <= 1e-12 * np.max(np.abs(y))


def _classic(p, rows=None, trunc=True):
    s = api.BsaSession(p, classic_truncation=trunc)
    try:
        if rows:
            s.set_rows(*rows)
        out = s.run()
    finally:
        s.close()
    return [out[k] for k in ("m3mf_cls", "m3mr_cls")]


# 64 modes: 2.1 MB a product, so 72 and 90 first rows are two and three chunks on the truncated grid; the
# diagonal form's 64 values a product fill a chunk at 4100 rows
@pytest.mark.parametrize("onlyd,nfreqs,trunc", [(0, 72, True), (0, 90, True), (0, 50, False), (1, 4200, True), (1, 2500, False)])
def test_chunks_of_first_rows(bsalib, onlyd, nfreqs, trunc):
    p = tall_building(nodes=2 if onlyd else 16, modes=64, nfreqs=nfreqs, df=2.0 / nfreqs, seed=4)
    p.settings.onlyd = onlyd
    nf = p.classic_nf()
    a, b = _classic(p, (0, nf // 2), trunc), _classic(p, (nf // 2, nf), trunc)
    _close(_classic(p, trunc=trunc), [x + y for x, y in zip(a, b)])


def _pieces(s, f1, f2, w):
    out = [s.msh_moments(f1[k:k + 16], f2[k:k + 16], w[k:k + 16]) for k in range(0, f1.size, 16)]
    return [sum(o[q] for o in out) for q in (0, 1)]


def test_batches_of_points(bsalib):
    """1020 points of 64 modes and 32 operand rows to a batch: two whole batches and one of a single point."""
    p = tall_building(nodes=16, modes=64, nfreqs=9, seed=4)
    f1, f2, w = np.random.default_rng(2).uniform(-2, 2, (3, 2041))
    s = api.BsaSession(p)
    try:
        _close(s.msh_moments(f1, f2, w)[:2], _pieces(s, f1, f2, w))
    finally:
        s.close()


def test_no_room_for_a_later_batch(bsalib):
    """The first batch is one frequency pair over and over, the second needs 6 GB for its products."""
    import torch

    p = tall_building(nodes=16, modes=64, nfreqs=9, seed=4)
    f1, f2, w = np.random.default_rng(2).uniform(-2, 2, (3, 2041))
    f1[:1020], f2[:1020] = 0.5, 0.25

    def run(want):
        s = api.BsaSession(p)
        try:
            out = _pieces(s, f1, f2, w) if want else s.msh_moments(f1, f2, w)[:2]
            return out, s.stats().kernels
        finally:
            s.close()
            assert bsalib.bsa_gpu_releaseDeviceCache() == 0

    want, _ = run(True)
    whole, n0 = run(False)
    torch.cuda.empty_cache()
    try:
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (3 << 30), dtype=torch.uint8, device="cuda")
    except torch.OutOfMemoryError:
        pytest.skip("another process took device memory meanwhile")
    try:
        got, n1 = run(False)
    finally:
        del hold
        torch.cuda.empty_cache()
    assert n1 < n0  # the second and third batches stayed with the point kernel
    _close(whole, want)
    _close(got, want)
