"""The issued work that bench.py states for the E-form kernel, against the products the kernel cannot do
without: E(f_p, f_q), q >= p, for all (a, b, j) over K in three BF16 passes.  Beyond them it issues what its
tiles pad: rows to 128, K to 16, and per grid row the columns of its first two N tiles before p and of its last
two behind the grid, at most 3 NC of (nf + 1) / 2 on average."""
import pytest

import bench


@pytest.mark.parametrize("nf,nm,nnl,ntc,nc,pad", [(1025, 24, 400, 2, 10, 640 / 576), (1025, 16, 400, 2, 16, 1.0),
                                                  (1025, 8, 200, 1, 16, 128 / 64 * 208 / 200)])
def test_issued_flops(bsalib, nf, nm, nnl, ntc, nc, pad):
    needed = nf * (nf + 1) // 2 * nm ** 3 * 2 * ntc * nnl * 3
    ratio = bench.issued_flops_e(nf, nm, nnl, ntc) / needed
    assert pad <= ratio <= pad * (1 + 3 * nc / ((nf + 1) / 2))
