"""FP64 point sets over pair products (bsa_list64.cu) and the zones' FRF tables against the point kernel.

Few points stay on the point kernel, so a zone list evaluated zone by zone, or a point list in short
pieces, is the reference for the whole list.  Same sums in another order: 1e-12 of the largest value."""
import numpy as np
import pytest

from bsalib_gb300 import api
from bsalib_gb300.problem import tall_building

pytestmark = pytest.mark.gpu


def _zones(p, rng, n, kind):
    F = 1.25 * float(p.natf.max())
    out = []
    for _ in range(n):
        x, y, h = rng.uniform(-F, F / 2), rng.uniform(-F, F / 2), rng.uniform(0.05, 0.3) * F
        ni, nj, fi, fj = (int(v) for v in rng.integers([2, 2, 1, 1], [5, 5, 5, 5]))
        d = (h / (ni - 1), 0.0, 0.0, h / (nj - 1))
        if kind == "swapped":
            d = (0.0, d[0], -d[3], 0.0)
        elif kind == "rotated":
            c, s = np.cos(0.4), np.sin(0.4)
            d = (c * d[0], s * d[0], -s * d[3], c * d[3])
        out.append(api.Zone(x, y, *d, ni, nj, fi, fj, 1.0, 0))
    return out


# blocks of 8 to 32 columns a frequency and two blocks above 32 modes; K past a pass of 512
@pytest.mark.parametrize("nodes,modes,nz", [(90, 7, 60), (40, 9, 60), (60, 16, 40), (30, 17, 30), (30, 24, 30), (260, 12, 20),
                                            (20, 33, 20), (16, 64, 12)])
@pytest.mark.parametrize("kind", ["axes", "swapped", "rotated"])
def test_zone_list_against_single_zones(bsalib, nodes, modes, nz, kind):
    p = tall_building(nodes=nodes, modes=modes, nfreqs=9, seed=modes)
    zones = _zones(p, np.random.default_rng(modes), nz, kind)
    s = api.BsaSession(p)
    try:
        mf, mr, cnt = s.msh_zones(zones)
        each = [s.msh_zones([z]) for z in zones]
    finally:
        s.close()
    assert np.array_equal(cnt, sum(e[2] for e in each))
    for a, b in ((mf, sum(e[0] for e in each)), (mr, sum(e[1] for e in each))):
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))


@pytest.mark.parametrize("nodes,modes,n", [(100, 16, 300), (60, 24, 100), (40, 40, 40)])
def test_point_list_against_pieces(bsalib, nodes, modes, n):
    p = tall_building(nodes=nodes, modes=modes, nfreqs=9, seed=modes)
    rng = np.random.default_rng(n)
    f1, f2 = rng.uniform(-3, 3, n), rng.uniform(-3, 3, n)
    f2[:4] = f1[:4]            # f1 = f2
    f2[4:8] = -f1[4:8]         # f1 + f2 = 0
    f1[8:10] = 0.0
    s = api.BsaSession(p)
    try:
        bf, br = s.msh_bispectra(f1, f2)
        parts = [s.msh_bispectra(f1[i:i + 2], f2[i:i + 2]) for i in range(0, n, 2)]
    finally:
        s.close()
    for a, k in ((bf, 0), (br, 1)):
        b = np.concatenate([x[k] for x in parts])
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
