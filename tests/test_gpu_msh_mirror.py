"""Split-precision zones that repeat or mirror an earlier zone's lattice read its term tensors
(bsa_msh_mixed.cu).  The reference is each zone on its own, where nothing is shared: the per-zone
diagonal moments are then the same numbers (FP32 arithmetic on the same bits, 1e-6 for the order of
the sums over cells)."""
import numpy as np
import pytest

from bsalib_gb300 import api
from bsalib_gb300.problem import tall_building

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("modes", [4, 13, 24, 40])
def test_mirrored_and_repeated_zones(bsalib, modes):
    p = tall_building(nodes=24, modes=modes, nfreqs=9, seed=modes)
    rng = np.random.default_rng(modes)
    base = []
    for _ in range(6):
        x, y = rng.uniform(-2, 1.5, 2)
        ni, nj, fi, fj = (int(v) for v in rng.integers([2, 2, 1, 1], [6, 6, 4, 4]))
        base.append((x, y, rng.uniform(0.02, 0.2), rng.uniform(0.02, 0.2), ni, nj, fi, fj))
    zones = [api.Zone(x, y, dx, 0, 0, dy, ni, nj, fi, fj, 1.0, 0) for x, y, dx, dy, ni, nj, fi, fj in base]
    # mirror images through the origin (other refinements), the same lattice again, f1 mirrored only, and
    # a lattice that is its own mirror image
    zones += [api.Zone(-(x + (ni - 1) * dx), -(y + (nj - 1) * dy), dx, 0, 0, dy, ni, nj, fj, fi, 1.0, 0)
              for x, y, dx, dy, ni, nj, fi, fj in base]
    zones += [api.Zone(x, y, dx, 0, 0, dy, ni, nj, 1, 2, 2.0, 0) for x, y, dx, dy, ni, nj, fi, fj in base[:2]]
    zones += [api.Zone(-(x + (ni - 1) * dx), y, dx, 0, 0, dy, ni, nj, fi, fj, 1.0, 0)
              for x, y, dx, dy, ni, nj, fi, fj in base[:2]]
    zones += [api.Zone(-0.2, -0.3, 0.1, 0, 0, 0.15, 5, 5, 2, 2, 1.0, 0)]
    s = api.BsaSession(p, precision=api.PREC_BF16X3)
    try:
        mf, mr, zd = s.msh_zones_diag(zones)
        each = [s.msh_zones_diag([z]) for z in zones]
    finally:
        s.close()
    for a, b in ((mf, sum(e[0] for e in each)), (mr, sum(e[1] for e in each))):
        assert np.max(np.abs(a - b)) <= 1e-6 * np.max(np.abs(b))
    ref = np.concatenate([e[2] for e in each])
    assert np.max(np.abs(zd - ref)) <= 1e-6 * np.max(np.abs(ref))
