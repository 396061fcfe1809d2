"""FP64 analyses when the device has no room for the pair products' scratch (bsa_pair64.cu, bsa_list64.cu).

The products are an optional form: without room the point kernel, which needs the A table alone, takes
the call.  Same sums in another order: 1e-12 of the largest value."""
import numpy as np
import pytest

from bsalib_gb300 import api
from bsalib_gb300.problem import tall_building

pytestmark = pytest.mark.gpu


def _classic(s, rng, F):
    out = s.run()
    return [out[k] for k in ("m2mf_cls", "m2mr_cls", "m3mf_cls", "m3mr_cls")]


def _points(s, rng, F):
    return s.msh_bispectra(rng.uniform(-F, F, 120), rng.uniform(-F, F, 120))


def _zones(s, rng, F):
    x = rng.uniform(-F, F / 2, (4, 2))
    return s.msh_zones([api.Zone(a, b, 0.02, 0.0, 0.0, 0.02, 4, 5, 2, 2, 1.0, 0) for a, b in x])[:2]


# With 400 nodes and 24 modes the row digits take 33 x 576 x 8 x 832 x 2 = 253 MB (Classic) and more than
# 500 MB (points, zones), the point kernel's tables and partial sums at most 130 MB.
@pytest.mark.parametrize("call,trunc", [(_classic, True), (_classic, False), (_points, True), (_zones, True)])
def test_no_room_for_products(bsalib, call, trunc):
    import torch

    p = tall_building(nodes=400, modes=24, nfreqs=32, df=0.05, seed=3)

    def run():
        s = api.BsaSession(p, classic_truncation=trunc)
        try:
            return call(s, np.random.default_rng(5), 1.6), s.stats().kernels
        finally:
            s.close()
            assert bsalib.bsa_gpu_releaseDeviceCache() == 0

    want, n0 = run()
    torch.cuda.empty_cache()
    try:
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (224 << 20), dtype=torch.uint8, device="cuda")
    except torch.OutOfMemoryError:
        pytest.skip("another process took device memory meanwhile")
    try:
        got, n1 = run()
    finally:
        del hold
        torch.cuda.empty_cache()
    assert n1 != n0  # another set of kernels ran
    for a, b in zip(got, want):
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
