"""An analysis that runs out of device memory half way: it says so, nothing it queued outlives the tables it
reads, and the next session runs as if nothing had been."""
import numpy as np
import pytest

from bsalib_gb300 import api
from bsalib_gb300.problem import tall_building

pytestmark = pytest.mark.gpu


def _out_of_room(s):
    """Bispectra of 40 000 listed points, 4.4 GB each of force and response."""
    f = np.random.default_rng(1).uniform(-2, 2, (2, 40000))
    return s.msh_bispectra(f[0], f[1])


def test_failing_call_leaves_the_library_usable(bsalib):
    import torch

    p = tall_building(nodes=200, modes=24, nfreqs=16, df=0.1, seed=3)

    def small():
        s = api.BsaSession(p)
        try:
            return s.run()["m3mr_cls"]
        finally:
            s.close()

    want = small()
    assert bsalib.bsa_gpu_releaseDeviceCache() == 0
    try:
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (3 << 30), dtype=torch.uint8, device="cuda")
    except torch.OutOfMemoryError:
        pytest.skip("another process took device memory meanwhile")
    s = api.BsaSession(p)
    try:
        with pytest.raises(api.BsaError) as exc:
            _out_of_room(s)
        assert exc.value.code == -6          # BSA_ERR_NOMEM
    finally:
        s.close()
        del hold
        torch.cuda.empty_cache()
    assert np.array_equal(small(), want)
    assert bsalib.bsa_gpu_releaseDeviceCache() == 0
