"""The bounded waits of the FP64 tensor-core kernels, run out without a fault (bsa_gpu_setWaitTestFP64): block 0
omits one ready signal, its waits end after 2 s and every other block's with the error flag; the host reports
BSA_ERR_TIMEOUT on each way the flag comes back (behind the moments, with the bispectra, after a table alone),
and the next session computes the same as before on the same context."""
import time

import numpy as np
import pytest

from bsalib_gb300 import api
from bsalib_gb300.problem import tall_building

pytestmark = pytest.mark.gpu


def _moments(s):
    return s.run()["m3mr_cls"]


def _second_order(s):
    return s.run()["m2mr_cls"]


def _bispectra(s):
    return s.classic_bispectra()[1]


def _listed(s):
    f = np.random.default_rng(1).uniform(-2, 2, (2, 200))
    return s.msh_moments(f[0], f[1], np.ones(200))[1]


@pytest.mark.parametrize("kernel,tile,call", [(0, 0, _moments), (0, 1, _second_order), (0, 0, _bispectra), (0, 1, _listed),
                                              (1, 0, _moments), (1, 1, _bispectra), (1, 2, _listed)])
def test_fp64_wait_budget_runs_out(bsalib, kernel, tile, call):
    p = tall_building(nodes=200, modes=10, nfreqs=24, df=0.1, seed=3)
    if call is _second_order:
        p.settings.ibisp = 0

    def session():
        return api.BsaSession(p)

    s = session()
    try:
        want = call(s)
    finally:
        s.close()
    s = session()
    try:
        assert bsalib.bsa_gpu_setWaitTestFP64(kernel, tile) == 0
        t0 = time.perf_counter()
        with pytest.raises(api.BsaError) as exc:
            call(s)
        assert "ran out of its budget" in str(exc.value)
        assert ("A-table" if kernel == 0 else "pair product") in str(exc.value)
        assert exc.value.code == -5          # BSA_ERR_TIMEOUT
        assert time.perf_counter() - t0 < 30.0
    finally:
        s.close()
    s = session()
    try:
        assert np.array_equal(call(s), want)
    finally:
        s.close()
