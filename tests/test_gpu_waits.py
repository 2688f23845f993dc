"""The FP64 factorisation's bounded waits: with those of the diagonal blocks and panels giving up at once and the
updates seeing their flag, the kernels end, report it, and leave the context as it was."""
import numpy as np
import pytest

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

pytestmark = pytest.mark.gpu


def test_waits_that_give_up_end_the_launch_and_are_reported():
    n, lmax = 400, 12
    rng = np.random.default_rng(3)
    v = rng.standard_normal((n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    cls, d = W.lognormal_batch(W.fiducial_cl(lmax), 2, 3), 20.0 * rng.standard_normal(n)
    with cg.Context(lmax=lmax, fwhm_deg=9.0, dirs=v, noise_sigma=2.0, max_batch=2) as ctx:
        want = ctx.loglike(cls, d, grad=True)
        for _ in range(3):
            assert ctx.selftest_wait_timeout() == cg.CG_ERR_TIMEOUT
            r = ctx.loglike(cls, d, grad=True)
            assert np.all(r["status"] == cg.CG_OK)
            for name in ("m2lnl", "chi2", "logdet", "grad"):
                assert np.array_equal(r[name], want[name]), name
