"""The 128 x 128 diagonal blocks of the mixed path's Cholesky (k_tc.cu): plain pivots go through the fast root, a
pivot that is not positive sends its panel through the general one.  Sizes of one 64-column half, of both halves
and of several blocks; an element that is not positive definite is reported and leaves its neighbours' bits alone."""
import numpy as np
import pytest

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [50, 100, 128, 129, 200, 300])
def test_an_element_that_is_not_positive_definite_is_reported_alone(n):
    rng = np.random.default_rng(n)
    lmax = 8
    v = rng.standard_normal((n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    fid = W.fiducial_cl(lmax)
    cls = W.lognormal_batch(fid, 3, n)
    cls[1] = -cls[1]
    d = 10.0 * rng.standard_normal(n)
    with cg.Context(lmax=lmax, fwhm_deg=9.0, dirs=v, noise_sigma=1.0, max_batch=3, precision="mixed", cl_ref=fid,
                    recenter="fixed") as ctx:
        r = ctx.loglike(cls, d)
        alone = [ctx.loglike(cls[b:b + 1], d) for b in (0, 2)]
    assert list(r["status"]) == [cg.CG_OK, cg.CG_ERR_NOT_PD, cg.CG_OK]
    for b, a in zip((0, 2), alone):
        for name in ("m2lnl", "chi2", "logdet"):
            assert r[name][b] == a[name][0]
    # the whitened covariances of 10 % perturbations: condition number below 2, FP32 sums over n terms
    with cg.Context(lmax=lmax, fwhm_deg=9.0, dirs=v, noise_sigma=1.0, max_batch=3) as ctx:
        want = ctx.loglike(cls[::2], d)
    tol = 8 * n * np.finfo(np.float32).eps
    for name in ("chi2", "logdet"):
        assert np.all(np.abs(r[name][::2] - want[name]) <= tol * (np.abs(want[name]) + n))
