"""Directions that are not quite on the unit sphere: the gradient is that of the P_l of their dot products.  Through
the harmonics it would be off by l (l + 1) / 2 of what |v|^2 lacks to 1, so only what rounding leaves takes that route.

Bars, of the sum of the terms' sizes: n eps kappa for the factorisation and l (l + 1) / 2 eps for the rounding of the
dot products and of |v|^2."""
import numpy as np
import pytest

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("lacks", [0.0, 2e-15, 8e-15, 5e-14, 1e-10])
@pytest.mark.parametrize("lmax", [20, 60])
def test_gradient_of_directions_off_the_unit_sphere(lmax, lacks):
    n = 60
    rng = np.random.default_rng(lmax)
    v = rng.standard_normal((n, 3))
    v *= np.sqrt(1.0 - lacks) / np.linalg.norm(v, axis=1)[:, None]
    cl = 1e-3 * W.fiducial_cl(lmax)
    d = 3.0 * rng.standard_normal(n)
    vl = v.astype(np.longdouble)
    x = np.clip(vl @ vl.T, -1, 1)
    p = [np.ones_like(x), x]
    for l in range(2, lmax + 1):
        p.append((2 - np.longdouble(1) / l) * x * p[-1] - (1 - np.longdouble(1) / l) * p[-2])
    w = (2 * np.arange(lmax + 1) + 1) / (4 * np.pi)
    cov = sum(cl[l] * w[l] * p[l] for l in range(2, lmax + 1)).astype(float) + 4.0 * np.eye(n)
    ev = np.linalg.eigvalsh(cov)
    inv = np.linalg.inv(cov)
    a = np.linalg.solve(cov, d)
    with cg.Context(lmax=lmax, fwhm_deg=0.0, beam=np.ones(lmax + 1), dirs=v, noise_sigma=2.0) as ctx:
        r = ctx.loglike(cl, d, grad=True)
    assert r["status"] == cg.CG_OK
    wt = (inv + inv.T) / 2 - np.outer(a, a)
    for l in range(2, lmax + 1):
        g = float(np.sum(wt * p[l])) * w[l]
        size = float(np.sum((np.abs(inv) + np.abs(np.outer(a, a))) * np.abs(p[l]))) * w[l]
        tol = n * EPS * ev[-1] / ev[0] + l * (l + 1) / 2 * EPS
        assert abs(r["grad"][l] - g) <= tol * size, (l, abs(r["grad"][l] - g) / size, tol)
