"""The orders in which the FP64 factorisation runs its work at larger sizes: with the identity as extra rows, the chain
beside the rest of the update (from 2000 pixels, or a batch of 1000), where the second stream writes the inverse into
tiles that the first one has left; and products whose CTAs take several jobs with several sets of images (more than
1536 kept values).  Bars as in test_gpu_digit.py: 8 n eps kappa, 16 n eps kappa for the products."""
import numpy as np
import pytest

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _spd(n, rng, diag):
    a = rng.standard_normal((n, n)) / np.sqrt(n)
    return a @ a.T + diag * np.eye(n)


def test_packed_likelihood_with_the_chain_beside_the_update():
    n = 2100
    rng = np.random.default_rng(n)
    c = _spd(n, rng, 0.5)
    t, f = rng.standard_normal(n), 1.0 + rng.standard_normal(n)
    ev = np.linalg.eigvalsh(c)
    tol = 8 * n * EPS * ev[-1] / ev[0]
    at, af = np.linalg.solve(c, np.stack([t, f], axis=1)).T
    tt, tf, ff = t @ at, t @ af, f @ af
    lik = cg.Likelihood(W.full_to_packed(c), None, np.zeros(n * (n + 1) // 2), foreground=f)
    got = [lik.calculate(t)[1] for _ in range(3)]
    assert abs(lik.logdet_raw - np.linalg.slogdet(c)[1]) <= tol
    assert abs(got[0] - (tt - tf * tf / ff)) <= 3 * tol * tt
    assert got[1] == got[0] and got[2] == got[0]
    lik.close()


def test_inverse_gradients_with_the_chain_beside_the_update():
    """Bit for bit those of single calls, whose steps run one after the other."""
    n, lmax, batch = 1000, 9, 8
    rng = np.random.default_rng(n)
    v = rng.standard_normal((n, 3))
    v *= (1.0 + 1e-13) / np.linalg.norm(v, axis=1)[:, None]
    cls, d = W.lognormal_batch(W.fiducial_cl(lmax), batch, 1), 20.0 * rng.standard_normal((batch, n))
    with cg.Context(lmax=lmax, fwhm_deg=9.0, dirs=v, noise_sigma=2.0, max_batch=batch) as ctx:
        for _ in range(3):
            full = ctx.loglike(cls, d, grad=True)
            assert np.all(full["status"] == cg.CG_OK)
            for b in range(batch):
                one = ctx.loglike(cls[b], d[b], grad=True)
                for name in ("m2lnl", "chi2", "logdet", "grad"):
                    assert np.array_equal(full[name][b], one[name]), (name, b)


@pytest.mark.parametrize("npix,ngood", [(800, 800), (1000, 850)])
def test_polarisation_products_of_several_jobs_per_cta(npix, ngood):
    rng = np.random.default_rng(ngood)
    size = 2 * npix
    c, ninv = _spd(size, rng, 0.5), _spd(size, rng, 2.0)
    good = np.sort(rng.permutation(npix)[:ngood]).astype(np.int32)
    k = np.concatenate([good, npix + good])
    n = len(k)
    v, sub = rng.standard_normal(n), 0.3 * rng.standard_normal(n)
    nk = ninv[np.ix_(k, k)]
    m = nk + nk @ c[np.ix_(k, k)] @ nk
    m = (m + m.T) / 2
    ev = np.linalg.eigvalsh(m)
    tol = 16 * n * EPS * ev[-1] / ev[0]
    w = v - nk @ sub
    s = np.linalg.solve(m, w)
    lik = cg.LikelihoodPolarization(W.full_to_packed(c), npix, good, ninv)
    _, chi2, _ = lik.calculate(v, sub)
    assert abs(lik.logdet_raw - np.linalg.slogdet(m)[1]) <= tol
    assert abs(chi2 - w @ s) <= tol * max((np.abs(v) + np.abs(nk) @ np.abs(sub)) @ np.abs(s), w @ s)
    lik.close()
