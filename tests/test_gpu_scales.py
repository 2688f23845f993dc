"""Matrices whose rows differ in scale: pixels in two units, noise variances over many orders of magnitude, maps
with a huge value in a pixel that the noise takes out.  A Cholesky factorisation in FP64 does not depend on such
scales: with S = D^-1 C D^-1 of unit diagonal and kappa = cond(S), chi2 moves by at most about n eps kappa of
itself, ln det by n eps kappa and the gradient by n eps kappa of the sum of its terms' sizes.  The bars are 8 times
these; ln det also carries the rounding of the scales' logarithms, 4 eps sum |2 ln D_i|.  The reference works on S."""
import numpy as np
import pytest

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _sky(n, lmax, seed, norm):
    """directions, C_l with variances of a few muK^2, their covariance and the terms of its gradient"""
    rng = np.random.default_rng(seed)
    v = rng.standard_normal((n, 3))
    v *= norm / np.linalg.norm(v, axis=1)[:, None]
    cl = 1e-3 * W.fiducial_cl(lmax)
    x = np.clip(v @ v.T, -1, 1)
    p = [np.ones_like(x), x]
    for l in range(2, lmax + 1):
        p.append((2 - 1.0 / l) * x * p[-1] - (1 - 1.0 / l) * p[-2])
    beam = np.exp(-0.002 * np.arange(lmax + 1.0) ** 2)
    w = (2 * np.arange(lmax + 1) + 1) / (4 * np.pi) * beam ** 2
    return v, cl, beam, [p[l] * w[l] for l in range(lmax + 1)], rng


def _factors(c):
    """D, S^-1, ln det C and kappa of S = D^-1 C D^-1"""
    dd = np.sqrt(np.diag(c))
    s = c / dd[:, None] / dd[None, :]
    np.fill_diagonal(s, 1.0)
    ev = np.linalg.eigvalsh(s)
    inv = np.linalg.inv(s)
    return dd, (inv + inv.T) / 2, np.linalg.slogdet(s)[1] + 2 * np.log(dd).sum(), ev[-1] / ev[0]


def _bars(n, dd, kappa):
    tol = 8 * n * EPS * kappa
    return tol, tol + 4 * EPS * np.abs(2 * np.log(dd)).sum()


def _noise(kind, n, rng):
    """noise variances and the map's scale per pixel"""
    var = np.full(n, 4.0)
    if kind == "interleaved":           # two instruments, 1e9 apart in sigma
        var[1::2] *= 1e18
    elif kind == "graded":              # sigma over nine decades
        var *= 10.0 ** rng.uniform(0, 18, n)
    elif kind == "masked":              # pixels taken out by their noise
        var[rng.permutation(n)[:20]] = 1e24
    elif kind == "unseen":              # the same, holding HEALPix's value for a missing pixel
        var[rng.permutation(n)[:20]] = 1e62
    d = 2.0 * np.sqrt(var) * rng.standard_normal(n)
    d[var == 1e24] = 1e10
    d[var == 1e62] = -1.6375e30
    return var, d


@pytest.mark.parametrize("norm", [1.0, 1.0 + 1e-13], ids=["harmonics", "inverse"])
@pytest.mark.parametrize("kind", ["even", "interleaved", "graded", "masked", "unseen"])
@pytest.mark.parametrize("n", [40, 64, 130, 257])
def test_noise_variances_of_many_scales(n, kind, norm):
    lmax = 10
    v, cl, beam, terms, rng = _sky(n, lmax, n, norm)
    var, d = _noise(kind, n, rng)
    cov = sum(cl[l] * terms[l] for l in range(2, lmax + 1)) + np.diag(var)
    dd, inv, ld, kappa = _factors(cov)
    tol, tol_ld = _bars(n, dd, kappa)
    y = inv @ (d / dd)
    chi2 = y @ (d / dd)
    with cg.Context(lmax=lmax, fwhm_deg=1.0, dirs=v, beam=beam, noise_var=var) as ctx:
        r = ctx.loglike(cl, d, grad=True)
        q = ctx.loglike(cl, d)
    assert r["status"] == cg.CG_OK and q["status"] == cg.CG_OK
    for k in (r, q):
        assert abs(k["chi2"] - chi2) <= tol * chi2, (abs(k["chi2"] / chi2 - 1), tol)
        assert abs(k["logdet"] - ld) <= tol_ld, (abs(k["logdet"] - ld), tol_ld)
    a = y / dd
    ci = inv / dd[:, None] / dd[None, :]
    for l in range(2, lmax + 1):
        g = np.sum((ci - np.outer(a, a)) * terms[l])
        size = np.sum((np.abs(ci) + np.abs(np.outer(a, a))) * np.abs(terms[l]))
        assert abs(r["grad"][l] - g) <= tol * size, (l, abs(r["grad"][l] - g) / size, tol)


def _units(kind, n, rng):
    if kind == "interleaved 1e-6":      # muK and K
        u = np.ones(n)
        u[1::2] = 1e-6
        return u
    span = {"graded 1e8": 8, "graded 1e14": 14}[kind]
    return 10.0 ** (span * (rng.permutation(n) / max(n - 1.0, 1.0) - 0.5))


@pytest.mark.parametrize("kind", ["interleaved 1e-6", "graded 1e8", "graded 1e14"])
@pytest.mark.parametrize("n", [2, 64, 65, 130, 300])
def test_packed_likelihood_in_mixed_units(n, kind):
    """u C u with u per pixel: the same chi2 for the map u t, ln det moved by 2 sum ln u; with a foreground u f."""
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n + 5))
    c = a @ a.T / n + 0.5 * np.eye(n)
    c = (c + c.T) / 2
    u = _units(kind, n, rng)
    m = u[:, None] * c * u[None, :]
    m = (m + m.T) / 2
    t, f = u * rng.standard_normal(n), u * (1.0 + rng.standard_normal(n))
    dd, inv, ld, kappa = _factors(m)
    tol, tol_ld = _bars(n, dd, kappa)
    tt, tf, ff = [(x / dd) @ inv @ (y / dd) for x, y in ((t, t), (t, f), (f, f))]
    zero = np.zeros(n * (n + 1) // 2)
    lik = cg.Likelihood(W.full_to_packed(m), None, zero)
    _, chi2, _ = lik.calculate(t)
    assert abs(lik.logdet_raw - ld) <= tol_ld, (abs(lik.logdet_raw - ld), tol_ld)
    assert abs(chi2 - tt) <= tol * tt, (abs(chi2 / tt - 1), tol)
    lik.close()
    lik = cg.Likelihood(W.full_to_packed(m), None, zero, foreground=f)
    _, chi2, _ = lik.calculate(t)
    assert abs(chi2 - (tt - tf * tf / ff)) <= 3 * tol * tt
    lik.close()


def test_packed_likelihood_with_an_unseen_pixel():
    n = 150
    rng = np.random.default_rng(7)
    a = rng.standard_normal((n, n + 5))
    c = a @ a.T / n
    c = (c + c.T) / 2
    var = np.full(n, 0.5)
    out = rng.permutation(n)[:12]
    var[out] = 1e62
    t = rng.standard_normal(n)
    t[out] = -1.6375e30
    dd, inv, ld, kappa = _factors(c + np.diag(var))
    tol, tol_ld = _bars(n, dd, kappa)
    want = (t / dd) @ inv @ (t / dd)
    lik = cg.Likelihood(W.full_to_packed(c), None, W.full_to_packed(np.diag(var)))
    _, chi2, _ = lik.calculate(t)
    assert abs(chi2 - want) <= tol * want, (abs(chi2 / want - 1), tol)
    assert abs(lik.logdet_raw - ld) <= tol_ld
    lik.close()
