"""The tensor-core FP64 factorisation (k_digit.cu) at the sizes where its tiling changes: one to a few
64-column steps, the edges of 64-row blocks and of 128-row pairs, extra rows that fill, exceed or leave
free the last pair, batches beyond one CTA wave, both gradient routes and the packed drop-in, against
FP64 numpy.

Tolerances: a backward-stable factorisation of C (condition number kappa) moves chi2 = d^T C^-1 d by at
most about n eps kappa chi2, ln det by n eps kappa, and C^-1 by n eps kappa |C^-1|; the bars below
are 8 times these, with the gradient's scale sum_ij |W_ij| |dC_ij/dC_l|."""
import numpy as np
import pytest

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def _legendre(x, lmax):
    p = [np.ones_like(x), x]
    for l in range(2, lmax + 1):
        p.append((2 - 1.0 / l) * x * p[-1] - (1 - 1.0 / l) * p[-2])
    return p


def _setup(n, lmax, seed, batch, norm=1.0):
    rng = np.random.default_rng(seed)
    v = rng.standard_normal((n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    cls = W.lognormal_batch(W.fiducial_cl(lmax), batch, seed + 1)
    d = 20.0 * rng.standard_normal((batch, n))
    return v * norm, cls, d


def _reference(v, cls, d, beam, var):
    n, lmax = len(v), cls.shape[1] - 1
    x = np.clip(v @ v.T, -1, 1)
    p = _legendre(x, lmax)
    w = (2 * np.arange(lmax + 1) + 1) / (4 * np.pi) * beam ** 2
    out = []
    for c, m in zip(cls, d):
        cov = sum(c[l] * w[l] * p[l] for l in range(2, lmax + 1)) + var * np.eye(n)
        ev = np.linalg.eigvalsh(cov)
        inv = np.linalg.inv(cov)
        inv = (inv + inv.T) / 2
        a = np.linalg.solve(cov, m)
        g, s = np.zeros(lmax + 1), np.zeros(lmax + 1)
        for l in range(2, lmax + 1):
            g[l] = np.sum((inv - np.outer(a, a)) * p[l]) * w[l]
            s[l] = np.sum(np.abs(inv) + np.abs(np.outer(a, a))) * w[l]
        out.append((m @ a, np.linalg.slogdet(cov)[1], g, s, 8 * n * EPS * ev[-1] / ev[0]))
    return out


def _check(r, ref, grad=True):
    assert np.all(r["status"] == 0), r["status"]
    for b, (chi2, ld, g, s, tol) in enumerate(ref):
        assert abs(r["chi2"][b] - chi2) <= tol * chi2, (b, r["chi2"][b], chi2)
        assert abs(r["logdet"][b] - ld) <= tol, (b, r["logdet"][b], ld)
        assert r["m2lnl"][b] == r["chi2"][b] + r["logdet"][b]
        if grad:
            assert np.all(np.abs(r["grad"][b] - g) <= tol * s + 1e-300), (b, np.abs(r["grad"][b] - g) / s.max(), tol)


# pixels: below, at and above one block, one pair, several pairs.  lmax 2, 7, 10, 12, 14: 5, 60, 117,
# 165, 221 harmonics, so that the map's row falls in the first, second, third or fourth block of E
@pytest.mark.parametrize("n,lmax,batch", [(1, 2, 1), (5, 3, 2), (63, 7, 1), (64, 7, 3), (65, 10, 1), (127, 10, 2),
                                          (128, 12, 1), (129, 14, 2), (192, 12, 1), (193, 7, 40), (321, 14, 3)])
@pytest.mark.parametrize("norm", [1.0, 1.0 + 1e-13], ids=["harmonics", "inverse"])
def test_value_and_gradient(n, lmax, batch, norm):
    """norm 1: the gradient through the harmonics; directions off the unit sphere by 1e-13 (no effect on
    the numbers at these bars) take the route through C^-1."""
    v, cls, d = _setup(n, lmax, 17 * n + lmax, batch, norm)
    beam = np.exp(-0.002 * np.arange(lmax + 1.0) ** 2)
    ref = _reference(v, cls, d, beam, 4.0)
    with cg.Context(lmax=lmax, fwhm_deg=1.0, dirs=v, beam=beam, noise_sigma=2.0, max_batch=batch) as ctx:
        val = ctx.loglike(cls, d)                 # value first: its workspace then grows for the gradient
        full = ctx.loglike(cls, d, grad=True)
        again = ctx.loglike(cls, d)               # and a value call on the grown workspace
        one = ctx.loglike(cls, d[0], grad=True)   # one map for every element
    _check(val, ref, grad=False)
    _check(full, ref)
    for k in ("m2lnl", "chi2", "logdet"):
        assert np.array_equal(val[k], again[k])
        assert one[k][0] == full[k][0]
    assert np.array_equal(one["grad"][0], full["grad"][0])


@pytest.mark.parametrize("scale", [1e-120, 1e-9, 1e7, 1e110])
def test_scale_of_the_map_and_of_the_covariance(scale):
    """Powers of two in the rows: covariance scale^2, map scale, chi2 unchanged to rounding."""
    v, cls, d = _setup(150, 9, 5, 1)
    beam = np.exp(-0.002 * np.arange(10.0) ** 2)
    chi2, _, _, _, tol = _reference(v, cls, d, beam, 4.0)[0]
    with cg.Context(lmax=9, fwhm_deg=1.0, dirs=v, beam=beam, noise_sigma=2.0 * scale) as ctx:
        r = ctx.loglike(cls[0] * scale ** 2, d[0] * scale, grad=True)
        q = ctx.loglike(cls[0] * scale ** 2, d[0] * scale * 1e-30)
    assert r["status"] == 0 and abs(r["chi2"] - chi2) <= 2 * tol * chi2
    assert abs(q["chi2"] - chi2 * 1e-60) <= 2 * tol * chi2 * 1e-60


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_nonfinite_map_stays_visible(bad):
    v, cls, d = _setup(130, 7, 6, 2)
    d[1, 77] = bad
    with cg.Context(lmax=7, fwhm_deg=1.0, dirs=v, noise_sigma=2.0, max_batch=2) as ctx:
        r = ctx.loglike(cls, d, grad=True)
    assert np.isfinite(r["m2lnl"][0]) and not np.isfinite(r["m2lnl"][1])
    assert np.all(np.isfinite(r["grad"][0])) and not np.any(np.isfinite(r["grad"][1][2:]))


@pytest.mark.parametrize("n", [1, 2, 64, 65, 128, 129, 300])
def test_packed_likelihood(n):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n + 5))
    c = a @ a.T / n
    c = (c + c.T) / 2
    t = rng.standard_normal(n)
    full = c + 0.5 * np.eye(n)
    ev = np.linalg.eigvalsh(full)
    tol = 8 * n * EPS * ev[-1] / ev[0]
    lik = cg.Likelihood(W.full_to_packed(c), None, W.full_to_packed(0.5 * np.eye(n)))
    for m in (t, -3 * t[::-1]):
        _, chi2, ld = lik.calculate(m)
        want = m @ np.linalg.solve(full, m)
        assert abs(chi2 - want) <= tol * want
        assert abs(lik.logdet_raw - np.linalg.slogdet(full)[1]) <= tol
    lik.close()


@pytest.mark.parametrize("n", [1, 63, 64, 65, 130, 257])
def test_packed_likelihood_foreground(n):
    """The marginalised foreground (source/likelihood.cpp:171-177) needs t^T C^-1 f and f^T C^-1 f: three
    quadratic forms, each within the bar of one."""
    rng = np.random.default_rng(1000 + n)
    a = rng.standard_normal((n, n + 5))
    c = a @ a.T / n
    full = (c + c.T) / 2 + 0.5 * np.eye(n)
    t, f = rng.standard_normal(n), 1.0 + rng.standard_normal(n)
    ev = np.linalg.eigvalsh(full)
    tol = 8 * n * EPS * ev[-1] / ev[0]
    lik = cg.Likelihood(W.full_to_packed(full), None, np.zeros(n * (n + 1) // 2), foreground=f)
    _, chi2, ld = lik.calculate(t)
    at, af = np.linalg.solve(full, t), np.linalg.solve(full, f)
    tt, tf, ff = t @ at, t @ af, f @ af
    assert abs(chi2 - (tt - tf * tf / ff)) <= 3 * tol * tt
    assert abs((ld - cg.DET_OFFSET) - (np.linalg.slogdet(full)[1] + np.log(ff / n))) <= 2 * tol + 8 * EPS * abs(ld)
    lik.close()


@pytest.mark.parametrize("npix,ngood", [(1, 1), (40, 32), (40, 33), (100, 64), (100, 65), (600, 544)])
def test_polarisation_products(npix, ngood):
    """N^-1 + N^-1 C N^-1 at 2, 64, 66, 128, 130 and 1088 kept values: one pair of blocks, the edges of the next, and
    more K blocks than are held at once (17 of 64).  A product of n terms is off by at most n eps |A| |B| per
    entry; chi2 and ln det then carry the factorisation's bar."""
    rng = np.random.default_rng(npix + ngood)
    size = 2 * npix
    a = rng.standard_normal((size, size)) / np.sqrt(size)
    b = rng.standard_normal((size, size)) / np.sqrt(size)
    c = a @ a.T + 0.5 * np.eye(size)
    ninv = b @ b.T + 2.0 * np.eye(size)
    good = np.sort(rng.permutation(npix)[:ngood]).astype(np.int32)
    k = np.concatenate([good, npix + good])
    n = len(k)
    v, sub = rng.standard_normal(n), 0.3 * rng.standard_normal(n)
    nk = ninv[np.ix_(k, k)]
    m = nk + nk @ c[np.ix_(k, k)] @ nk
    m = (m + m.T) / 2
    ev = np.linalg.eigvalsh(m)
    tol = 16 * n * EPS * ev[-1] / ev[0]
    lik = cg.LikelihoodPolarization(W.full_to_packed(c), npix, good, np.ascontiguousarray(ninv))
    _, chi2, _ = lik.calculate(v, sub)
    w = v - nk @ sub
    # chi2 = w^T cInv w, cInv the inverse of m (the factored matrix)
    want = w @ np.linalg.solve(m, w)
    scale = (np.abs(v) + np.abs(nk) @ np.abs(sub)) @ np.abs(np.linalg.solve(m, w))
    assert abs(lik.logdet_raw - np.linalg.slogdet(m)[1]) <= tol
    assert abs(chi2 - want) <= tol * max(scale, want)
    lik.close()


@pytest.mark.parametrize("batch", [1, 2, 3, 4, 5, 9])
def test_packed_covariances_of_a_batch_are_those_of_each(batch):
    """Elements that share the recurrence (two or four at a time, and what is left over) keep the bits of a call
    of their own."""
    v, cls, _ = _setup(70, 11, 3, batch)
    with cg.Context(lmax=11, fwhm_deg=9.0, dirs=v, max_batch=batch) as ctx:
        full = ctx.build_cmatrix(cls)
        for b in range(batch):
            assert np.array_equal(full[b], ctx.build_cmatrix(cls[b]))


@pytest.mark.parametrize("which", ["c", "fid", "noise"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_nonfinite_packed_matrices_are_refused(which, bad):
    n = 130
    eye = W.full_to_packed(np.eye(n))
    m = dict(c=eye.copy(), fid=0.0 * eye, noise=eye.copy())
    m[which][len(eye) // 3] = bad
    with pytest.raises(cg.CGError) as e:
        cg.Likelihood(m["c"], m["fid"], m["noise"])
    assert e.value.code == cg.CG_ERR_NONFINITE


@pytest.mark.parametrize("pixel,refused", [(3, True), (4, False)])
def test_nonfinite_polarisation_entries_count_where_they_are_kept(pixel, refused):
    npix, good = 40, np.array([1, 3, 7, 39], dtype=np.int32)
    c, ninv = np.eye(2 * npix), 2.0 * np.eye(2 * npix)
    for k, m in enumerate((c, ninv)):
        bad = [c.copy(), ninv.copy()]
        bad[k][pixel, pixel] = np.nan
        args = (W.full_to_packed(bad[0]), npix, good, bad[1])
        if refused:
            with pytest.raises(cg.CGError) as e:
                cg.LikelihoodPolarization(*args)
            assert e.value.code == cg.CG_ERR_NONFINITE
        else:
            cg.LikelihoodPolarization(*args).close()


@pytest.mark.parametrize("batch", [1, 2, 4])
@pytest.mark.parametrize("case", ["plain", "exact ties", "zeros", "tiny beam", "range of exponents", "negative"])
def test_packed_covariance_rounds_every_operation(case, batch):
    """The integer products of the packed covariance keep the bits of the FP64 operations in order, and what is
    outside their range (zero terms and polynomials, exponents far from 1) takes those operations themselves."""
    rng = np.random.default_rng(5)
    lmax = 21
    v = rng.standard_normal((40, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    v = np.concatenate([v, np.eye(3), -np.eye(3), [[0.5, 0.5, 0.5], [0.75, 0.25, 0.0]]])  # x = 0, 1, -1, short x
    cls = np.abs(rng.standard_normal((batch, lmax + 1))) + 0.1
    beam = np.exp(-0.01 * np.arange(lmax + 1.0) ** 2)
    if case == "exact ties":
        cls = 4 * np.pi * 2.0 ** rng.integers(-3, 4, cls.shape)
        beam = 1.0 + 2.0 ** -rng.integers(20, 53, lmax + 1)
    elif case == "zeros":
        cls[:, 2::3] = 0.0
        cls[0, 4] = 0.0
        beam[9] = 0.0
    elif case == "tiny beam":
        beam = np.exp(-0.8 * np.arange(lmax + 1.0) ** 2)
    elif case == "range of exponents":
        cls *= 10.0 ** rng.integers(-120, 121, cls.shape)
    elif case == "negative":
        cls *= rng.choice([-1.0, 1.0], cls.shape)
    x = (v[:, None, 0] * v[None, :, 0] + v[:, None, 1] * v[None, :, 1]) + v[:, None, 2] * v[None, :, 2]
    p = [np.ones_like(x), np.clip(x, -1, 1)]
    for l in range(2, lmax + 1):
        p.append(((2 - 1.0 / l) * p[1]) * p[-1] - (1 - 1.0 / l) * p[-2])
    with cg.Context(lmax=lmax, fwhm_deg=0.0, beam=beam, dirs=v, max_batch=batch) as ctx:
        got = ctx.build_cmatrix(cls).reshape(batch, -1)
    for b in range(batch):
        want = np.zeros_like(x)
        for l in range(2, lmax + 1):
            want += ((((cls[b, l] * (2 * l + 1)) / (4 * np.pi)) * p[l]) * beam[l]) * beam[l]
        assert np.array_equal(got[b], W.full_to_packed(want))


@pytest.mark.parametrize("n,lmax,batch", [(450, 11, 100), (700, 14, 40), (1300, 20, 12), (200, 20, 150)])
def test_elements_of_a_batch_keep_the_bits_of_a_call_of_their_own(n, lmax, batch):
    """A CTA's runs of jobs over several rounds and a remainder, the chain beside the rest of an update or before it,
    and the split of a column pair between them order the work differently, never an element's operations."""
    v, cls, d = _setup(n, lmax, 17, batch)
    with cg.Context(lmax=lmax, fwhm_deg=9.0, dirs=v, noise_sigma=1.0, max_batch=batch) as ctx:
        full = ctx.loglike(cls, d[0], grad=True)
        assert np.all(full["status"] == cg.CG_OK)
        for b in (0, batch // 2, batch - 1):
            one = ctx.loglike(cls[b:b + 1], d[0], grad=True)
            for name in ("m2lnl", "chi2", "logdet", "grad"):
                assert np.array_equal(full[name][b], one[name][0]), (name, b)
