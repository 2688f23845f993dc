"""The Q/U likelihood's M = N^-1 + N^-1 C N^-1 where the scales of C and N^-1 differ from value to value: units that
C and N^-1 carry in opposite directions, and one-scale signals under noise of many scales.

FP64 products are off by at most 2 n eps (|N^-1| + |N^-1| |C| |N^-1|) per entry.  With D = diag(M)^(1/2), S = D^-1 M
D^-1, kappa = cond(S) and rho the largest such entry over D_i D_j, chi2 moves by at most about 2 n^2 eps rho kappa of
itself and ln det by as much times n; entries' errors being independent, n eps rho kappa is what is seen, and the
bars are 8 times that."""
import numpy as np
import pytest

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


@pytest.mark.parametrize("kind", ["one", "units 1e4", "units 1e8", "units 1e12", "noise 1e8", "noise 1e16", "no signal"])
@pytest.mark.parametrize("ngood", [1, 32, 33, 65, 200])
def test_graded_signal_and_noise(ngood, kind):
    rng = np.random.default_rng(ngood)
    npix, n = ngood, 2 * ngood
    a, b = rng.standard_normal((2, n, n)) / np.sqrt(n)
    c0, n0 = a @ a.T + 0.5 * np.eye(n), b @ b.T + 2.0 * np.eye(n)
    u = np.ones(n)                      # units of the signal; N^-1 has their inverse
    s = np.ones(n)                      # 1 / sigma on top of that
    name, _, span = kind.partition(" 1e")
    grade = 10.0 ** (float(span or 0) * (rng.permutation(n) / (n - 1.0) - 0.5))
    if name == "units":
        u = grade
    elif name == "noise":
        s = np.sqrt(grade)
        n0 = np.eye(n) + 0.2 * (n0 - np.diag(np.diag(n0)))
    elif kind == "no signal":           # pixels without signal: zero rows of C
        c0[::3] = 0.0
        c0[:, ::3] = 0.0
        u[1::3] = 1e-6
    n0 = s[:, None] * n0 * s[None, :]
    c = u[:, None] * c0 * u[None, :]
    ninv = n0 / u[:, None] / u[None, :]
    c, ninv = (c + c.T) / 2, (ninv + ninv.T) / 2
    # in the scale of unit u = 1: M0 = n0 + n0 c0 n0, w0 = u w
    m = n0 + n0 @ c0 @ n0
    m = (m + m.T) / 2
    dd = np.sqrt(np.diag(m))
    sm = m / dd[:, None] / dd[None, :]
    ev = np.linalg.eigvalsh(sm)
    rho = ((np.abs(n0) + np.abs(n0) @ np.abs(c0) @ np.abs(n0)) / dd[:, None] / dd[None, :]).max()
    tol = 8 * n * EPS * rho * ev[-1] / ev[0]
    v0, t0 = s * rng.standard_normal(n), 0.3 * rng.standard_normal(n) / s
    w0 = v0 - n0 @ t0
    x = w0 / dd
    want = x @ np.linalg.solve(sm, x)
    size = ((np.abs(v0) + np.abs(n0) @ np.abs(t0)) / dd) @ np.abs(np.linalg.solve(sm, x))
    logs = 2 * np.log(dd / u)
    lik = cg.LikelihoodPolarization(W.full_to_packed(c), npix, np.arange(npix, dtype=np.int32), ninv)
    _, chi2, _ = lik.calculate(v0 / u, u * t0)
    ld = np.linalg.slogdet(sm)[1] + logs.sum()
    assert abs(lik.logdet_raw - ld) <= tol + 4 * EPS * np.abs(logs).sum(), (abs(lik.logdet_raw - ld), tol)
    assert abs(chi2 - want) <= tol * max(size, want), (abs(chi2 / want - 1), tol)
    lik.close()
