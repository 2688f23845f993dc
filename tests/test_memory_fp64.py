"""Memory admission of the FP64 path: the harmonics' rows of the gradient cost no more than 24 GB or the route through
C^-1 (planned for directions off the unit sphere), whichever is more."""
import numpy as np
import pytest

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

GB = 10 ** 9


def _plans(n, lmax, batch, budget):
    rng = np.random.default_rng(n)
    v = rng.standard_normal((n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    kw = dict(lmax=lmax, fwhm_deg=1.0, noise_sigma=1.0, max_batch=batch)
    return cg.plan_memory(budget, dirs=v, **kw), cg.plan_memory(budget, dirs=1.001 * v, **kw)


@pytest.mark.parametrize("n,lmax,batch", [(150, 12, 1), (150, 12, 30000), (190, 100, 6000), (2469, 47, 16), (2469, 47, 256),
                                          (6131, 95, 8), (6131, 95, 64), (11039, 95, 100)])
def test_workspace_of_a_piece(n, lmax, batch):
    p, q = _plans(n, lmax, batch, 280 * GB)
    assert q["chunk"] == min(batch, q["max_batch_fit"])
    assert p["bytes_per_element"] > q["bytes_per_element"]      # the harmonics' route
    staging = q["bytes_fixed"]                                  # geometry and staging, the same for both
    used = p["bytes_fixed"] - staging + p["chunk"] * p["bytes_per_element"]
    assert used <= max(24 << 30, batch * q["bytes_per_element"])
    # no smaller than that asks for
    if p["chunk"] < min(batch, p["max_batch_fit"]):
        assert used + p["bytes_per_element"] > max(24 << 30, batch * q["bytes_per_element"])
    assert 1 <= p["chunk"] <= min(batch, p["max_batch_fit"])


@pytest.mark.gpu
def test_pieces_keep_the_bits_of_a_call_of_their_own():
    """Few pixels and many l: a batch that runs in two pieces, the largest smaller than it."""
    n, lmax, batch = 190, 100, 650
    p, _ = _plans(n, lmax, batch, 280 * GB)
    assert p["chunk"] < batch
    rng = np.random.default_rng(2)
    v = rng.standard_normal((n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    cls, d = W.lognormal_batch(W.fiducial_cl(lmax), batch, 2), 20.0 * rng.standard_normal(n)
    with cg.Context(lmax=lmax, fwhm_deg=1.0, dirs=v, noise_sigma=1.0, max_batch=batch) as ctx:
        full = ctx.loglike(cls, d, grad=True)
        assert np.all(full["status"] == cg.CG_OK)
        for b in (0, batch // 2 - 1, batch // 2, batch - 1):
            one = ctx.loglike(cls[b:b + 1], d, grad=True)
            for name in ("m2lnl", "chi2", "logdet", "grad"):
                assert np.array_equal(full[name][b], one[name][0]), (name, b)
