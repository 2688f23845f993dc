"""A C_l that is not a number leaves no number behind: every output of that element (the gradient from l = 2 on)
is NaN, whatever the size (one block, whose factor replaces what it cannot scale, or several), and with no status
asked for; its neighbours keep the bits of a call of their own."""
import numpy as np
import pytest
import torch

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norm", [1.0, 1.0 + 1e-13], ids=["harmonics", "inverse"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("n", [5, 64, 130])
def test_outputs_of_a_nonfinite_element(n, bad, norm):
    rng = np.random.default_rng(n)
    lmax = 8
    v = rng.standard_normal((n, 3))
    v *= norm / np.linalg.norm(v, axis=1)[:, None]
    cls = W.lognormal_batch(W.fiducial_cl(lmax), 3, n)
    d = 20.0 * rng.standard_normal(n)
    good = cls.copy()
    cls[1, 5] = bad
    with cg.Context(lmax=lmax, fwhm_deg=9.0, dirs=v, noise_sigma=2.0, max_batch=3) as ctx:
        for grad in (True, False):
            want = ctx.loglike(good, d, grad=grad)
            r = ctx.loglike(cls, d, grad=grad)
            assert list(r["status"]) == [cg.CG_OK, cg.CG_ERR_NONFINITE, cg.CG_OK]
            for name in ("m2lnl", "chi2", "logdet") + (("grad",) if grad else ()):
                assert np.all(np.isnan(r[name][1][2:] if name == "grad" else r[name][1])), name
                assert np.array_equal(r[name][::2], want[name][::2]), name
        t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")
        tc, td, m2 = t(cls), t(d), t(np.zeros(3))
        torch.cuda.synchronize()
        ctx.loglike_device(3, tc.data_ptr(), td.data_ptr(), 0, m2.data_ptr(), stream=torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        m2 = m2.cpu().numpy()
        assert np.isnan(m2[1]) and np.array_equal(m2[::2], want["m2lnl"][::2])
