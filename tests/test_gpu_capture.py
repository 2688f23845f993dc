"""FP64 calls captured by the caller: the workspace depends on the number of elements alone, so a gradient call can be
captured after value calls, and what was captured stays valid through later calls of either kind.  Sizes where a
step runs on one stream and where its update is forked to a second one; both gradient routes."""
import numpy as np
import pytest
import torch

import cosmopp_gb300 as cg
from cosmopp_gb300 import workload as W

pytestmark = pytest.mark.gpu


class _Call:
    """a device call of B elements, its buffers and, once captured, its graph"""

    def __init__(self, ctx, cls, d, grad):
        t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")
        self.ctx, self.B, self.grad = ctx, len(cls), grad
        self.cl, self.d = t(cls), t(d)
        self.out = {k: t(np.zeros(self.B)) for k in ("m2lnl", "chi2", "logdet")}
        if grad:
            self.out["grad"] = t(np.zeros(cls.shape))
        torch.cuda.synchronize()

    def run(self, stream):
        o = self.out
        self.ctx.loglike_device(self.B, self.cl.data_ptr(), self.d.data_ptr(), 0, o["m2lnl"].data_ptr(),
                                o["chi2"].data_ptr(), o["logdet"].data_ptr(), o["grad"].data_ptr() if self.grad else None,
                                stream=stream.cuda_stream)

    def capture(self, stream):
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph, stream=stream, capture_error_mode="relaxed"):
            self.run(torch.cuda.current_stream())

    def replay(self):
        for o in self.out.values():
            o.zero_()
        self.graph.replay()
        torch.cuda.synchronize()
        return {k: v.cpu().numpy() for k, v in self.out.items()}


@pytest.mark.parametrize("norm", [1.0, 1.0 + 1e-13], ids=["harmonics", "inverse"])
@pytest.mark.parametrize("n,lmax,batch", [(150, 9, 3), (1300, 20, 2)])
def test_captured_calls(n, lmax, batch, norm):
    rng = np.random.default_rng(n)
    v = rng.standard_normal((n, 3))
    v *= norm / np.linalg.norm(v, axis=1)[:, None]
    cls = W.lognormal_batch(W.fiducial_cl(lmax), batch, n)
    d = 20.0 * rng.standard_normal(n)
    stream = torch.cuda.Stream()
    with cg.Context(lmax=lmax, fwhm_deg=9.0, dirs=v, noise_sigma=2.0, max_batch=batch) as ctx:
        want = [ctx.loglike(cls, d)]                    # value calls only until the captures are done
        calls = [_Call(ctx, cls, d, False), _Call(ctx, cls, d, True)]
        for c in calls:
            c.capture(stream)
        got = [c.replay() for c in calls]
        want.append(ctx.loglike(cls, d, grad=True))
        again = [c.replay() for c in calls]
        later = [ctx.loglike(cls, d), ctx.loglike(cls, d, grad=True)]
        for k in (0, 1):
            assert np.all(want[k]["status"] == cg.CG_OK)
            for name in calls[k].out:
                for r in (got, again, later):
                    assert np.array_equal(r[k][name], want[k][name]), (k, name)


def test_the_first_gradient_call_allocates_nothing():
    n, lmax = 400, 20
    rng = np.random.default_rng(1)
    v = rng.standard_normal((n, 3))
    v /= np.linalg.norm(v, axis=1)[:, None]
    cls, d = W.lognormal_batch(W.fiducial_cl(lmax), 40, 1), 20.0 * rng.standard_normal(n)
    with cg.Context(lmax=lmax, fwhm_deg=9.0, dirs=v, noise_sigma=2.0, max_batch=40) as ctx:
        ctx.loglike(cls, d)
        free = torch.cuda.mem_get_info()[0]
        ctx.loglike(cls, d, grad=True)
        # (loading the gradient's kernels may take a little)
        assert free - torch.cuda.mem_get_info()[0] < (16 << 20)
