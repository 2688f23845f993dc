"""The work a user of cosmopp_gb300 has it do, case by case, through its public entry points.

A case is a dict of plain values.  Sizes are those of cosmopp_gb300/workload.py: HEALPix nside 4 to
32, lmax = 3 nside - 1 or 3 nside, a Gaussian beam of 3520 / nside arcmin (440', 220', 110'), a mask
that keeps a share of the sky, C_l = 1e3 2 pi / (l (l + 1)), white noise of 0.5 to 1 muK.

kind "loglike"    Context.loglike: -2lnL, chi2, ln det C and, with grad, d(-2lnL)/dC_l of a batch of
                  C_l vectors on one map or one map per vector; precision "fp64" or "mixed"
kind "hmc"        Context.hmc: one trajectory of many chains over ln C_l
kind "likelihood" Likelihood(C, F, N).calculate(map): the packed drop-in, built and evaluated
kind "pol"        LikelihoodPolarization(C, ..., N^-1).calculate: the Q/U pixel likelihood
kind "cmatrix"    Context.build_cmatrix: packed covariance matrices on the host
"""
import math

import numpy as np
import torch

import cosmopp_gb300 as cg


def listed():
    return [
        # the smallest call: a coarse-map value, one C_l vector (a sampler's step on a toy problem)
        dict(name="fp64_value_nside4_b1", kind="loglike", precision="fp64", nside=4, lmax=12, n=150, sigma=1.0,
             batch=1, grad=False, maps=False),
        # one value and gradient at nside 8, lmax 24: an optimiser's or a single HMC chain's step
        dict(name="fp64_grad_nside8_b1", kind="loglike", precision="fp64", nside=8, lmax=24, n=614, sigma=1.0,
             batch=1, grad=True, maps=False),
        # the same at nside 16, lmax 47, 80 % of the sky: the size the low-l likelihood is used at
        dict(name="fp64_grad_nside16_b1", kind="loglike", precision="fp64", nside=16, lmax=47, n=2469, sigma=1.0,
             batch=1, grad=True, maps=False),
        # a batch of C_l vectors with gradients (several chains in step)
        dict(name="fp64_grad_nside16_b16", kind="loglike", precision="fp64", nside=16, lmax=47, n=2469, sigma=1.0,
             batch=16, grad=True, maps=False),
        # values only, one simulated map per C_l vector (calibration against simulations)
        dict(name="fp64_value_nside16_b8_maps", kind="loglike", precision="fp64", nside=16, lmax=47, n=2457,
             sigma=1.0, batch=8, grad=False, maps=True),
        # the largest: half the sky at nside 32, lmax 95, value and gradient
        dict(name="fp64_grad_nside32_b1", kind="loglike", precision="fp64", nside=32, lmax=95, n=6131, sigma=0.5,
             batch=1, grad=True, maps=False),
        # the batched mixed path at the benchmark's batch
        dict(name="mixed_grad_nside16_b256", kind="loglike", precision="mixed", nside=16, lmax=47, n=2469, sigma=1.0,
             batch=256, grad=True, maps=False),
        # the mixed path with a single vector, value only (one Metropolis-Hastings chain)
        dict(name="mixed_value_nside16_b1", kind="loglike", precision="mixed", nside=16, lmax=47, n=2469, sigma=1.0,
             batch=1, grad=False, maps=False),
        # one HMC trajectory of 64 chains on the mixed path
        dict(name="hmc_nside16_c64", kind="hmc", precision="mixed", nside=16, lmax=47, n=2469, sigma=1.0, batch=64,
             nleap=4),
        # the packed drop-in with a fiducial matrix and a foreground map, four maps after the set-up
        dict(name="likelihood_nside16", kind="likelihood", nside=16, lmax=47, n=2469, sigma=1.0, nmaps=4),
        # the Q/U likelihood of a masked nside 8 sky (2 x 614 kept values of 2 x 768), two maps
        dict(name="pol_nside8", kind="pol", npix=768, ngood=614, nmaps=2),
        # covariance matrices for a host program (a table of models), nside 16
        dict(name="cmatrix_nside16_b4", kind="cmatrix", nside=16, lmax=47, n=2469, batch=4),
    ]


def draw(rng):
    """One more case of the ranges above: 100 to 6144 pixels, batches 1 to 256, odd sizes."""
    kind = rng.choice(["fp64", "fp64", "fp64", "fp64", "mixed", "likelihood", "pol", "cmatrix"])
    nside = rng.choice([4, 8, 16])
    npix = 12 * nside * nside
    if kind == "pol":
        npix = 12 * rng.choice([4, 8]) ** 2
        ngood = max(24, int(npix * rng.uniform(0.3, 1.0)))
        return dict(kind="pol", npix=npix, ngood=ngood, nmaps=rng.randint(1, 3))
    if kind == "fp64" and rng.random() < 0.2:
        nside, npix = 32, 12 * 32 * 32
        n = int(math.exp(rng.uniform(math.log(1500), math.log(6131))))
    else:
        n = max(100, int(npix * rng.uniform(0.5, 1.0)))
    lmax = rng.randint(2 * nside, 3 * nside) if nside < 32 else rng.randint(60, 95)
    sigma = round(rng.uniform(0.5, 1.5), 2)
    if kind == "likelihood":
        return dict(kind="likelihood", nside=nside, lmax=lmax, n=n, sigma=sigma, nmaps=rng.randint(1, 6))
    if kind == "cmatrix":
        return dict(kind="cmatrix", nside=nside, lmax=lmax, n=n, batch=rng.randint(1, 4))
    if kind == "mixed":
        batch = int(math.exp(rng.uniform(0, math.log(256.99))))
        return dict(kind="loglike", precision="mixed", nside=nside, lmax=lmax, n=n, sigma=sigma, batch=batch,
                    grad=rng.random() < 0.6, maps=rng.random() < 0.3)
    most = max(1, min(100, int(2.3e11 / float(n) ** 3)))  # no more work than the largest listed case
    batch = int(math.exp(rng.uniform(0, math.log(most + 0.99))))
    return dict(kind="loglike", precision="fp64", nside=nside, lmax=lmax, n=n, sigma=sigma, batch=batch,
                grad=rng.random() < 0.6, maps=rng.random() < 0.3)


# ---- inputs ---------------------------------------------------------------------------------

def _fwhm(nside):
    return 3520.0 / nside / 60.0


def _pixels(case, rng):
    return np.sort(rng.permutation(12 * case["nside"] ** 2)[:case["n"]]).astype(np.int32)


def _fiducial(lmax):
    cl = np.zeros(lmax + 1)
    ell = np.arange(2, lmax + 1)
    cl[2:] = 1e3 * 2.0 * np.pi / (ell * (ell + 1.0))
    return cl


def _lognormal(cl, batch, rng):
    """10 % lognormal perturbations per l, the batches of workload.py"""
    out = cl[None, :] * np.exp(0.1 * rng.standard_normal((batch, len(cl))))
    out[:, :2] = 0.0
    return out


def _beam(lmax, nside):
    """Gaussian beam B_l = exp(-l (l + 1) sigma^2 / 2)"""
    s = _fwhm(nside) * math.pi / 180.0 / math.sqrt(8.0 * math.log(2.0))
    ell = np.arange(lmax + 1)
    return np.exp(-0.5 * ell * (ell + 1) * s * s)


def _ring_vectors(nside):
    """Unit vectors of the HEALPix RING pixel centres (Gorski et al. 2005)."""
    npix, ncap = 12 * nside * nside, 2 * nside * (nside - 1)
    p = np.arange(npix)
    z, phi = np.empty(npix), np.empty(npix)
    north = p < ncap
    south = p >= npix - ncap
    for cap, q, sign in ((north, p[north], 1.0), (south, npix - 1 - p[south], -1.0)):
        i = ((1 + np.sqrt(1 + 2 * q)) / 2).astype(np.int64)
        i = np.where(2 * i * (i - 1) > q, i - 1, i)
        i = np.where(2 * i * (i + 1) <= q, i + 1, i)
        j = q + 1 - 2 * i * (i - 1)
        if sign < 0:
            j = 4 * i + 1 - j
        z[cap] = sign * (1 - i * i / (3.0 * nside * nside))
        phi[cap] = (j - 0.5) * np.pi / (2 * i)
    belt = ~(north | south)
    q = p[belt] - ncap
    i, j = q // (4 * nside) + nside, q % (4 * nside) + 1
    z[belt] = 4.0 / 3.0 - 2.0 * i / (3.0 * nside)
    phi[belt] = np.pi / (2 * nside) * (j - 0.5 * (1 + (i + nside) % 2))
    st = np.sqrt((1 - z) * (1 + z))
    return np.stack([st * np.cos(phi), st * np.sin(phi), z], axis=1)


def _legendre(pix, nside, lmax, dev):
    """Yields (l, P_l(n_i . n_j)) for l = 0 .. lmax as [n, n] float64 tensors"""
    v = torch.tensor(_ring_vectors(nside)[pix], dtype=torch.float64, device=dev)
    x = (v @ v.T).clamp_(-1.0, 1.0)
    x.fill_diagonal_(1.0)
    p0, p1 = torch.ones_like(x), x.clone()
    yield 0, p0
    yield 1, p1
    for l in range(2, lmax + 1):
        p0, p1 = p1, (2 - 1.0 / l) * x * p1 - (1 - 1.0 / l) * p0
        yield l, p1


def _covariance(cls, pix, nside, dev):
    """[B, n, n] signal covariances of the C_l vectors [B, lmax + 1]"""
    lmax = cls.shape[1] - 1
    w = cls * ((2 * np.arange(lmax + 1) + 1) / (4 * np.pi) * _beam(lmax, nside) ** 2)
    w[:, :2] = 0.0
    out = torch.zeros((len(cls), len(pix), len(pix)), dtype=torch.float64, device=dev)
    for l, p in _legendre(pix, nside, lmax, dev):
        for b in range(len(cls)):
            out[b].add_(p, alpha=float(w[b, l]))
    return out


def _draw_maps(cov, count, rng):
    """count maps of covariance cov: L z with z ~ N(0, 1)"""
    L = torch.linalg.cholesky(cov)
    z = torch.tensor(rng.standard_normal((len(cov), count)), dtype=torch.float64, device=cov.device)
    return (L @ z).T.contiguous().cpu().numpy()


def _pack(m):
    """Reference packed storage: entry (i <= j) at j (j + 1) / 2 + i, on the host"""
    n = len(m)
    j, i = torch.tril_indices(n, n, device=m.device)
    return m[j, i].cpu().numpy()


def _inputs(case, seed, dev):
    """Host arrays of one seed, the same for every tree"""
    rng = np.random.default_rng([seed, 20131])
    kind = case["kind"]
    if kind == "pol":
        size = 2 * case["npix"]
        a = torch.tensor(rng.standard_normal((size, size)), dtype=torch.float64, device=dev) / math.sqrt(size)
        b = torch.tensor(rng.standard_normal((size, size)), dtype=torch.float64, device=dev) / math.sqrt(size)
        eye = torch.eye(size, dtype=torch.float64, device=dev)
        good = np.sort(rng.permutation(case["npix"])[:case["ngood"]]).astype(np.int32)
        n2 = 2 * case["ngood"]
        ninv = b @ b.T + 2.0 * eye
        return dict(c=_pack(a @ a.T + 0.5 * eye), ninv=((ninv + ninv.T) / 2).cpu().numpy(), good=good,
                    v=rng.standard_normal((case["nmaps"], n2)), sub=0.3 * rng.standard_normal((case["nmaps"], n2)))
    pix = _pixels(case, rng)
    fid = _fiducial(case["lmax"])
    if kind == "cmatrix":
        return dict(pix=pix, cls=_lognormal(fid, case["batch"], rng))
    cov = _covariance(fid[None, :], pix, case["nside"], dev)[0]
    noise = case["sigma"] ** 2
    eye = torch.eye(len(pix), dtype=torch.float64, device=dev)
    if kind == "likelihood":
        # the fiducial matrix of the low-l flow: a large monopole and dipole (1 + x) term
        v = torch.tensor(_ring_vectors(case["nside"])[pix], dtype=torch.float64, device=dev)
        f = 100.0 * float(fid[2]) * (1.0 + v @ v.T)
        maps = _draw_maps(cov + noise * eye, case["nmaps"], rng)
        x = _ring_vectors(case["nside"])[pix]
        return dict(c=_pack(cov), f=_pack((f + f.T) / 2), nz=_pack(noise * eye), maps=maps,
                    fg=np.cos(3 * x[:, 2]) + 0.3 * x[:, 0])
    maps = _draw_maps(cov + noise * eye, case["batch"] if case.get("maps") else 1, rng)
    cls = _lognormal(fid, case["batch"], rng)
    return dict(pix=pix, fid=fid, cls=cls, d=maps if case.get("maps") else maps[0])


def prepare(case, seed):
    inp = _inputs(case, seed, "cuda")
    kind = case["kind"]
    if kind in ("likelihood", "pol"):
        return dict(case=case, inp=inp)
    ctx = cg.Context(lmax=case["lmax"], fwhm_deg=_fwhm(case["nside"]), nside=case["nside"], good_pixels=inp["pix"],
                     scheme="RING", noise_sigma=case.get("sigma", 1.0), max_batch=case["batch"],
                     precision=case.get("precision", "fp64"),
                     cl_ref=inp["fid"] if case.get("precision") == "mixed" else None, recenter="fixed")
    return dict(case=case, inp=inp, ctx=ctx, seed=int(seed) % (1 << 31))


def run(state):
    case, inp = state["case"], state["inp"]
    kind = case["kind"]
    if kind == "loglike":
        r = state["ctx"].loglike(inp["cls"], inp["d"], grad=case["grad"])
        out = dict(m2lnl=r["m2lnl"], chi2=r["chi2"], logdet=r["logdet"], status=r["status"])
        if case["grad"]:
            out["grad"] = r["grad"]
        return out
    if kind == "hmc":
        chain, acc = state["ctx"].hmc(inp["d"], np.log(inp["cls"][:, 2:]), inp["fid"], niter=1, nleap=case["nleap"],
                                      tau=0.05, seed=state["seed"])
        return dict(chain=chain, accept=acc)
    if kind == "likelihood":
        lik = cg.Likelihood(inp["c"], inp["f"], inp["nz"], foreground=inp["fg"])
        out = np.array([lik.calculate(t) for t in inp["maps"]])
        lik.close()
        return out
    if kind == "pol":
        lik = cg.LikelihoodPolarization(inp["c"], case["npix"], inp["good"], inp["ninv"])
        out = np.array([lik.calculate(v, s) for v, s in zip(inp["v"], inp["sub"])])
        lik.close()
        return out
    return state["ctx"].build_cmatrix(inp["cls"])


def work(case):
    """Least work of one pass: matrix factorisation n^3 / 3, a triangular solve n^2 per right-hand
    side, the gradient's traces through the (lmax + 1)^2 - 4 harmonics of the pixels, the Legendre
    recurrence per pixel pair where C itself is formed; inputs read and outputs written once."""
    kind = case["kind"]
    if kind == "pol":
        n, size = 2.0 * case["ngood"], 2.0 * case["npix"]
        return dict(bytes=8.0 * (size * (size + 1) / 2 + size * size + 4 * case["nmaps"] * n),
                    flops=4.0 * n ** 3 + n ** 3 / 3 + case["nmaps"] * 4 * n * n)
    n, lmax = float(case["n"]), case["lmax"]
    pairs, l1, nh = n * (n + 1) / 2, lmax + 1, (lmax + 1) ** 2 - 4
    if kind == "cmatrix":
        return dict(bytes=8.0 * case["batch"] * (pairs + l1), flops=4.0 * pairs * l1 * case["batch"])
    if kind == "likelihood":
        return dict(bytes=8.0 * (3 * pairs + case["nmaps"] * n), flops=n ** 3 / 3 + 2 * n * n * (case["nmaps"] + 1))
    B = case["batch"]
    evals = B * (case["nleap"] + 1) if kind == "hmc" else B
    grad = kind == "hmc" or case["grad"]
    flops = 4.0 * pairs * l1 + n ** 3 / 3 + n * n + (n * n * nh if grad else 0.0)
    maps = B if case.get("maps") else 1
    return dict(bytes=8.0 * (B * l1 + maps * n + B * (4 + (l1 if grad else 0))), flops=evals * flops)


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    kind = case["kind"]
    if kind == "hmc" or (kind == "loglike" and case["batch"] * (case["n"] / 2500.0) ** 3 > 24):
        return None
    inp = _inputs(case, seed, dev)
    if kind == "cmatrix":
        cov = _covariance(inp["cls"], inp["pix"], case["nside"], dev)
        return np.stack([_pack(c) for c in cov])
    t = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)
    if kind == "pol":
        size, ng = 2 * case["npix"], case["ngood"]
        c = torch.zeros((size, size), dtype=torch.float64, device=dev)
        j, i = torch.tril_indices(size, size, device=dev)
        c[j, i] = t(inp["c"])
        c[i, j] = t(inp["c"])
        k = torch.tensor(np.concatenate([inp["good"], case["npix"] + inp["good"]]), device=dev, dtype=torch.long)
        c, ninv = c[k][:, k], t(inp["ninv"])[k][:, k]
        m = ninv + ninv @ c @ ninv
        m = (m + m.T) / 2
        L = torch.linalg.cholesky(m)
        logdet = 2.0 * float(torch.log(torch.diagonal(L)).sum()) - cg.DET_OFFSET_POL
        out = []
        for v, s in zip(inp["v"], inp["sub"]):
            w = t(v) - ninv @ t(s)
            chi2 = float((torch.linalg.solve_triangular(L, w[:, None], upper=False) ** 2).sum())
            out.append((chi2 + logdet, chi2, logdet))
        return np.array(out)
    if kind == "likelihood":
        n = case["n"]
        m = torch.zeros((n, n), dtype=torch.float64, device=dev)
        j, i = torch.tril_indices(n, n, device=dev)
        m[j, i] = t(inp["c"]) + t(inp["f"]) + t(inp["nz"])
        L = torch.linalg.cholesky(m)
        base = 2.0 * float(torch.log(torch.diagonal(L)).sum()) + cg.DET_OFFSET
        fw = torch.linalg.solve_triangular(L, t(inp["fg"])[:, None], upper=False)[:, 0]
        ff = float(fw @ fw)
        out = []
        for d in inp["maps"]:
            y = torch.linalg.solve_triangular(L, t(d)[:, None], upper=False)[:, 0]
            # the foreground is marginalised (source/likelihood.cpp:171-177); the offset is added
            # to ln det before the marginal's log term
            chi2 = float(y @ y) - float(y @ fw) ** 2 / ff
            logdet = base + math.log(ff / n)
            out.append((chi2 + logdet, chi2, logdet))
        return np.array(out)
    B, lmax, n = case["batch"], case["lmax"], case["n"]
    eye = case["sigma"] ** 2 * torch.eye(n, dtype=torch.float64, device=dev)
    res = dict(m2lnl=np.zeros(B), chi2=np.zeros(B), logdet=np.zeros(B), status=None)
    if case["grad"]:
        res["grad"] = np.zeros((B, lmax + 1))
    bl = _beam(lmax, case["nside"])
    for b in range(B):
        c = _covariance(inp["cls"][b:b + 1], inp["pix"], case["nside"], dev)[0] + eye
        L = torch.linalg.cholesky(c)
        d = t(inp["d"][b] if case["maps"] else inp["d"])
        y = torch.linalg.solve_triangular(L, d[:, None], upper=False)[:, 0]
        res["chi2"][b] = float(y @ y)
        res["logdet"][b] = 2.0 * float(torch.log(torch.diagonal(L)).sum())
        res["m2lnl"][b] = res["chi2"][b] + res["logdet"][b]
        if case["grad"]:
            w = torch.cholesky_inverse(L)
            a = w @ d
            w = w - a[:, None] * a[None, :]
            for l, p in _legendre(inp["pix"], case["nside"], lmax, dev):
                if l >= 2:
                    g = float((w * p).sum())
                    res["grad"][b, l] = g * (2 * l + 1) / (4 * math.pi) * bl[l] ** 2
    return res
