"""The calls a user of this library makes, with inputs: the linear power spectrum, its gradients and
the CMB spectra of drawn cosmologies, at the sizes of the library's own workloads, defaults and tests.

``listed`` gives the fixed cases, ``draw`` one more of the same ranges; ``prepare`` makes what a
program holds before the call (parameters, backgrounds, the problem objects that keep device
inputs), ``run`` is one pass through the public entry points, ``work`` the bytes and operations that
pass cannot do without and ``exact`` its outputs in plain 64-bit torch where they have a closed form.
"""
import math
import os
import sys
import warnings

import numpy as np
import torch

# the package lives one folder below the repository's root (the working folder)
_PKG = os.path.join(os.getcwd(), "disco-eb_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from discoeb_b200 import cmb, gradients, observables, perturbations  # noqa: E402
from discoeb_b200.background import evolve_background  # noqa: E402
from discoeb_b200.workloads import A_OUT_4Z, W0_LCDM, cosmo_params, crosses_phantom_divide, sample_thetas  # noqa: E402

# the hierarchy sizes in use: the reference's defaults, the P(k) workloads (with and without a
# massive neutrino), and the CMB workload at l_max 50
_SIZES = {
    "default": dict(lmaxg=11, lmaxgp=11, lmaxr=11, lmaxnu=8, nqmax=3),
    "massless": dict(lmaxg=12, lmaxgp=12, lmaxr=17, lmaxnu=3, nqmax=3),
    "mnu": dict(lmaxg=12, lmaxgp=12, lmaxr=17, lmaxnu=17, nqmax=5),
    "lmax50": dict(lmaxg=50, lmaxgp=50, lmaxr=17, lmaxnu=17, nqmax=5),
    "ragged": dict(lmaxg=9, lmaxgp=10, lmaxr=13, lmaxnu=6, nqmax=4),
}
_OUTPUTS = {1: (1.0,), 2: (0.5, 1.0), 4: tuple(A_OUT_4Z)}  # scale factors: z = 0; 1, 0; 2, 1, 0.5, 0


def listed():
    return [
        # the smallest solve: a few modes at the defaults (interactive use, one likelihood bin)
        dict(name="pk_default_k16", kind="pk", size="default", num_k=16, kmax=0.5, nout=1, rtol=1e-4, atol=1e-4),
        # P(k) of a massless-neutrino cosmology, the small workload
        dict(name="pk_massless_k128", kind="pk", size="massless", num_k=128, kmax=1.0, nout=1, rtol=1e-5, atol=1e-8),
        # P(k) at four redshifts with a massive neutrino, the batched workload
        dict(name="pk_mnu_k512_z4", kind="pk", size="mnu", num_k=512, kmax=10.0, nout=4, rtol=1e-5, atol=1e-8),
        # a batch of cosmologies in one launch (training set of an emulator)
        dict(name="pk_batch_c48_k256", kind="batch", size="mnu", n_cosmo=48, num_k=256, kmax=5.0, nout=1, rtol=1e-5,
             atol=1e-8),
        # P(k) with its Jacobian, the gradient workload (a Fisher forecast)
        dict(name="jac_mnu_k512_z4", kind="jac", size="mnu", num_k=512, kmax=10.0, nout=4, rtol=1e-5, atol=1e-8),
        # the same for a few cosmologies at once (chains of a gradient sampler), a ragged mode count
        dict(name="jac_batch_c3_k203", kind="jac_batch", size="mnu", n_cosmo=3, num_k=203, kmax=5.0, nout=1, rtol=1e-5,
             atol=1e-8),
        # reverse mode: the gradient of a scalar loss of P(k) (forward, recorded, then backward)
        dict(name="adjoint_mnu_k96", kind="adjoint", size="mnu", num_k=96, kmax=1.0, nout=2, rtol=1e-5, atol=1e-8),
        # C_l^TT of a cosmology at the defaults
        dict(name="cl_tt", kind="cl", size="default", nmodes=128, ellmax=2500, n_k_dense=8192, n_fftlog=16384,
             pol=False),
        # temperature and polarisation spectra, odd sizes
        dict(name="cl_tt_te_ee", kind="cl", size="ragged", nmodes=101, ellmax=1999, n_k_dense=5001, n_fftlog=8192,
             pol=True),
        # C_l^TT with its gradient at the defaults
        dict(name="cl_jac", kind="cl_jac", size="default", nmodes=128, ellmax=2500, n_k_dense=8192, n_fftlog=16384),
        # the same with long photon hierarchies
        dict(name="cl_jac_lmax50", kind="cl_jac", size="lmax50", nmodes=80, ellmax=1200, n_k_dense=2048,
             n_fftlog=8192),
        # what is made of P(k) afterwards: smoothed power, Kaiser multipoles and the correlation function
        dict(name="observables_k2048", kind="observables", num_k=2048, ell=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pk", "pk", "states", "batch", "jac", "jac_batch", "adjoint", "cl", "cl_jac", "los",
                       "observables"])
    size = rng.choice(["default", "massless", "mnu", "ragged"])
    tol = rng.choice([dict(rtol=1e-4, atol=1e-4), dict(rtol=1e-5, atol=1e-8)])
    kmax = round(math.exp(rng.uniform(math.log(0.2), math.log(8.0))), 4)
    nout = rng.choice([1, 2, 4])
    grid = dict(ellmax=_log_int(rng, 300, 2500), n_k_dense=_log_int(rng, 700, 8192),
                n_fftlog=rng.choice([4096, 8192, 16384]))
    if kind in ("pk", "jac"):
        return dict(kind=kind, size=size, num_k=_log_int(rng, 4, 512), kmax=kmax, nout=nout, **tol)
    if kind == "states":
        return dict(kind=kind, size=size, num_k=_log_int(rng, 4, 256), kmax=min(kmax, 2.0), nout=_log_int(rng, 8, 200),
                    **tol)
    if kind in ("batch", "jac_batch"):
        return dict(kind=kind, size=size, n_cosmo=rng.randint(2, 32 if kind == "batch" else 3),
                    num_k=_log_int(rng, 16, 200), kmax=min(kmax, 5.0), nout=nout, **tol)
    if kind == "adjoint":
        return dict(kind=kind, size=size, num_k=_log_int(rng, 4, 96), kmax=min(kmax, 1.0), nout=rng.choice([1, 2]),
                    **tol)
    if kind == "cl":
        return dict(kind=kind, size=rng.choice(["default", "ragged", "mnu"]), nmodes=_log_int(rng, 32, 200),
                    pol=rng.random() < 0.4, **grid)
    if kind == "cl_jac":
        return dict(kind=kind, size=rng.choice(["default", "ragged"]), nmodes=_log_int(rng, 32, 128), **grid)
    if kind == "los":
        return dict(kind=kind, nmodes=_log_int(rng, 32, 200), ntau=_log_int(rng, 200, 600), pol=rng.random() < 0.4,
                    **grid)
    return dict(kind=kind, num_k=2 * _log_int(rng, 64, 4096), ell=rng.choice([0, 2, 4]))


def _theta(rng):
    """A cosmology around the LCDM point: the sampled box without its dark-energy directions (the
    fluid equations are singular where w crosses -1)."""
    u = rng.uniform(size=6)
    return dict(omega_c=0.11 + 0.02 * u[0], omega_b=0.0215 + 0.002 * u[1], h=0.64 + 0.08 * u[2],
                n_s=0.94 + 0.05 * u[3], ln10As=2.95 + 0.2 * u[4], w0=W0_LCDM, wa=0.0, m_nu=0.04 + 0.1 * u[5])


def _thetas(rng, n):
    """Cosmologies of the many-cosmology box whose w(a) stays on one side of -1."""
    got, seed = [], int(rng.integers(1 << 30))
    while len(got) < n:
        got += [t for t in sample_thetas(4 * n, seed) if not crosses_phantom_divide(t)]
        seed += 1
    return got[:n]


def _params(theta, massive=True):
    t = dict(theta)
    return cosmo_params(h=t["h"], omega_b=t["omega_b"], omega_c=t["omega_c"], A_s=math.exp(t["ln10As"]) / 1e10,
                        n_s=t["n_s"], m_nu=t["m_nu"] if massive else 0.0, w0=t["w0"], wa=t["wa"])


def _background(theta, massive=True):
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        return evolve_background(param=_params(theta, massive))


def _recomb_tau(ntau):
    """Output times like the pipeline's: dense through recombination, sparse before and after."""
    n1, n2 = ntau // 5, ntau // 2
    return np.concatenate([np.geomspace(5.0, 180.0, n1, endpoint=False), np.linspace(180.0, 420.0, n2, endpoint=False),
                           np.geomspace(420.0, 14000.0, ntau - n1 - n2)])


def prepare(case, seed):
    c, rng = dict(case), np.random.default_rng(seed)
    kind = c["kind"]
    if kind == "observables":
        n = c["num_k"]
        k = np.geomspace(1e-4, 20.0, n)
        # transfer-function-like amplitudes with acoustic wiggles, and noise at the solver's level
        q = k / 0.015
        delta = 6e4 * k**2 * np.log(1 + 0.17 * q) / (0.17 * q) / (1 + 3.9 * q + (1.6 * q) ** 2) ** 0.5
        delta = delta / (1 + 0.3 * q) * (1 + 0.03 * np.sin(105.0 * k) * np.exp(-((k / 0.2) ** 2)))
        y = rng.standard_normal((n, 20))
        y[:, 4] = -delta * (1 + 1e-6 * rng.standard_normal(n))
        y[:, 5] = 0.52 * delta * (1 + 1e-6 * rng.standard_normal(n))
        param = dict(A_s=2.1e-9 * rng.uniform(0.9, 1.1), n_s=rng.uniform(0.94, 0.98), k_p=0.05)
        return dict(c, k=k, y=y, param=param, d_k=torch.from_numpy(k).cuda(), d_y=torch.from_numpy(y).cuda(),
                    bias=float(rng.uniform(1.0, 2.5)))
    if kind == "los":
        tau = _recomb_tau(c["ntau"])
        k = np.geomspace(1e-4, 0.5, c["nmodes"])
        S = np.exp(-0.5 * ((tau[None, :] - 280.0) / 18.0) ** 2) * np.cos(160.0 * k[:, None] + rng.uniform(0, 6)) / 18.0
        S = S * (1 + 0.1 * rng.standard_normal()) + 1e-5 * np.exp(-((k[:, None] * 50) ** 2)) * tau[None, :] / 14000.0
        return dict(c, k=k, tau=tau, tau0=14000.0 + 30.0 * float(rng.uniform(0.5, 1.0)),
                    d_k=torch.from_numpy(k).cuda(), d_tau=torch.from_numpy(tau).cuda(), d_S=torch.from_numpy(S).cuda())
    if kind == "cl":
        theta = _theta(rng)
        return dict(c, param=_params(theta))
    if kind == "cl_jac":
        return dict(c, theta=_theta(rng))
    L = _SIZES[c["size"]]
    aexp = np.geomspace(0.01, 1.0, c["nout"]) if kind == "states" else np.array(_OUTPUTS[c["nout"]])
    opts = dict(L, rtol=c["rtol"], atol=c["atol"])
    if kind in ("pk", "states"):
        bg = _background(_theta(rng), massive=c["size"] != "massless")
        return dict(c, bg=bg, aexp=aexp, opts=dict(opts, max_steps=100000, kmin=1e-4, kmax=c["kmax"], num_k=c["num_k"],
                                                   k_sampling_method="log"))
    if kind == "jac":
        return dict(c, theta=_theta(rng), opts=dict(opts, aexp_out=aexp, kmin=1e-4, kmax=c["kmax"], num_k=c["num_k"]))
    kmodes = np.geomspace(1e-4, c["kmax"], c["num_k"])
    if kind == "batch":
        params = perturbations.backgrounds([_params(t) for t in _thetas(rng, c["n_cosmo"])])
        return dict(c, problem=perturbations.CosmologyBatch(params=params, kmodes=kmodes, aexp_out=aexp, **opts))
    if kind == "jac_batch":
        return dict(c, problem=gradients.JacobianBatch(_thetas(rng, c["n_cosmo"]), kmodes=kmodes, aexp_out=aexp,
                                                       **opts))
    if kind == "adjoint":
        prob = gradients.AdjointProblem(_theta(rng), kmodes=kmodes, aexp_out=aexp, **opts)
        weights = rng.uniform(0.5, 2.0, size=(c["num_k"], c["nout"])) * kmodes[:, None] ** 1.5
        return dict(c, problem=prob, weights=weights)
    raise ValueError(kind)


def run(state):
    s = state
    kind = s["kind"]
    if kind in ("pk", "states"):
        y, k, param = perturbations.evolve_perturbations(param=dict(s["bg"]), aexp_out=s["aexp"],
                                                         return_full=kind == "states", **s["opts"])
        if kind == "states":
            return y
        return perturbations.get_power(k=k[:, None], y=y, idx=4, param=param), y
    if kind in ("batch", "jac_batch"):
        s["problem"].launch()
        r = s["problem"].result()
        return r[0] if kind == "batch" else r[:2]
    if kind == "jac":
        return gradients.power_spectrum_jacobian(s["theta"], **s["opts"])[1:]
    if kind == "adjoint":
        p = s["problem"]
        p.launch_forward()
        P = p.forward_power()[0][0]
        p.launch_backward(s["weights"])
        return P, p.gradient(s["weights"])
    if kind == "cl":
        out, _ = cmb.compute_Cell_spectrum_from_cosmo_params(
            s["param"], ellmax=s["ellmax"], nmodes=s["nmodes"], n_k_dense=s["n_k_dense"], n_fftlog=s["n_fftlog"],
            spectra=("TT", "TE", "EE") if s["pol"] else ("TT",), **_SIZES[s["size"]])
        return out
    if kind == "cl_jac":
        cell, J, _ = cmb.compute_Cell_jacobian(s["theta"], ellmax=s["ellmax"], nmodes=s["nmodes"],
                                               n_k_dense=s["n_k_dense"], n_fftlog=s["n_fftlog"], **_SIZES[s["size"]])
        return cell, J
    if kind == "los":
        return cmb.compute_theta_ell(s["ellmax"], s["d_k"], s["d_tau"], s["d_S"], s["tau0"], n_fftlog=s["n_fftlog"],
                                     n_k_dense=s["n_k_dense"], kind="E" if s["pol"] else "T")
    smooth = observables.get_power_smoothed(k=s["k"], y=s["d_y"], dlogk=0.2, idx=4, param=s["param"])
    multi = observables.power_multipoles(y=s["d_y"], kmodes=s["d_k"], b=s["bias"], param=s["param"])
    xi, r = observables.get_xi_from_P(k=s["d_k"], Pk=smooth, ell=s["ell"])
    return smooth, multi, xi, r


def _n(size):
    return perturbations.nvar_of(**_SIZES[size])


def _attempts(kmax, num_k, rtol):
    """Step attempts of num_k modes over [1e-4, kmax] (log-spaced): the per-mode counts of the
    P(k) workload at rtol 1e-5, scaled by the order of the error estimate."""
    lk = np.log([1e-4, 1e-3, 1e-2, 0.1, 0.5, 1.0, 3.0, 10.0])
    n = np.array([77.0, 145.0, 360.0, 345.0, 362.0, 450.0, 860.0, 1410.0])
    return float(np.interp(np.linspace(lk[0], math.log(kmax), num_k), lk, n).sum() * (1e-5 / rtol) ** (1.0 / 6.0) * 0.7)


# operations per state entry and step attempt of the structured Rosenbrock step (eight right-hand
# sides and banded solves, one factorisation); a tangent direction costs about twice that
_FLOPS = 840.0


def work(case):
    c = case
    kind = c["kind"]
    if kind == "observables":
        n = c["num_k"]
        return {"bytes": 8.0 * n * (20 + 2 + 6), "flops": n * (60.0 + 10.0 * math.log2(n))}
    if kind in ("los", "cl", "cl_jac"):
        nt = c.get("ntau", 320)
        rows, nl, nf = c["n_k_dense"], c["ellmax"] + 1, c["n_fftlog"]
        los = 2.0 * rows * nl * (nf + 2) + 2.5 * rows * nf * math.log2(nf) * 2
        if kind == "los":
            return {"bytes": 8.0 * (c["nmodes"] * nt + rows * nl), "flops": los * (2 if c["pol"] else 1)}
        n = _n(c["size"])
        steps = _attempts(1.0, c["nmodes"], 1e-4) + 0.3 * c["nmodes"] * nt
        flops = steps * n * _FLOPS + c["nmodes"] * nt * n * 60.0
        if kind == "cl":
            return {"bytes": 8.0 * nl * (3 if c["pol"] else 1) + 8.0 * c["nmodes"] * n,
                    "flops": flops + los * (3 if c["pol"] else 1)}
        return {"bytes": 8.0 * nl * 9 + 8.0 * c["nmodes"] * n * 7, "flops": flops * 13.0 + los * 8}
    n, modes = _n(c["size"]), c["num_k"] * c.get("n_cosmo", 1)
    flops = _attempts(c["kmax"], c["num_k"], c["rtol"]) * c.get("n_cosmo", 1) * n * _FLOPS
    byt = 8.0 * modes * (n + 5) + 8.0 * modes * c["nout"] * (n if kind == "states" else 21)
    if kind in ("jac", "jac_batch"):
        return {"bytes": byt + 8.0 * modes * (6 * n + 8 * c["nout"]), "flops": flops * 13.0}
    if kind == "adjoint":
        return {"bytes": byt + 8.0 * modes * n, "flops": flops * 5.0}
    return {"bytes": byt, "flops": flops}


# ---- closed forms in 64 bits -------------------------------------------------------------------
_LANCZOS = (0.99999999999980993227684700473478, 676.520368121885098567009190444019, -1259.13921672240287047156078755283,
            771.3234287776530788486528258894, -176.61502916214059906584551354, 12.507343278686904814458936853,
            -0.13857109526572011689554707, 9.984369578019570859563e-6, 1.50563273514931155834e-7)


def _loggamma(z):
    """log Gamma(z) for Re z > 0.5 or by reflection (Lanczos), complex torch."""
    low = z.real <= 0.5
    w = torch.where(low, 1.0 - z, z) - 1.0
    acc = torch.full_like(w, _LANCZOS[0])
    for j in range(1, 9):
        acc = acc + _LANCZOS[j] / (w + j)
    lg = (w + 0.5) * torch.log(w + 7.5) - (w + 7.5) + 0.5 * math.log(2 * math.pi) + torch.log(acc)
    # log sin(pi z) without overflow for large |Im z|
    s = torch.where(z.imag >= 0, 1.0, -1.0)
    ls = -1j * s * math.pi * z + torch.log((1 - torch.exp(2j * s * math.pi * z)) / 2) + 1j * s * math.pi / 2
    return torch.where(low, math.log(math.pi) - ls - lg, lg)


def _spline_second(x, Y):
    """Second derivatives of natural cubic splines through (x [n], Y [n, m])."""
    n = x.shape[0]
    h = np.diff(x)
    S, cp, dp = np.zeros_like(Y), np.zeros(n), np.zeros_like(Y)
    for i in range(1, n - 1):
        d = 6.0 * ((Y[i + 1] - Y[i]) / h[i] - (Y[i] - Y[i - 1]) / h[i - 1])
        den = 2.0 * (h[i - 1] + h[i]) - h[i - 1] * cp[i - 1]
        cp[i] = h[i] / den
        dp[i] = (d - h[i - 1] * dp[i - 1]) / den
    for i in range(n - 2, 0, -1):
        S[i] = dp[i] - cp[i] * S[i + 1]
    return S


def _spline(x, Y, xn):
    S = _spline_second(x, Y)
    i = np.clip(np.searchsorted(x, xn, side="left") - 1, 0, x.shape[0] - 2)
    h = (x[i + 1] - x[i])[:, None]
    B = (xn - x[i])[:, None] / h
    A = 1.0 - B
    return A * Y[i] + B * Y[i + 1] + ((A**3 - A) * S[i] + (B**3 - B) * S[i + 1]) * h**2 / 6.0


def _theta_exact(c, s):
    dev = s["d_S"].device
    k, S = s["k"], s["d_S"].cpu().numpy()
    lkd = np.linspace(math.log(k[0]), math.log(k[-1]), c["n_k_dense"])
    S = _spline(np.log(k), S, lkd)
    chi = (s["tau0"] - s["tau"])[::-1]
    nf = c["n_fftlog"]
    lo, hi = math.log(max(chi[0], 1.0)) - 2.0, math.log(chi[-1]) + 2.0
    dl = (hi - lo) / nf
    lf = lo + np.arange(nf) * dl
    Sf = _spline(np.log(np.maximum(chi, 1e-10)), np.ascontiguousarray(S[:, ::-1].T), np.log(np.exp(lf)))
    F = torch.from_numpy(np.ascontiguousarray(Sf.T)).to(dev) * torch.from_numpy(np.exp(lf) ** 1.1).to(dev)
    eta = 2.0 * math.pi * torch.arange(nf // 2 + 1, dtype=torch.float64, device=dev) / (nf * dl)
    p = torch.complex(torch.full_like(eta, -1.1), eta)
    kd = torch.from_numpy(lkd).to(dev)
    ck = torch.fft.rfft(F, dim=1) * torch.exp(-1j * eta * lo) / nf * torch.exp(-(p[None] + 1.0) * kd[:, None])
    ell = torch.arange(c["ellmax"] + 1, dtype=torch.float64, device=dev)[:, None]
    M = torch.exp((p[None] - 1.0) * math.log(2.0) + 0.5 * math.log(math.pi) + _loggamma((1.0 + ell + p[None]) / 2.0)
                  - _loggamma((2.0 + ell - p[None]) / 2.0))
    w = torch.full_like(eta, 2.0)
    w[0] = w[-1] = 1.0
    th = (ck.real * w) @ M.real.T
    im = w.clone()
    im[0] = im[-1] = 0.0
    return th - (ck.imag * im) @ M.imag.T, torch.exp(kd)


def exact(case, seed):
    c = case
    if c["kind"] == "los" and not c["pol"]:
        return _theta_exact(c, prepare(case, seed))
    if c["kind"] != "observables":
        return None  # an adaptive solve has no closed form, and a converged one takes minutes
    s = prepare(case, seed)
    k, y, par = s["k"], s["y"], s["param"]
    P = 2 * math.pi**2 * par["A_s"] * (k / par["k_p"]) ** (par["n_s"] - 1) * k**-3 * y[:, 4] ** 2
    amp = np.sqrt(2 * math.pi**2 * par["A_s"] * (k / par["k_p"]) ** (par["n_s"] - 1) * k**-3)
    wl = int(round(0.2 / (math.log(k[1]) - math.log(k[0]))))
    wl += (wl + 1) % 2
    x = np.arange(-(wl // 2), wl // 2 + 1, dtype=float)[::-1]
    coef = np.linalg.lstsq(x ** np.arange(4).reshape(-1, 1), np.array([1.0, 0, 0, 0]), rcond=None)[0]
    smooth = np.exp(np.convolve(np.log(P), coef, mode="same"))
    smooth[: wl // 2] = P[: wl // 2]
    smooth[-wl // 2:] = P[-wl // 2:]
    d, t, b = amp * y[:, 4], amp * y[:, 5], s["bias"]
    multi = (b**2 * d**2 - 2 * b / 3 * d * t + t**2 / 5, -4 * b / 3 * d * t + 4 / 7 * t**2, 8 / 35 * t**2)
    n = k.shape[0]
    ki = np.pi * np.arange(n // 2 + 1) / math.log(k[-1] / k[0])
    ph = _loggamma(torch.complex(torch.full((n // 2 + 1,), (1.5 + c["ell"]) / 2, dtype=torch.float64),
                                 torch.from_numpy(ki))).imag.numpy()
    f = np.fft.rfft(smooth * k**1.5) * np.exp(2j * (ph - math.log(math.pi) * ki))
    r = 2 * math.pi / k
    xi = np.real(1j ** c["ell"] * np.fft.irfft(f) / (2 * math.pi * r) ** 1.5)
    return smooth, multi, np.ascontiguousarray(xi[::-1]), np.ascontiguousarray(r[::-1])
