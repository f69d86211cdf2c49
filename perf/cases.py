"""Timed cases of the angular power spectrum path.

Each case is one call (or one short sequence of calls) that a program using this
package makes through its public entry points.  The kinds:

* ``cl``     ``angular_cl`` of one cosmology or a batch (device tensors);
* ``host``   ``angular_cl_host``: host parameters in, host C_ell out (CPU samplers);
* ``cov``    ``gaussian_cl_covariance_and_mean`` (dense is the default form);
* ``grad``   mean and covariance, log-likelihood and its gradient at one cosmology;
* ``vjp``    C_ell of a batch and the product of a cotangent with dC_ell/dtheta
             (the backward pass of a likelihood that the caller wrote);
* ``jac``    ``angular_cl_jacobian`` (Fisher forecasts);
* ``like``   batched ``gaussian_log_likelihood``, its gradient in the mean and the covariance;
* ``serve``  one sampler chain's log-likelihood + gradient request to the server;
* ``power``  ``nonlinear_matter_power`` at (k, a) points.

A survey is ``n_wl`` WeakLensing bins and ``n_nc`` NumberCounts bins, Smail n(z)
(a = 1, b = 2, z0 from 0.3 to 1.5) and ``n_ell`` log-spaced ell.  Cosmologies come
from the seeded box of the batched workload (``curved``: with Omega_k and wa too).

``exact`` restates the path in plain torch float64 (the grids, Simpson and
Romberg rules, RK4 steps and interpolation rule of jax_cosmo).
"""
import functools
import math

import numpy as np
import torch
import torch.autograd.forward_ad as fw

import jax_cosmo_gb300 as jc

NAMES = ("Omega_c", "Omega_b", "h", "n_s", "sigma8", "Omega_k", "w0", "wa")
BOX = {"Omega_c": (0.20, 0.35), "Omega_b": (0.04, 0.06), "h": (0.60, 0.80), "n_s": (0.90, 1.00),
       "sigma8": (0.60, 1.00), "w0": (-1.3, -0.7)}
CURVED = {"Omega_k": (-0.02, 0.02), "wa": (-0.3, 0.3)}
F_SKY, SIGMA_E, GALS = 0.25, 0.26, 10.0
F64 = torch.float64


def _case(kind, **kw):
    base = {"kind": kind, "n_cosmo": 1, "n_wl": 5, "n_nc": 0, "n_ell": 100, "ell_min": 20.0, "ell_max": 3000.0,
            "n_limber": 512, "zmax": 10.0, "precision": "fp64", "nonlinear": "takahashi2012",
            "transfer": "eisenhu_osc", "special_bias": False, "curved": False}
    base.update(kw)
    return base


def listed():
    """The configurations of the tests and the benchmark, small to large."""
    def one(name, kind, **kw):
        return dict(_case(kind, **kw), name=name)

    return [
        # a notebook plot: P(k) today at a few hundred wavenumbers of one cosmology
        one("power_curve", "power", n_points=256),
        # quick start: one cosmology, two lensing bins, the call of a plot or a by-hand minimiser
        one("quickstart_fp64", "cl", n_wl=2, n_ell=50, ell_min=10.0, n_limber=256, zmax=4.0),
        # one HMC chain of a 5-bin lensing survey waiting for its next gradient
        one("serve_one_fp32c", "serve", n_wl=5, n_ell=50, ell_min=10.0, precision="fp32c"),
        # README likelihood: mean and covariance at the cosmology, log-likelihood, gradient
        one("like_grad_fp64", "grad", n_wl=5, n_ell=50, ell_min=10.0),
        # ten-tracer data vector with its dense covariance (the default form)
        one("cov_10tracers_fp64", "cov", n_wl=5, n_nc=5, n_ell=200, ell_min=10.0, ell_max=5000.0),
        # Fisher forecast of the ten-tracer survey: the whole Jacobian
        one("jac_10tracers_fp64", "jac", n_wl=5, n_nc=5, n_ell=200, ell_min=10.0, ell_max=5000.0),
        # walkers of an ensemble sampler with the covariance of each: value and the
        # gradients that a parameter-dependent covariance needs, ten tracers
        one("like_batch", "like", n_cosmo=16, n_wl=5, n_nc=5, n_ell=200, ell_min=10.0, ell_max=5000.0),
        # gradients of a batch of chains with intrinsic alignment, evolving bias,
        # curvature and the smith2003 fit, default precision, odd sizes
        one("grad_options_fp64", "vjp", n_cosmo=61, n_wl=3, n_nc=2, n_ell=97, nonlinear="smith2003",
            special_bias=True, curved=True),
        # CPU sampler with host arrays, an odd batch
        one("host_batch_fp32c", "host", n_cosmo=2501, n_wl=5, n_ell=100, precision="fp32c"),
        # the batched workload (emulator training sets, importance sampling), FP32 compensated
        one("batch_fp32c", "cl", n_cosmo=4096, n_wl=5, n_ell=100, precision="fp32c"),
        # the same with the backward pass of a likelihood
        one("batch_grad_fp32c", "vjp", n_cosmo=4096, n_wl=5, n_ell=100, precision="fp32c"),
        # the same values in the default precision
        one("batch_fp64", "cl", n_cosmo=4096, n_wl=5, n_ell=100),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["cl", "cl", "cl", "host", "cov", "grad", "vjp", "vjp", "jac", "like", "serve", "power"])
    if kind == "power":
        return _case(kind, n_points=_log_int(rng, 1, 20000), n_cosmo=_log_int(rng, 1, 64),
                     curved=rng.random() < 0.5)
    n_wl, n_nc = rng.randint(1, 5), rng.randint(0, 5)
    if rng.random() < 0.15:
        n_wl, n_nc = 0, max(1, n_nc)
    n_ell = _log_int(rng, 20, 500)
    c = _case(kind, n_wl=n_wl, n_nc=n_nc, n_ell=n_ell, ell_min=rng.choice([10.0, 20.0, 30.0]),
              ell_max=rng.choice([2000.0, 3000.0, 5000.0]), n_limber=rng.choice([256, 512, 512, 512]),
              zmax=rng.choice([3.0, 4.0, 6.0, 10.0]))
    nodes = n_ell * (c["n_limber"] + 1)
    n_cls = (n_wl + n_nc) * (n_wl + n_nc + 1) // 2
    most = 150_000_000 // nodes  # cosmologies, so that a case costs less than the largest listed one
    if kind in ("cl", "host", "vjp", "jac"):
        c["precision"] = "fp32c" if kind == "host" else rng.choice(["fp64", "fp32c"])
        c["nonlinear"] = rng.choice(["takahashi2012", "takahashi2012", "smith2003", "linear"])
        c["transfer"] = rng.choice(["eisenhu_osc", "eisenhu_osc", "eisenhu_osc", "eisenhu"])
        c["special_bias"] = rng.random() < 0.4
        c["curved"] = rng.random() < 0.4
        if kind == "cl":
            c["n_cosmo"] = _log_int(rng, 1, min(4096, most))
        elif kind == "host":
            c["n_cosmo"] = _log_int(rng, 16, min(4096, most))
        elif kind == "vjp":
            c["n_cosmo"] = _log_int(rng, 1, min(4096 if c["precision"] == "fp32c" else 256, most // 8))
        else:
            c["n_cosmo"] = _log_int(rng, 1, max(1, min(64, most // 16, 20_000_000 // (n_cls * n_ell * 8))))
    elif kind == "serve":
        c["precision"] = "fp32c"
    elif kind == "cov":
        c["n_ell"] = min(n_ell, 11000 // n_cls)
    elif kind == "like":
        c["n_cosmo"] = _log_int(rng, 1, max(1, 10_000_000 // (n_cls * n_cls * n_ell)))
    return c


# ------------------------------------------------------------------ inputs --
def _cosmologies(case, seed):
    """[B, 8] float64 (host), uniform in the box."""
    rng = np.random.default_rng([20261204, seed])
    rows = np.zeros((case["n_cosmo"], 8))
    for i, n in enumerate(NAMES):
        lo_hi = BOX.get(n) or (CURVED.get(n) if case["curved"] else None)
        if lo_hi:
            rows[:, i] = rng.uniform(*lo_hi, case["n_cosmo"])
    return rows


def _z0(n):
    return np.linspace(0.3, 1.5, n) if n > 1 else np.array([0.7])


def _ell(case):
    return np.logspace(math.log10(case["ell_min"]), math.log10(case["ell_max"]), case["n_ell"])


def _probes(case):
    def bins(n):
        return [jc.redshift.smail_nz(1.0, 2.0, float(z), gals_per_arcmin2=GALS, zmax=case["zmax"]) for z in _z0(n)]

    out = []
    if case["n_wl"]:
        ia = jc.bias.des_y1_ia_bias(0.8, 1.3, 0.62) if case["special_bias"] else None
        out.append(jc.probes.WeakLensing(bins(case["n_wl"]), ia_bias=ia, sigma_e=SIGMA_E))
    if case["n_nc"]:
        b = jc.bias.inverse_growth_linear_bias(1.2) if case["special_bias"] else jc.bias.constant_linear_bias(1.2)
        out.append(jc.probes.NumberCounts(bins(case["n_nc"]), b))
    return out


def _operators(case):
    nl = (jc.power.linear_matter_power if case["nonlinear"] == "linear"
          else functools.partial(jc.power.halofit, prescription=case["nonlinear"]))
    return {"transfer_fn": functools.partial(jc.transfer.Eisenstein_Hu, type=case["transfer"]), "nonlinear_fn": nl}


def _cosmo(rows, device="cuda", grad=False):
    """One row: a Cosmology of numbers (or leaf tensors); more: of length-B tensors."""
    if grad:
        leaves = [torch.tensor(rows[0, i] if len(rows) == 1 else rows[:, i], dtype=F64, device=device,
                               requires_grad=True) for i in range(8)]
        return jc.Cosmology(*leaves), leaves
    if len(rows) == 1:
        return jc.Cosmology(*[float(v) for v in rows[0]]), None
    return jc.Cosmology(*[torch.tensor(rows[:, i], dtype=F64, device=device) for i in range(8)]), None


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) + 77)


def _points(case, seed):
    """k log-spaced over the range of a P(k) plot, a today (odd seeds of a batch: earlier)."""
    rng = np.random.default_rng([7, seed])
    k = np.logspace(-4, 1, case["n_points"]) * rng.uniform(0.9, 1.1)
    a = np.ones(case["n_points"]) if case["n_points"] <= 512 else rng.uniform(0.25, 1.0, case["n_points"])
    return torch.tensor(k, dtype=F64, device="cuda"), torch.tensor(a, dtype=F64, device="cuda")


def _like_inputs(case, seed):
    """(data [N], mean [B, N], covariance [B, n_cls, n_cls, n_ell]) with spectra of the
    size and shape of a lensing survey's, their own Gaussian covariance."""
    g = _generator(seed)
    B, n = case["n_cosmo"], case["n_wl"] + case["n_nc"]
    ell = torch.tensor(_ell(case), dtype=F64, device="cuda")
    u = lambda *s: torch.rand(*s, dtype=F64, device="cuda", generator=g)  # noqa: E731
    amp = 1e-4 * (1.0 + u(B, n))
    tilt = (ell / 100.0) ** (-1.1)
    dist = torch.arange(n, dtype=F64, device="cuda")
    corr = torch.exp(-0.3 * (dist[:, None] - dist[None, :]).abs())
    i, j = _pairs(n)
    cl = (amp[:, i] * amp[:, j] * corr[i, j])[:, :, None] * tilt * (1.0 + 0.05 * u(B, len(i), 1))
    cov = _knox(cl, _noise(case).to(cl.device), _ell(case), n)
    mean = cl.reshape(B, -1)
    sig = torch.diagonal(cov[0], dim1=0, dim2=1).T.reshape(-1).sqrt()
    data = mean[0] + sig * torch.randn(sig.shape, dtype=F64, device="cuda", generator=g)
    return data, mean, cov


def prepare(case, seed):
    kind = case["kind"]
    st = {"kind": kind, "case": case}
    if kind == "like":
        data, mean, cov = _like_inputs(case, seed)
        st.update(data=data, mean=mean.requires_grad_(True), cov=cov.requires_grad_(True))
        return st
    rows = _cosmologies(case, seed)
    st.update(ops=_operators(case))
    if kind == "power":
        st["k"], st["a"] = _points(case, seed)
        st["cosmo"], _ = _cosmo(rows)
        return st
    st.update(ell=_ell(case), probes=_probes(case))
    if kind == "host":
        st["params"] = torch.tensor(rows, dtype=F64).pin_memory()
        n_tr = case["n_wl"] + case["n_nc"]
        st["out"] = torch.empty(len(rows), n_tr * (n_tr + 1) // 2, case["n_ell"], dtype=F64).pin_memory()
        st["physics"] = jc.cl.physics_code(**st["ops"])
        return st
    st["cosmo"], st["leaves"] = _cosmo(rows, grad=kind in ("grad", "vjp"))
    g = _generator(seed)
    if kind == "vjp":
        n_tr = case["n_wl"] + case["n_nc"]
        # a likelihood's cotangent: residuals of either sign over the variance,
        # the same order of magnitude for every spectrum times C_ell
        st["cl_bar"] = torch.randn(len(rows), n_tr * (n_tr + 1) // 2, case["n_ell"], dtype=F64, device="cuda",
                                   generator=g) * torch.tensor(st["ell"], device="cuda") * 1e6
    if kind in ("grad", "serve"):
        mean, cov = jc.cl.gaussian_cl_covariance_and_mean(jc.Planck15(), st["ell"], st["probes"], f_sky=F_SKY,
                                                          sparse=True, n_limber=case["n_limber"])
        z = torch.randn(mean.shape, dtype=F64, device="cuda", generator=g)
        st["data"] = mean + z * torch.diagonal(cov, dim1=0, dim2=1).T.reshape(-1).sqrt()
        if kind == "serve":
            st["chain"] = _Chain(jc, st["probes"], st["ell"], st["data"], cov, case)
            st["params"] = rows[0]
    return st


class _Chain:
    """A server with one chain's model; stopped when the state goes."""

    def __init__(self, pkg, probes, ell, data, cov, case):
        from jax_cosmo_gb300 import serving

        self.model = serving.ChainModel(probes, ell, data, cov, n_limber=case["n_limber"])
        self.server = serving.Server(hbm_budget=1 << 28, precision=case["precision"]).start()

    def __del__(self):
        if hasattr(self, "server"):
            self.server.stop()


def run(state):
    c, kind = state["case"], state["kind"]
    if kind == "like":
        ll = jc.likelihood.gaussian_log_likelihood(state["data"], state["mean"], state["cov"])
        dmu, dcov = torch.autograd.grad(ll.sum(), [state["mean"], state["cov"]])
        return {"loglike": ll.detach(), "dmean": dmu, "dcov": dcov}
    if kind == "power":
        return jc.power.nonlinear_matter_power(state["cosmo"], state["k"], state["a"])
    if kind == "host":
        out = jc.cl.angular_cl_host(state["params"], state["ell"], state["probes"], precision=c["precision"],
                                    n_limber=c["n_limber"], out=state["out"], physics=state["physics"])
        return out
    if kind == "serve":
        r = state["chain"].server.submit(state["chain"].model, state["params"]).result()
        return {"loglike": r.loglike, "grad": r.grad}
    opt = dict(state["ops"], precision=c["precision"], n_limber=c["n_limber"])
    if kind == "cl":
        return jc.cl.angular_cl(state["cosmo"], state["ell"], state["probes"], **opt)
    if kind == "cov":
        mean, cov = jc.cl.gaussian_cl_covariance_and_mean(state["cosmo"], state["ell"], state["probes"], f_sky=F_SKY,
                                                          **opt)
        return {"mean": mean, "cov": cov}
    if kind == "jac":
        cl, jac = jc.autodiff.angular_cl_jacobian(state["cosmo"], state["ell"], state["probes"], **opt)
        return {"cl": cl, "jac": jac}
    if kind == "vjp":
        cl = jc.cl.angular_cl(state["cosmo"], state["ell"], state["probes"], **opt)
        bar = state["cl_bar"] if cl.dim() == 3 else state["cl_bar"][0]
        return {"cl": cl.detach(), "grad": list(torch.autograd.grad(cl, state["leaves"], bar))}
    mean, cov = jc.cl.gaussian_cl_covariance_and_mean(state["cosmo"], state["ell"], state["probes"], f_sky=F_SKY,
                                                      sparse=True, **opt)
    ll = jc.likelihood.gaussian_log_likelihood(state["data"], mean, cov)
    return {"loglike": ll.detach(), "grad": list(torch.autograd.grad(ll, state["leaves"]))}


def work(case):
    """Bytes: inputs and outputs once.  Operations: about 150 for P(k, a) at a
    node with each function counted as one, two per spectrum and node for the
    sum; the lensing integrals (257 points, 10 each), the halofit moments (257
    nodes, 8 each); a gradient three times its value, a Jacobian row 8 more."""
    B = case["n_cosmo"]
    if case["kind"] == "power":
        n = case["n_points"]
        return {"bytes": 8.0 * (8 * B + 2 * n + B * n), "flops": 150.0 * B * n + B * 256 * 257 * 4.0}
    n_tr, n_ell, na = case["n_wl"] + case["n_nc"], case["n_ell"], case["n_limber"] + 1
    n_cls = n_tr * (n_tr + 1) // 2
    if case["kind"] == "like":
        return {"bytes": 8.0 * B * n_ell * (2 * n_cls * n_cls + 3.0 * n_cls), "flops": B * n_ell * 2.0 * n_cls**3}
    flops = B * na * (n_ell * (150.0 + 2 * n_cls) + case["n_wl"] * 257 * 10.0 + 257 * 8.0) + B * 256 * 257 * 4.0
    out = 8.0 * B * (8 + n_cls * n_ell)
    if case["kind"] == "cov":
        out += 8.0 * (n_cls * n_ell) ** 2
    elif case["kind"] == "jac":
        flops, out = 3 * flops + B * na * n_ell * n_cls * 16.0, out * 9
    elif case["kind"] in ("vjp", "grad", "serve"):
        flops, out = 3 * flops, out + 8.0 * B * (8 + n_cls * n_ell)
    return {"bytes": out, "flops": flops}


# ------------------------------------------ the same results in plain torch --
C_KMS, RH, T27 = 299792.458, 2997.92458, (2.726 / 2.7) ** 2
E1 = math.exp(1.0)


@functools.lru_cache(maxsize=None)
def _pair_lists(n):
    return [i for i in range(n) for _ in range(i, n)], [j for i in range(n) for j in range(i, n)]


def _pairs(n):
    i, j = _pair_lists(n)
    return torch.tensor(i, device="cuda"), torch.tensor(j, device="cuda")


def _noise(case):
    per = GALS * 11818102.86004228
    return torch.tensor([SIGMA_E**2 / per] * case["n_wl"] + [1.0 / per] * case["n_nc"], dtype=F64)


def _knox(cl, noise, ell, n):
    """[B, n_cls, n_cls, n_ell] Gaussian covariance of [B, n_cls, n_ell] spectra."""
    i, j = _pairs(n)
    pos = torch.zeros(n, n, dtype=torch.long, device=cl.device)
    pos[i, j] = torch.arange(len(i), device=cl.device)
    pos[j, i] = pos[i, j]
    obs = cl + torch.where(i == j, noise[i], 0.0 * noise[i])[:, None]
    norm = torch.tensor((2 * ell + 1) * np.gradient(ell) * F_SKY, dtype=F64, device=cl.device)
    im, jn = pos[i[:, None], i[None, :]], pos[j[:, None], j[None, :]]
    in_, jm = pos[i[:, None], j[None, :]], pos[j[:, None], i[None, :]]
    return (obs[:, im] * obs[:, jn] + obs[:, in_] * obs[:, jm]) / norm


def _t(x):
    return torch.tensor(np.asarray(x), dtype=F64, device="cuda")


def _simpson_w(n, dx):
    w = np.ones(n + 1)
    w[1:-1:2], w[2:-1:2] = 4.0, 2.0
    return _t(w) * dx / 3.0


def _segment(x, xp):
    """(i, j) of jax_cosmo's interp on an increasing grid: the nearest node, and the
    neighbour on the side of x."""
    n = len(xp)
    hi = torch.searchsorted(xp, x.contiguous()).clamp(1, n - 1)
    i = torch.where((x - xp[hi - 1]) ** 2 <= (xp[hi] - x) ** 2, hi - 1, hi).clamp(1, n - 2)
    side = x.clamp(float(xp[1]), float(xp[n - 2])) - xp[i]
    return i, torch.where(side >= 0, i + 1, i - 1)


def _interp(x, xp, fp):
    """x any shape (shared), fp [B, n] -> [B, *x.shape]."""
    i, j = _segment(x, xp)
    a = (fp[:, j] - fp[:, i]) / (xp[j] - xp[i])
    return a * x + (fp[:, i] - a * xp[i])


class _Model:
    """Tables of a batch of cosmologies; p is a list of 8 tensors [B, 1]."""

    def __init__(self, p, transfer="eisenhu_osc"):
        self.Oc, self.Ob, self.h, self.ns, self.s8, self.Ok, self.w0, self.wa = p
        self.transfer = transfer
        self.Om = self.Oc + self.Ob
        self.Ode = 1.0 - self.Ok - self.Om
        self._background()
        self._eh_scalars()
        logk = np.linspace(math.log(1e-4), math.log(1e4), 257)
        self.kh, self.wk = torch.exp(_t(logk)), _simpson_w(256, (math.log(1e4) - math.log(1e-4)) / 256)
        self._norm()
        self.pk3 = self.plin(self.kh) * self.kh**3
        self.logr = _t(np.linspace(math.log(1e-4), math.log(1e1), 256))
        self.sig = (self.pk3 * self.wk / (2 * math.pi**2)) @ torch.exp(-(torch.outer(self.kh, self.logr.exp()) ** 2))

    # background (E^2, chi and growth tables)
    def efde(self, a):
        return torch.exp(-3.0 * (1.0 + self.w0 + self.wa) * torch.log(a) + 3.0 * self.wa * (a - 1.0))

    def e2(self, a):
        return self.Om / a**3 + self.Ok / a**2 + self.Ode * self.efde(a)

    def om(self, a):
        return self.Om / a**3 / self.e2(a)

    def ode(self, a):
        return self.Ode * self.efde(a) / self.e2(a)

    def w(self, a):
        return self.w0 + (1.0 - a) * self.wa

    def dchi(self, a):
        return RH / (a**2 * torch.sqrt(self.e2(a)))

    def _background(self):
        at = np.logspace(-3.0, 0.0, 256)
        self.achi, x = _t(at), _t(np.log(at))
        f = lambda t: self.dchi(torch.exp(t)) * torch.exp(t)  # noqa: E731
        h = x[1:] - x[:-1]
        fn, fm = f(x), f(x[:-1] + h / 2)
        inc = h / 6.0 * (fn[:, :-1] + 4.0 * fm + fn[:, 1:])
        y = torch.cat([torch.zeros_like(inc[:, :1]), torch.cumsum(inc, dim=1)], dim=1)
        self.chitab = y[:, -1:] - y
        self.agr = g = _t(np.logspace(-3.0, 0.0, 128))
        hm = g[1:] - g[:-1]

        def qr(a):
            om, de = self.om(a), self.ode(a)
            return (2.0 - 0.5 * (om + (1.0 + 3.0 * self.w(a)) * de)) / a, 1.5 * om / a / a

        (q0, r0), (qm, rm) = qr(g), qr(g[:-1] + hm / 2)
        y0, y1 = g[:1].expand(q0.shape[0]), torch.ones_like(q0[:, 0])
        out = [y0]
        for s in range(127):
            d, qa, ra, qb, rb, qc, rc = hm[s], q0[:, s], r0[:, s], qm[:, s], rm[:, s], q0[:, s + 1], r0[:, s + 1]
            k1, l1 = y1, -qa * y1 + ra * y0
            a2, b2 = y0 + d * k1 / 2, y1 + d * l1 / 2
            k2, l2 = b2, -qb * b2 + rb * a2
            a3, b3 = y0 + d * k2 / 2, y1 + d * l2 / 2
            k3, l3 = b3, -qb * b3 + rb * a3
            a4, b4 = y0 + d * k3, y1 + d * l3
            k4, l4 = b4, -qc * b4 + rc * a4
            y0 = y0 + d / 6.0 * (k1 + 2 * k2 + 2 * k3 + k4)
            y1 = y1 + d / 6.0 * (l1 + 2 * l2 + 2 * l3 + l4)
            out.append(y0)
        gt = torch.stack(out, dim=1)
        self.gtab = gt / gt[:, -1:]

    def chi(self, a):
        return _interp(a, self.achi, self.chitab).clamp(min=0.0)

    def growth(self, a):
        return _interp(a, self.agr, self.gtab).clamp(0.0, 1.0)

    # Eisenstein & Hu (1998)
    def _eh_scalars(self):
        wm, wb = self.Om * self.h**2, self.Ob * self.h**2
        fb, fc = self.Ob / self.Om, (self.Om - self.Ob) / self.Om
        keq, zeq = 7.46e-2 * wm / T27 / self.h, 2.50e4 * wm / T27**2
        b1, b2 = 0.313 * wm**-0.419 * (1.0 + 0.607 * wm**0.674), 0.238 * wm**0.223
        zd = 1291.0 * wm**0.251 / (1.0 + 0.659 * wm**0.828) * (1.0 + b1 * wb**b2)
        Rd, Req = 31.5 * wb / T27**2 * (1e3 / zd), 31.5 * wb / T27**2 * (1e3 / zeq)
        sh = 2.0 / (3.0 * keq) * torch.sqrt(6.0 / Req) * torch.log(
            (torch.sqrt(1.0 + Rd) + torch.sqrt(Req + Rd)) / (1.0 + torch.sqrt(Req)))
        ks = 1.6 * wb**0.52 * wm**0.73 * (1.0 + (10.4 * wm) ** -0.95) / self.h
        a1 = (46.9 * wm) ** 0.670 * (1.0 + (32.1 * wm) ** -0.532)
        a2 = (12.0 * wm) ** 0.424 * (1.0 + (45.0 * wm) ** -0.582)
        ac = a1 ** (-fb) * a2 ** (-(fb**3))
        bb1, bb2 = 0.944 / (1.0 + (458.0 * wm) ** -0.708), (0.395 * wm) ** -0.0266
        bc = 1.0 / (1.0 + bb1 * (fc**bb2 - 1.0))
        y = (1.0 + zeq) / (1.0 + zd)
        x = torch.sqrt(1.0 + y)
        G = y * (-6.0 * x + (2.0 + 3.0 * y) * torch.log((x + 1.0) / (x - 1.0)))
        ab = 2.07 * keq * sh * (1.0 + Rd) ** -0.75 * G
        bn = 8.41 * wm**0.435
        bb = 0.5 + fb + (3.0 - 2.0 * fb) * torch.sqrt((17.2 * wm) ** 2 + 1.0)
        ag = 1.0 - 0.328 * torch.log(431.0 * wm) * wb / wm + 0.38 * torch.log(22.3 * wm) * fb**2
        self.eh = [keq, sh, ks, ac, bc, ab, bn, bb, fb, fc, ag]

    def T(self, k):
        """k [n] or [B, n_ell, n_a]"""
        keq, sh, ks, ac, bc, ab, bn, bb, fb, fc, ag = [v if k.dim() < 3 else v[..., None] for v in self.eh]
        if self.transfer == "eisenhu":
            Omh = self.Om * self.h
            Omh = Omh if k.dim() < 3 else Omh[..., None]
            q = k * T27 / (Omh * (ag + (1.0 - ag) / (1.0 + (0.43 * k * sh) ** 4)))
            L = torch.log(2.0 * E1 + 1.8 * q)
            return L / (L + (14.2 + 731.0 / (1.0 + 62.5 * q)) * q * q)
        q = k / (13.41 * keq)
        C0 = 386.0 / (1.0 + 69.9 * q**1.08)
        L1, L2 = torch.log(E1 + 1.8 * bc * q), torch.log(E1 + 1.8 * q)
        f = 1.0 / (1.0 + (k * sh / 5.4) ** 4)
        Tc = f * L1 / (L1 + (14.2 + C0) * q * q) + (1.0 - f) * L1 / (L1 + (14.2 / ac + C0) * q * q)
        st = sh * (1.0 + (bn / (k * sh)) ** 3) ** (-1.0 / 3.0)
        Tb = (L2 / (L2 + (14.2 + C0) * q * q) / (1.0 + (k * sh / 5.2) ** 2)
              + ab / (1.0 + (bb / (k * sh)) ** 3) * torch.exp(-((k / ks) ** 1.4))) * torch.sin(k * st) / (k * st)
        return fb * Tb + fc * Tc

    def _norm(self):
        """sigma^2(8): 7 levels of Romberg over ln k in [-4, 3]."""
        def f(x):
            k = torch.exp(x)
            u = 8.0 * k
            W = 3.0 * (torch.sin(u) - u * torch.cos(u)) / u**3
            return k * (k * W) ** 2 * self.T(k) ** 2 * k**self.ns

        a, b = -4.0, 3.0
        s = 0.5 * f(_t([a, b])).sum(1, keepdim=True)
        row = [(b - a) * s] * 8
        for i in range(1, 8):
            m = 2 ** (i - 1)
            h = (b - a) / m
            s = s + f(_t(a + 0.5 * h + h * np.arange(m))).sum(1, keepdim=True)
            new = [(b - a) * s / 2**i]
            for q in range(7):
                new.append((4.0 ** (q + 1) * new[q] - row[q]) / (4.0 ** (q + 1) - 1.0))
            row = new
        self.norm = self.s8**2 / (row[7] / (2 * math.pi**2))

    def plin(self, k):
        """Linear power today."""
        ns, norm = (self.ns, self.norm) if k.dim() < 3 else (self.ns[..., None], self.norm[..., None])
        return norm * k**ns * self.T(k) ** 2

    def halofit_scale(self, a):
        """(k_nl, n_eff, C), [B, na] each."""
        g2 = self.growth(a) ** 2
        sig = self.sig[:, None, :] * g2[:, :, None]
        d = sig.detach()
        i = ((1.0 - d) ** 2).argmin(dim=-1, keepdim=True).clamp(1, 254)
        one = torch.ones_like(d[..., :1])
        x = torch.minimum(torch.maximum(one, d[..., 1:2]), d[..., 254:255])
        j = torch.where(x - d.gather(-1, i) >= 0, i + 1, i - 1)
        si, sj = sig.gather(-1, i), sig.gather(-1, j)
        s = (self.logr[j] - self.logr[i]) / (sj - si)
        R = torch.exp(s + (self.logr[i] - s * si))[..., 0].clamp(min=1e-6)
        y2 = (R[:, :, None] * self.kh) ** 2
        e = (self.pk3 * self.wk / (2 * math.pi**2))[:, None, :] * torch.exp(-y2) * g2[:, :, None]
        dn = (2.0 * e * y2).sum(-1)
        return 1.0 / R, dn - 3.0, dn**2 + (4.0 * e * (y2 - y2 * y2)).sum(-1)

    def pnl(self, k, a, nonlinear):
        """k [B, n_ell, na] at a [na]."""
        g = self.growth(a)
        p = self.plin(k) * (g**2)[:, None, :]
        if nonlinear == "linear":
            return p
        kn, n, C = self.halofit_scale(a)
        om, de, w = self.om(a), self.ode(a), self.w(a)
        if nonlinear == "smith2003":
            an = 10 ** (1.4861 + 1.8369 * n + 1.6762 * n**2 + 0.7940 * n**3 + 0.1670 * n**4 - 0.6206 * C)
            bn = 10 ** (0.9463 + 0.9466 * n + 0.3084 * n**2 - 0.9400 * C)
            cn = 10 ** (-0.2807 + 0.6669 * n + 0.3214 * n**2 - 0.0793 * C)
            ga = 0.8649 + 0.2989 * n + 0.1631 * C
            al = 1.3884 + 0.3700 * n - 0.1452 * n**2
            be = 0.8291 + 0.9854 * n + 0.3401 * n**2
            mu, nu = 10 ** (-3.5442 + 0.1908 * n), 10 ** (0.9585 + 1.2857 * n)
            fr = de / (1.0 - om)
            f1 = fr * om**-0.0307 + (1 - fr) * om**-0.0732
            f2 = fr * om**-0.0585 + (1 - fr) * om**-0.1423
            f3 = fr * om**0.0743 + (1 - fr) * om**0.0725
        else:
            an = 10 ** (1.5222 + 2.8553 * n + 2.3706 * n**2 + 0.9903 * n**3 + 0.2250 * n**4 - 0.6038 * C
                        + 0.1749 * de * (1 + w))
            bn = 10 ** (-0.5642 + 0.5864 * n + 0.5716 * n**2 - 1.5474 * C + 0.2279 * de * (1 + w))
            cn = 10 ** (0.3698 + 2.0404 * n + 0.8161 * n**2 + 0.5869 * C)
            ga = 0.1971 - 0.0843 * n + 0.8460 * C
            al = (6.0835 + 1.3373 * n - 0.1959 * n**2 - 5.5274 * C).abs()
            be = 2.0379 - 0.7354 * n + 0.3157 * n**2 + 1.2490 * n**3 + 0.3980 * n**4 - 0.1682 * C
            mu, nu = 0.0 * n, 10 ** (5.2105 + 3.6902 * n)
            f1, f2, f3 = om**-0.0307, om**-0.0585, om**0.0743
        kn, an, bn, cn, ga, al, be, mu, nu, f1, f2, f3 = [v[:, None, :] for v in
                                                         (kn, an, bn, cn, ga, al, be, mu, nu, f1, f2, f3)]
        d2l = k**3 * p / (2 * math.pi**2)
        y = k / kn
        d2q = d2l * (1.0 + d2l) ** be / (1.0 + al * d2l) * torch.exp(-(y / 4.0 + y**2 / 8.0))
        d2h = an * y ** (3.0 * f1) / (1.0 + bn * y**f2 + (cn * f3 * y) ** (3.0 - ga)) / (1.0 + mu / y + nu / y**2)
        return 2 * math.pi**2 / k**3 * (d2q + d2h)

    # tracers
    def _nz(self, z0, zmax, z):
        f = lambda x: x * torch.exp(-((x / z0) ** 2))  # noqa: E731
        return f(z) / (f(_t(np.linspace(0.0, zmax, 257))) * _simpson_w(256, zmax / 256)).sum()

    def kernels(self, case, a):
        """[B, n_tr, na] without the lensing ell factor."""
        z, zmax = 1.0 / a - 1.0, case["zmax"]
        zs = np.asarray(z.cpu())
        out, H = [], 100.0 * torch.sqrt(self.e2(a))
        if case["n_wl"]:
            zp = _t(np.linspace(zs, zmax, 257))  # [257, na]
            chi, chip = self.chi(a), self.chi(1.0 / (1.0 + zp))
            ratio = (chip - chi[:, None, :]).clamp(min=0.0) / chip.clamp(min=1.0)
            w = _simpson_w(256, 1.0)[:, None] * (zmax - z) / 256
            for z0 in _z0(case["n_wl"]):
                k = (ratio * (self._nz(z0, zmax, zp) * w)).sum(1) * (1.0 + z) * chi * 1.5 * 1e4 * self.Om / C_KMS
                if case["special_bias"]:
                    b = 0.8 * ((1.0 + z) / 1.62) ** 1.3
                    k = k + self._nz(z0, zmax, z) * b * H * (-(5e-14 * 2.7750e11) * self.Om / self.growth(a))
                out.append(k)
        for z0 in _z0(case["n_nc"]) if case["n_nc"] else ():
            b = 1.2 / self.growth(a) if case["special_bias"] else 1.2
            out.append(self._nz(z0, zmax, z) * b * H)
        return torch.stack(out, dim=1)


def _theory(p, case):
    """C_ell [B, n_cls, n_ell] of parameter columns p (8 tensors [B, 1])."""
    m = _Model(p, case["transfer"])
    ell, N, zmax = _t(_ell(case)), case["n_limber"], case["zmax"]
    a0 = 1.0 / (1.0 + zmax)
    a = _t(np.linspace(a0, 1.0, N + 1))
    chi = m.chi(a)
    k = (ell[:, None] + 0.5) / chi.clamp(min=1.0)[:, None, :]
    u = _simpson_w(N, (1.0 - a0) / N) * m.dchi(a) / (chi**2).clamp(min=1.0) / C_KMS**2
    K = m.kernels(case, a)
    i, j = _pairs(K.shape[1])
    M = K[:, i] * K[:, j] * u[:, None, :]
    cl = torch.bmm(M, m.pnl(k, a, case["nonlinear"]).transpose(1, 2))
    ef = torch.sqrt((ell - 1) * ell * (ell + 1) * (ell + 2)) / (ell + 0.5) ** 2
    n_wl_in_pair = (i < case["n_wl"]).to(F64) + (j < case["n_wl"]).to(F64)
    return cl * ef ** n_wl_in_pair[:, None]


def _columns(rows):
    return [_t(rows[:, i : i + 1]) for i in range(8)]


def _chunks(case, nodes):
    step = max(1, nodes // (case["n_ell"] * (case["n_limber"] + 1)))
    return [slice(s, s + step) for s in range(0, case["n_cosmo"], step)]


def _loglike(data, mean, cov, logdet=True):
    """[B] of mean [B, N], covariance [B, n_cls, n_cls, n_ell]; the reference's sign of the log-determinant."""
    B, n, _, nl = cov.shape
    r = (mean - data).reshape(B, n, nl).permute(0, 2, 1)[..., None]
    blocks = cov.permute(0, 3, 1, 2)
    q = (r * torch.linalg.solve(blocks, r)).sum((1, 2, 3))
    return -0.5 * (q - torch.linalg.slogdet(blocks)[1].sum(-1)) if logdet else -0.5 * q


def _fiducial_data(case, seed, noise=True):
    """(data, covariance) that ``prepare`` makes for the likelihood kinds."""
    cl = _theory(_columns(np.array([[0.2589, 0.04860, 0.6774, 0.9667, 0.8159, 0.0, -1.0, 0.0]])),
                 dict(case, nonlinear="takahashi2012", transfer="eisenhu_osc"))
    cov = _knox(cl, _noise(case).cuda(), _ell(case), case["n_wl"] + case["n_nc"])[0]
    mean = cl.reshape(-1)
    z = torch.randn(mean.shape, dtype=F64, device="cuda", generator=_generator(seed))
    return mean + z * torch.diagonal(cov, dim1=0, dim2=1).T.reshape(-1).sqrt(), cov


def exact(case, seed):
    kind = case["kind"]
    if kind == "like":
        data, mean, cov = _like_inputs(case, seed)
        ll = _loglike(data, mean.requires_grad_(True), cov.requires_grad_(True))
        dmean, dcov = torch.autograd.grad(ll.sum(), [mean, cov])
        return {"loglike": ll.detach(), "dmean": dmean, "dcov": dcov}
    rows = _cosmologies(case, seed)
    n_tr = case["n_wl"] + case["n_nc"]
    if kind == "power":
        k, a = _points(case, seed)
        out, m = [], _Model(_columns(rows))
        for s in range(0, len(k), 256):  # one k for each a
            ks = k[None, None, s : s + 256].expand(len(rows), 1, -1)
            out.append(m.pnl(ks, a[s : s + 256], case["nonlinear"])[:, 0])
        out = torch.cat(out, dim=1)
        return out[0] if len(rows) == 1 else out
    if kind in ("cl", "host", "cov"):
        cl = torch.cat([_theory(_columns(rows[s]), case) for s in _chunks(case, 1 << 22)])
        if kind == "cov":
            cov = _knox(cl, _noise(case).cuda(), _ell(case), n_tr)[0]
            n, nl = cov.shape[0], cov.shape[2]
            dense = torch.zeros(n, nl, n, nl, dtype=F64, device="cuda")
            d = torch.arange(nl, device="cuda")
            dense[:, d, :, d] = cov.permute(2, 0, 1)
            return {"mean": cl.reshape(-1), "cov": dense.reshape(n * nl, n * nl)}
        return cl.cpu() if kind == "host" else cl[0] if len(rows) == 1 else cl
    if kind == "jac":
        cls, jacs = [], []
        for s in _chunks(case, 1 << 21):
            p = _columns(rows[s])
            cols = []
            for d in range(8):
                with fw.dual_level():
                    dual = _theory([fw.make_dual(v, torch.full_like(v, float(q == d))) for q, v in enumerate(p)], case)
                    cl, t = fw.unpack_dual(dual)
                    cols.append(t.clone())
                    cl = cl.clone()
            cls.append(cl)
            jacs.append(torch.stack(cols, dim=-1))
        cl, jac = torch.cat(cls), torch.cat(jacs)
        return {"cl": cl[0], "jac": jac[0]} if len(rows) == 1 else {"cl": cl, "jac": jac}
    if kind == "vjp":
        bar = torch.randn(len(rows), n_tr * (n_tr + 1) // 2, case["n_ell"], dtype=F64, device="cuda",
                          generator=_generator(seed)) * _t(_ell(case)) * 1e6
        cls, grads = [], []
        for s in _chunks(case, 1 << 21):
            p = [v.requires_grad_(True) for v in _columns(rows[s])]
            cl = _theory(p, case)
            grads.append(torch.cat(torch.autograd.grad(cl, p, bar[s]), dim=1))
            cls.append(cl.detach())
        cl, grad = torch.cat(cls), torch.cat(grads)
        one = len(rows) == 1
        return {"cl": cl[0] if one else cl, "grad": [grad[0, i] if one else grad[:, i] for i in range(8)]}
    data, cov = _fiducial_data(case, seed)
    p = [v.requires_grad_(True) for v in _columns(rows)]
    cl = _theory(p, case)
    if kind == "grad":
        cov = _knox(cl, _noise(case).cuda(), _ell(case), n_tr)[0]
    ll = _loglike(data, cl.reshape(1, -1), cov[None], logdet=kind == "grad")[0]
    grad = [g.reshape(()) for g in torch.autograd.grad(ll, p)]
    if kind == "serve":
        return {"loglike": float(ll), "grad": np.array([float(g) for g in grad])}
    return {"loglike": ll.detach(), "grad": grad}
