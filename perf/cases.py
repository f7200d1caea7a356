"""Workloads of this package that its performance is measured on.

Each case is one call of the package's public Python interface (the mirror of the
reference API over the C ABI), at a size that its users run:

  xsec      compute_voigt_cross_sections on a caller's grid
  forward   forward_model_batch (and VP_Y line mixing), double and mixed precision
  jacobian  analytic_jacobian_batch
  vjp       vjp_batch, the reverse-mode pullback
  oe        optimal_estimation_batch, a whole retrieval
  infer     Surrogate.predict_device on tensors that stay on the GPU
  train     Surrogate.gradients, one training batch's loss and gradient

listed() names the measured cases, draw() gives more of the same ranges, prepare()
makes what a program holds before the call, run() is the call, work() its necessary
bytes and operations, and exact() the same result in 64-bit arithmetic written here
in plain torch, apart from the package's own code.

The line lists are the spectroscopic database: one seeded list per size and range,
the same for every seed and uploaded once, as a program loads HITRAN once.  A seed
changes what changes from call to call: profiles, angles, surface, layer states,
observations, batches.

Spectra of the mixed-precision path, Jacobians (stored in single precision on the
device) and what a retrieval makes of them carry single precision, and are kept in it.
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
PACKAGE = ROOT / "irsounderlbl.jl_b200"


def _package():
    if "irs_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("irs_b200", PACKAGE / "__init__.py",
                                                      submodule_search_locations=[str(PACKAGE)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["irs_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["irs_b200"]


# ------------------------------------------------------------------ the cases
def _forward(name, **kw):
    c = dict(kind="forward", name=name, nu_lo=645.0, nu_hi=700.0, dnu=0.25, opd=2.0, fwhm=0.5, internal_dnu=0.0025,
             species=1, lines=5000, profiles=1, precision="mixed", mixing=False, eps=1.0, source="cim",
             apodization="gaussian")
    c.update(kw)
    return c


def listed():
    return [
        # one layer's cross sections on a coarse window: the smallest call, interactive use
        dict(kind="xsec", name="xsec_small", nu_lo=645.0, nu_hi=700.0, points=5501, lines=5000, precision="fp64",
             method=3),
        # one species over the whole IASI range at the internal grid, default precision
        dict(kind="xsec", name="xsec_iasi_fp64", nu_lo=645.0, nu_hi=2760.0, points=846001, lines=66667,
             precision="fp64", method=3),
        # forward_model with its default (double) precision: the CO2 band on the 5,000-line list
        _forward("forward_band_fp64", precision="fp64"),
        # double precision over two more species and a short-wave window, grey surface, Toon source
        _forward("forward_mix3_fp64", nu_lo=1210.0, nu_hi=1290.0, species=3, lines=9000, precision="fp64", eps=0.97,
                 source="toon"),
        # a single scene in mixed precision: latency of an interactive or per-scene call
        _forward("forward_scene", lines=5000),
        # the headline: 400,000 lines, IASI, the six AFGL-like profiles in mixed precision
        _forward("forward_iasi", nu_hi=2760.0, species=6, lines=400000, profiles=6),
        # CrIS long-wave band with first-order line mixing on CO2, grey surface
        _forward("forward_cris_vpy", nu_lo=650.0, nu_hi=1095.0, dnu=0.625, opd=0.8, fwhm=0.0, species=6, lines=30000,
                 profiles=2, mixing=True, eps=0.98),
        # the retrieval's inner step: Jacobians of a batch of scenes on the 5,000-line list
        dict(kind="jacobian", name="jacobian_scenes", nu_lo=645.0, nu_hi=700.0, dnu=0.25, opd=2.0, fwhm=0.5,
             internal_dnu=0.0025, species=1, lines=5000, profiles=16, retrieved=1, mixing=False, eps=1.0),
        # one full IASI Jacobian, 400,000 lines with VP_Y, 151-element state
        dict(kind="jacobian", name="jacobian_iasi", nu_lo=645.0, nu_hi=2760.0, dnu=0.25, opd=2.0, fwhm=0.5,
             internal_dnu=0.0025, species=6, lines=400000, profiles=1, retrieved=2, mixing=True, eps=1.0),
        # the pullback of a variational or learning loop over a mid-size band
        dict(kind="vjp", name="vjp_band", nu_lo=645.0, nu_hi=1000.0, dnu=0.25, opd=2.0, fwhm=0.5, internal_dnu=0.0025,
             species=6, lines=67139, profiles=2, retrieved=2, mixing=False, eps=0.98),
        # a whole retrieval: Levenberg-Marquardt on a batch of scenes from the a priori
        dict(kind="oe", name="oe_scenes", nu_lo=645.0, nu_hi=700.0, dnu=0.25, opd=2.0, fwhm=0.5, internal_dnu=0.0025,
             species=1, lines=5000, profiles=24, retrieved=1, mixing=False, eps=1.0),
        # surrogate serving: batches of 4096 through the 152 -> 4 x 1024 -> 8461 network
        dict(kind="infer", name="surrogate_4096", batch=4096, hidden=1024, layers=4, out=8461),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["xsec", "xsec", "forward", "forward", "forward", "jacobian", "vjp", "oe", "infer", "train"])
    if kind == "xsec":
        width = _log(rng, 20.0, 2115.0)
        lo = round(rng.uniform(645.0, 2760.0 - width), 2)
        return dict(kind=kind, nu_lo=lo, nu_hi=round(lo + width, 2),
                    points=int(width / rng.choice([0.0025, 0.0025, 0.005, 0.01])) + 1,
                    lines=int(max(200, width * _log(rng, 10.0, 90.0)) / (1.0 + width / 900.0)),
                    precision=rng.choice(["fp64", "fp64", "mixed"]), method=rng.choice([3, 3, 3, 1, 2]))
    if kind == "infer":
        return dict(kind=kind, batch=int(_log(rng, 1, 4096)), hidden=rng.choice([256, 512, 1000, 1024]),
                    layers=rng.choice([2, 3, 4]), out=rng.choice([221, 717, 2001, 8461]))
    if kind == "train":
        return dict(kind=kind, batch=int(_log(rng, 32, 1024)), hidden=rng.choice([256, 512, 1024]),
                    layers=rng.choice([2, 3, 4]), out=rng.choice([221, 717, 2001, 8461]))
    dnu, opd, fwhm = rng.choice([(0.25, 2.0, 0.5), (0.25, 2.0, 0.5), (0.625, 0.8, 0.0), (0.125, 4.0, 0.25)])
    c = dict(kind=kind, dnu=dnu, opd=opd, fwhm=fwhm, internal_dnu=rng.choice([0.0025, 0.0025, 0.005]),
             mixing=kind != "oe" and rng.random() < 0.3, eps=rng.choice([1.0, 1.0, 0.98, 0.9]))
    fp64 = kind == "forward" and rng.random() < 0.35
    width = _log(rng, 8.0, 60.0 if fp64 or kind == "oe" else 300.0)
    steps = max(4, int(width / dnu))
    c["nu_lo"] = 645.0 + 5.0 * rng.randrange(0, 150)
    c["nu_hi"] = c["nu_lo"] + steps * dnu
    c["species"] = rng.choice([1, 2, 3, 6])
    c["lines"] = int((width + 50.0) * _log(rng, 15.0, 90.0)) * c["species"]
    c["profiles"] = int(_log(rng, 1, 12))
    if kind == "forward":
        c.update(precision="fp64" if fp64 else "mixed", source=rng.choice(["cim", "cim", "toon"]),
                 apodization=rng.choice(["gaussian", "gaussian", "norton_beer_strong"]))
    else:
        c["retrieved"] = rng.choice([1, 1, 2])
    if kind == "oe":
        c.update(eps=1.0, profiles=int(_log(rng, 2, 24)))
    # points times lines per cm^-1, at most what the listed cases of the kind come to
    most = 2e7 if fp64 else {"forward": 8e8, "oe": 7e7}.get(kind, 1.2e8)
    while c["profiles"] > 1 and _density(c) > most:
        c["profiles"] -= 1
    c["lines"] = int(c["lines"] * min(1.0, most / _density(c)))
    return c


def _density(c):
    return c["profiles"] * _grid_points(c)[0] * c["lines"] / (c["nu_hi"] - c["nu_lo"])


# ------------------------------------------------------------------ inputs
# the molecules of a case, CO2 first (the 5,000-line list of the tests is CO2 alone)
MOLECULES = (2, 1, 3, 6, 4, 5)
_held = {}  # the line lists and the context that a program keeps


def _lists(case):
    """{molecule: line list} covering the case's range and the ILS and cutoff margins."""
    pkg = _package()
    lo, hi = case["nu_lo"], case["nu_hi"]
    n_sp = case.get("species", 1)
    key = (lo, hi, case["lines"], n_sp)
    if key not in _held:
        base, extra = divmod(case["lines"], n_sp)
        _held[key] = {mol: pkg.synthetic_linelist(base + (k < extra), mol, 1001 + k, lo, hi)
                      for k, mol in enumerate(MOLECULES[:n_sp])}
    return _held[key]


def _y0(case, lists):
    key = ("y0", len(lists[2]))
    if key not in _held:
        _held[key] = _package().synthetic.vpy_y0(len(lists[2]))
    return _held[key]


def _mixing(case, lists):
    if not case.get("mixing"):
        return None
    key = ("vpy", len(lists[2]))
    if key not in _held:
        _held[key] = _package().VPYLineMixing(_y0(case, lists))
    return _held[key]


def _sounder(case):
    return _package().Sounder.make(case["nu_lo"], case["nu_hi"], case["dnu"], opd_max=case["opd"],
                                   fwhm_gauss=case["fwhm"])


def _scenes(case, seed):
    """Perturbed AFGL profiles, viewing geometries and surface temperatures."""
    pkg = _package()
    profs, scan = pkg.synthetic.perturbed_profiles(case["profiles"], seed=seed)
    geoms = [pkg.ViewingGeometry(pkg.scan_angle_to_local_zenith(a)) for a in scan]
    g = np.random.Generator(np.random.PCG64(seed + 77))
    return profs, geoms, [float(p.temperature[0] + g.normal(0.0, 2.0)) for p in profs]


RETRIEVED = (1, 3)  # log H2O, log O3


def _spec(case, n_lev):
    return _package().StateVectorSpec(n_lev, list(RETRIEVED[:case["retrieved"]]), include_emissivity=False)


def _network(case, seed):
    """Weights, biases, scaling and inputs of the surrogate, as float32 arrays."""
    g = np.random.Generator(np.random.PCG64(seed))
    dims = [152] + [case["hidden"]] * case["layers"] + [case["out"]]
    w = [((g.standard_normal((o, i), dtype=np.float32) * np.float32(1.3 / math.sqrt(i))),
          g.standard_normal(o, dtype=np.float32) * np.float32(0.1)) for i, o in zip(dims[:-1], dims[1:])]
    x_mean = g.uniform(-10.0, 280.0, 152).astype(np.float32)
    x_sd = g.uniform(0.3, 12.0, 152).astype(np.float32)
    y_mean = g.uniform(200.0, 300.0, case["out"]).astype(np.float32)
    y_sd = g.uniform(1.0, 12.0, case["out"]).astype(np.float32)
    x = x_mean + x_sd * g.standard_normal((case["batch"], 152), dtype=np.float32)
    return w, (x_mean, x_sd, y_mean, y_sd), x


def _targets(case, seed, scaling):
    g = np.random.Generator(np.random.PCG64(seed + 5))
    return scaling[2] + scaling[3] * g.standard_normal((case["batch"], case["out"]), dtype=np.float32)


def prepare(case, seed):
    pkg = _package()
    ctx = pkg.default_context()
    s = dict(case=case, ctx=ctx)
    if case["kind"] in ("infer", "train"):
        w, scaling, x = _network(case, seed)
        sur = pkg.Surrogate(ctx, n_in=152, n_hidden=case["hidden"], n_layers=case["layers"], n_out=case["out"],
                            seed=seed)
        sur.set_params(np.concatenate([np.concatenate([a.ravel(), b]) for a, b in w]))
        pkg.check(sur.lib.irs_surrogate_set_scaling(sur.h, *(pkg._lib.fptr(a) for a in scaling)))
        s["sur"] = sur
        if case["kind"] == "infer":
            s["x"] = torch.from_numpy(x).cuda()
            s["out"] = torch.empty((case["batch"], case["out"]), dtype=torch.float32, device="cuda")
            s["ood"] = torch.empty(case["batch"], dtype=torch.float32, device="cuda")
        else:
            s["x"], s["y"] = x, _targets(case, seed, scaling)
        return s
    lists = _lists(case)
    s["lists"] = lists
    if case["kind"] == "xsec":
        g = np.random.Generator(np.random.PCG64(seed))
        s["grid"] = np.linspace(case["nu_lo"], case["nu_hi"], case["points"])
        s["T"], s["p"] = float(g.uniform(190.0, 310.0)), float(10.0 ** g.uniform(-2.5, 0.0))
        s["vmr"] = float(10.0 ** g.uniform(-5.0, -2.0))
        return s
    s["profs"], s["geoms"], s["T_sfc"] = _scenes(case, seed)
    s["sounder"], s["lm"] = _sounder(case), _mixing(case, lists)
    s["kw"] = dict(internal_dnu=case["internal_dnu"], continua=("h2o", "co2"))
    n_lev = len(s["profs"][0].pressure)
    if case["kind"] != "forward":
        s["spec"] = _spec(case, n_lev)
    n_ch = int(round((case["nu_hi"] - case["nu_lo"]) / case["dnu"])) + 1
    g = np.random.Generator(np.random.PCG64(seed + 99))
    if case["kind"] == "vjp":
        s["dy"] = g.standard_normal((case["profiles"], n_ch))
    if case["kind"] == "oe":
        # observations: the scenes' own spectra (two-digit agreement with the path that fits
        # them is not needed, so they come from it) plus noise of 0.2 K
        base = pkg.afgl_atmosphere("us_standard")
        afgl = [pkg.afgl_atmosphere(a) for a in pkg.synthetic.AFGL]
        truth = []
        for k, p in enumerate(s["profs"]):
            b = afgl[k % len(afgl)]  # the profile that this scene is a perturbation of
            truth.append(pkg.AtmosphericProfile(base.pressure, base.temperature + 0.3 * (p.temperature - b.temperature),
                                                base.altitude, {**base.vmr, 1: base.vmr[1] * p.vmr[1] / b.vmr[1]}))
        nu, _, bt = pkg.forward_model_batch(truth, lists, sounder=s["sounder"], geoms=s["geoms"], backend=ctx,
                                            precision="mixed", dptmn=0.0, **s["kw"])
        s["base"] = base
        s["xa"] = pkg.pack_state(s["spec"], base)
        corr = 3.0 * float(np.median(np.abs(np.diff(np.log(base.pressure)))))
        s["Sa"] = pkg.build_sa(s["spec"], base, sigma_T=1.0, L_T=corr, sigma_vmr=0.3, L_vmr=corr)
        s["Se"] = np.stack([pkg.scene_nedt(nu, b, nedt_280K=0.2) ** 2 for b in bt])
        s["y"] = bt + np.sqrt(s["Se"]) * g.standard_normal(bt.shape)
    return s


# ------------------------------------------------------------------ the calls
def run(s):
    pkg, case, ctx = _package(), s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "xsec":
        mol, = s["lists"]
        sigma = pkg.compute_voigt_cross_sections(s["grid"], s["lists"][mol], s["T"], s["p"], vmr_self=s["vmr"],
                                                 method=pkg.VoigtMethod(case["method"]), precision=case["precision"],
                                                 backend=ctx)
        return sigma if case["precision"] == "fp64" else sigma.astype(np.float32)
    if kind == "infer":
        s["sur"].predict_device(s["x"], s["out"], s["ood"])
        return s["out"], s["ood"]
    if kind == "train":
        g, loss = s["sur"].gradients(s["x"], s["y"])
        return g, np.float32(loss)
    if kind == "oe":
        r = pkg.optimal_estimation_batch(s["y"], s["spec"], [s["base"]] * case["profiles"], s["lists"], xa=s["xa"],
                                         Sa=s["Sa"], Se=s["Se"], sounder=s["sounder"], geoms=s["geoms"], backend=ctx,
                                         fm_kwargs=s["kw"])
        return dict(n_iter=r["n_iter"], **{k: r[k].astype(np.float32) for k in ("x", "y_fit", "M", "cost")})
    kw = dict(sounder=s["sounder"], geoms=s["geoms"], T_sfcs=s["T_sfc"], eps_sfcs=[case["eps"]] * case["profiles"],
              backend=ctx, line_mixing=s["lm"], **s["kw"])
    if kind == "forward":
        _, R, BT = pkg.forward_model_batch(s["profs"], s["lists"], precision=case["precision"],
                                           source_function=case["source"], apodization=case["apodization"], **kw)
        return (R, BT) if case["precision"] == "fp64" else (R.astype(np.float32), BT.astype(np.float32))
    if kind == "jacobian":
        _, K, y = pkg.analytic_jacobian_batch(s["profs"], s["lists"], s["spec"], **kw)
        return K.astype(np.float32), y.astype(np.float32)
    y, dx = pkg.vjp_batch(s["profs"], s["lists"], s["spec"], s["dy"], **kw)
    return y.astype(np.float32), dx.astype(np.float32)


# ------------------------------------------------------------------ necessary work
LAYERS, LEVELS = 49, 50


def _grid_points(case):
    hrf = math.ceil(case["dnu"] / case["internal_dnu"] - 1e-9)
    d = case["dnu"] / hrf
    n_ch = int(round((case["nu_hi"] - case["nu_lo"]) / case["dnu"])) + 1
    return (n_ch - 1) * hrf + 1 + 2 * math.ceil(16.0 / d), n_ch, d, hrf


def work(case):
    """Bytes: every input read and every output written once.  Operations: each line's
    parameters per layer, the few lines whose centre lies near a point (0.3 cm^-1, where the
    Voigt core is and no smooth sum of distant lines can stand in), the radiative transfer
    of each point and layer, and the ILS taps of each channel."""
    if case["kind"] in ("infer", "train"):
        dims = [152] + [case["hidden"]] * case["layers"] + [case["out"]]
        mac = sum(a * b for a, b in zip(dims[:-1], dims[1:]))
        params, b = mac + sum(dims[1:]), case["batch"]
        if case["kind"] == "infer":
            return {"bytes": 4 * b * (dims[0] + dims[-1] + 1) + 2 * params, "flops": 2.0 * b * mac}
        return {"bytes": 4 * b * (dims[0] + dims[-1]) + 6 * params, "flops": 6.0 * b * mac}
    if case["kind"] == "xsec":
        near = case["points"] * (case["lines"] / (case["nu_hi"] - case["nu_lo"])) * 0.6
        return {"bytes": 56 * case["lines"] + 16 * case["points"], "flops": 100.0 * case["lines"] + 10.0 * near}
    n, n_ch, d, _ = _grid_points(case)
    near = n * case["lines"] / (case["nu_hi"] - case["nu_lo"]) * 0.6
    once = LAYERS * (100.0 * case["lines"] + 10.0 * near + 40.0 * n)
    taps = 2.0 * n_ch * 32.0 / d
    p = case["profiles"]
    out = 16 * n_ch * p
    if case["kind"] == "forward":
        return {"bytes": 56 * case["lines"] + out, "flops": p * (once + taps)}
    n_state = LEVELS * (1 + case["retrieved"]) + 1
    if case["kind"] == "vjp":
        return {"bytes": 56 * case["lines"] + out, "flops": p * (4.0 * once + 2.0 * taps)}
    jac = p * (4.0 * once + (n_state + 1) * taps)
    if case["kind"] == "jacobian":
        return {"bytes": 56 * case["lines"] + out + 8 * n_state * n_ch * p, "flops": jac}
    steps = 3  # Levenberg-Marquardt steps, each a Jacobian and a trial spectrum, after the first Jacobian
    return {"bytes": 56 * case["lines"] + out + 8 * n_state * n_state * p,
            "flops": (1 + steps) * (jac + 2.0 * p * n_state ** 2 * n_ch) + steps * p * (once + taps)}


# ------------------------------------------------------------------ the same in 64 bits
C1, C2, C2_LINES = 1.191042953e-5, 1.4387769, 1.4387752
INV_SQRT_PI, SQRT_LN2 = 1.0 / math.sqrt(math.pi), math.sqrt(math.log(2.0))
MASS = {1: 18.010, 2: 44.010, 3: 47.998, 4: 44.013, 5: 28.010, 6: 16.043}
CUTOFF, X_FAR, DPTMN = 25.0, 122.0, 1e-6
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device=DEV)


def _weideman(n):
    """Weideman's rational series for w(z) (SIAM J. Numer. Anal. 31, 1994)."""
    m = 2 * n
    k = np.arange(-m + 1, m)
    L = math.sqrt(n / math.sqrt(2.0))
    t = L * np.tan(k * math.pi / m / 2)
    f = np.concatenate([[0.0], np.exp(-t * t) * (L * L + t * t)])
    a = np.real(np.fft.fft(np.fft.fftshift(f))) / (2 * m)
    return L, a[1:n + 1]


def _w(x, y):
    """Faddeeva w(x + iy), y >= 0."""
    z = torch.complex(x, y)
    out = torch.empty_like(z)
    far = x.abs() + y >= 8.0
    zf = z[far]
    r = torch.zeros_like(zf)
    for k in range(40, 0, -1):  # Laplace continued fraction
        r = (0.5 * k) / (zf - r)
    out[far] = 1j * INV_SQRT_PI / (zf - r)
    L, a = _weideman(64)
    zn = z[~far]
    Z = (L + 1j * zn) / (L - 1j * zn)
    p = torch.zeros_like(zn)
    for c in a[::-1]:
        p = p * Z + float(c)
    out[~far] = 2.0 * p / (L - 1j * zn) ** 2 + INV_SQRT_PI / (L - 1j * zn)
    return out


def _voigt24(x, y):
    """The 24-node trapezoid rule of the Weideman method, Re w."""
    L = math.sqrt(24 / math.log(2.0))
    acc = torch.zeros_like(x)
    wsum = torch.zeros_like(x)
    for n in range(1, 25):
        t = L * math.tan((2 * n - 25) * math.pi / 48)
        w = L * L + t * t
        d = (x - t) ** 2 + y * y
        acc += w * math.exp(-t * t) / d
        wsum += w / d
    sc = y / (24 * L)
    return torch.clamp(torch.exp(-x * x) * (1.0 - wsum * sc) + acc * sc, min=0.0)


_tables = {}


def _table(name):
    if name not in _tables:
        rows = [r.strip().split(",") for r in open(PACKAGE / "data" / name) if not r.startswith("#") and r.strip()]
        if name.startswith("tips"):
            _tables[name] = {(int(r[0]), int(r[1])): np.array([float(v) for v in r[2:]]) for r in rows}
        else:
            _tables[name] = np.array([[float(v) for v in r] for r in rows[1:]]).T
    return _tables[name]


def _partition(mol, T):
    q = _table("tips2024_q.csv")[(mol, 1)]
    i = int(min(max(math.floor(T) - 70, 0), len(q) - 1))
    f = T - math.floor(T)
    return q[i] * (1.0 - f) + q[min(i + 1, len(q) - 1)] * f


def _line_sum(grid, lines, mol, T, p, vs, method=3, coef=None, y0=None):
    """Cross section (cm^2) on grid of one species' lines at one (T, p, self VMR); with
    coef the lines whose peak optical depth stays under DPTMN are left out."""
    nu = _t(lines["wavenumber"])
    n_air = _t(lines["temp_depend"])
    n_self = {1: 0.95, 2: 0.75}.get(mol)
    d_self = {1: 0.002, 2: -0.003}.get(mol, 0.0)
    tr = 296.0 / T
    e_air = tr ** n_air
    e_self = e_air if n_self is None else tr ** n_self
    gl = e_air * _t(lines["air_broad"]) * (1.0 - vs) * p + e_self * _t(lines["self_broad"]) * vs * p
    gd = torch.clamp(nu * 3.58126e-7 * math.sqrt(T / MASS[mol]), min=1e-10)
    S = (_t(lines["intensity"]) * (_partition(mol, 296.0) / _partition(mol, T))
         * torch.exp(-C2_LINES * _t(lines["lower_energy"]) * (1.0 / T - 1.0 / 296.0))
         * (1.0 - torch.exp(-C2_LINES * nu / T)) / (1.0 - torch.exp(-C2_LINES * nu / 296.0)))
    centre = nu + (_t(lines["pressure_shift"]) * (1.0 - vs) + d_self * vs) * p
    f = SQRT_LN2 / gd
    y = gl * f
    Sn = S * f * INV_SQRT_PI
    YSn = None if y0 is None else _t(y0) * tr ** 0.75 * p * Sn
    if coef is not None:
        keep = Sn * torch.special.erfcx(y) * coef > DPTMN
        nu, gd, gl, S, centre, f, y, Sn = (v[keep] for v in (nu, gd, gl, S, centre, f, y, Sn))
        YSn = None if YSn is None else YSn[keep]
    order = torch.argsort(centre)
    gd, gl, S, centre, f, y, Sn = (v[order] for v in (gd, gl, S, centre, f, y, Sn))
    YSn = None if YSn is None else YSn[order]
    if method == 2:
        fG, fL = 2.0 * gd, 2.0 * gl
        gV = 0.5 * (fG ** 5 + 2.69269 * fG ** 4 * fL + 2.42843 * fG ** 3 * fL ** 2 + 4.47163 * fG ** 2 * fL ** 3
                    + 0.07842 * fG * fL ** 4 + fL ** 5) ** 0.2
        r = fL / (2.0 * gV)
        eta = 1.36603 * r - 0.47719 * r * r + 0.11116 * r ** 3

        def profile(d, s):
            g = math.sqrt(math.log(2.0) / math.pi) / gV[s, None] * torch.exp(-math.log(2.0) * (d / gV[s, None]) ** 2)
            lo = gV[s, None] / math.pi / (d * d + gV[s, None] ** 2)
            return eta[s, None] * lo + (1.0 - eta[s, None]) * g
        base = S * profile(torch.full_like(gV, CUTOFF)[:, None], slice(None))[:, 0]
    else:
        Hc = y * INV_SQRT_PI / ((CUTOFF * f) ** 2 + y * y)
    sigma = torch.zeros_like(grid)
    mix = torch.zeros_like(grid) if YSn is not None else None
    lo = torch.searchsorted(grid, centre - CUTOFF).tolist()
    hi = torch.searchsorted(grid, centre + CUTOFF, right=True).tolist()
    j = 0
    while j < len(lo):
        m = j + 1  # lines j..m-1 against the points that any of them reaches, 16 M pairs at most
        while m < len(lo) and (m + 1 - j) * (hi[m] - lo[j]) <= 1 << 24:
            m += 1
        s, a, b = slice(j, m), lo[j], max(hi[j:m])
        j = m
        if b <= a:
            continue
        d = grid[None, a:b] - centre[s, None]
        inside = d.abs() <= CUTOFF
        zr = d / CUTOFF
        if method == 2:
            v = S[s, None] * profile(d, s) - (2.0 - zr * zr) * base[s, None]
        else:
            x = d * f[s, None]
            yy = y[s, None]
            core = inside & (x.abs() <= X_FAR)
            den = INV_SQRT_PI / (x * x + yy * yy)
            H = yy * den
            xc, yc = x[core], yy.expand_as(x)[core]
            w = None
            if xc.numel():
                w = _w(xc, yc) if method == 3 else None
                H[core] = w.real if method == 3 else _voigt24(xc, yc)
            v = Sn[s, None] * (H - (2.0 - zr * zr) * Hc[s, None])
            if mix is not None:
                D = x * den
                if w is not None:
                    D[core] = w.imag
                mix[a:b] += torch.where(inside, YSn[s, None] * D, 0.0).sum(0)
        sigma[a:b] += torch.where(inside, v, 0.0).sum(0)
    sigma = torch.clamp(sigma, min=0.0)
    return sigma if mix is None else torch.clamp(sigma + mix, min=0.0)


def _near(a, b):
    return abs(a - b) <= 1.4901161193847656e-8 * max(abs(a), abs(b))


def _column_vmr(v1, v2, p1, p2):  # Curtis-Godson mean VMR and pressure of a layer
    if v1 <= 0 or v2 <= 0:
        return 0.5 * (v1 + v2), 0.5 * (p1 + p2)
    if _near(v1, v2):
        return v1, 0.5 * (p1 + p2)
    al, r = math.log(v2 / v1) / math.log(p2 / p1), p2 / p1
    b1, b2 = al + 1.0, al + 2.0
    v = (v1 - v2) / math.log(v1 / v2) if abs(b1) < 1e-8 else v1 * p1 * (1.0 - r ** b1) / (b1 * abs(p1 - p2))
    if abs(b1) < 1e-8:
        return v, abs(p1 - p2) / math.log(p1 / p2)
    if abs(b2) < 1e-8:
        return v, p2 * math.log(p2 / p1) / (p2 / p1 - 1.0)
    return v, p1 * b1 / b2 * (1.0 - r ** b2) / (1.0 - r ** b1)


def _mean_temperature(T1, T2, p1, p2):
    al = math.log(p2 / p1)
    be = p2 / p1
    return T1 if _near(T1, T2) else T1 + (T2 - T1) * (0.5 + al / 12.0 if abs(al) < 1e-3 else
                                                      ((al - 1.0) * be + 1.0) / (al * (be - 1.0)))


def _planck(nu, T):
    return C1 * nu ** 3 / torch.expm1(C2 * nu / T)


def _interp(table, k, nu):
    x = table[0]
    return _t(np.interp(nu, x, table[k]))


def _radiance(grid, prof, lists, case, mu, T_sfc, dptmn, y0):
    """Monochromatic radiance of one profile."""
    P, T, src, eps = prof.pressure, prof.temperature, case.get("source", "cim"), case["eps"]
    nu_h = grid.cpu().numpy()
    h2o, co2 = _table("mt_ckd43_h2o_coeffs.csv"), _table("mt_ckd_co2_coeffs.csv")
    cs, cf, te = (_interp(h2o, k, nu_h) for k in (1, 2, 3))
    se, td = _t(np.interp(nu_h, co2[0], co2[1] * co2[2])), _interp(co2, 3, nu_h)
    order = np.argsort(np.log(P))

    def at(v, p):
        return float(np.interp(math.log(p), np.log(P)[order], np.asarray(v)[order]))
    taus, temps = [], []
    for k in range(len(P) - 1):
        dp, pm = abs(P[k] - P[k + 1]), 0.5 * (P[k] + P[k + 1])
        tau = torch.zeros_like(grid)
        for mol, ll in lists.items():
            v, pcg = _column_vmr(prof.vmr[mol][k], prof.vmr[mol][k + 1], P[k], P[k + 1])
            if v == 0.0:
                continue
            coef = v * dp * 2.1209e22
            lm = y0 if mol == 2 else None
            tau += coef * _line_sum(grid, ll.lines, mol, at(T, pcg), pcg / 1013.25, v if mol == 1 else 0.0,
                                    coef=coef if dptmn and lm is None else None, y0=lm)
        Tm, vh, vc = at(T, pm), at(prof.vmr[1], pm), at(prof.vmr[2], pm)
        dz = 8.314462 * Tm / (0.028964 * 9.80665) * dp / pm * 100.0
        rho, x = (pm / 1013.0) * (296.0 / Tm), C2 * grid / Tm
        rad = torch.where(x <= 0.01, 0.5 * x * grid,
                          torch.where(x <= 10.0, grid * (1.0 - torch.exp(-x)) / (1.0 + torch.exp(-x)), grid))
        n = pm * 100.0 / (1.380649e-23 * Tm) * 1e-6
        tau += (cs * (296.0 / Tm) ** te * vh + cf * (1.0 - vh)) * rho * rad * (n * vh) * dz
        tau += se * torch.where(td == 0.0, torch.ones_like(td), (Tm / 246.0) ** td) * (1e-20 * n * vc * rho) * rad * dz
        taus.append(tau / mu)
        temps.append((_mean_temperature(T[k], T[k + 1], P[k], P[k + 1]), T[k], T[k + 1]))

    def cim(s):
        e = torch.exp(-s)
        return torch.where(s < 0.06, s / 6.0, 1.0 - 2.0 * (e / (e - 1.0) + 1.0 / s))

    def lit(s):
        e = torch.exp(-s)
        return torch.where(s < 1e-4, s * (0.5 - s * (1.0 / 3.0 - s * 0.125)), (1.0 - e) / s - e)
    up = torch.ones_like(grid)
    I = torch.zeros_like(grid)
    for k in range(len(taus) - 1, -1, -1):
        s, (Ta, Tb, Tt) = taus[k], temps[k]
        down = up * torch.exp(-s)
        Bt = _planck(grid, Tt)
        if src == "cim":
            Ba = _planck(grid, Ta)
            I += (up - down) * (Ba + (Bt - Ba) * cim(s))
        else:
            I += Bt * (up - down) + (_planck(grid, Tb) - Bt) * up * lit(s)
        up = down
    I += eps * _planck(grid, T_sfc) * up
    if eps < 1.0:
        sky, g = torch.zeros_like(grid), torch.ones_like(grid)
        for s, (Ta, Tb, Tt) in zip(taus, temps):
            u, Bb = 1.0 - torch.exp(-s), _planck(grid, Tb)
            if src == "cim":
                Ba = _planck(grid, Ta)
                sky += g * u * (Ba + (Bb - Ba) * cim(s))
            else:
                sky += g * (Bb * u + (_planck(grid, Tt) - Bb) * lit(s))
            g = g * torch.exp(-s)
        I += (1.0 - eps) * sky * up
    return I


def _ils(case, d):
    half = math.ceil(16.0 / d)
    dv = torch.arange(-half, half + 1, dtype=torch.float64, device=DEV) * d
    L = torch.arange(2048, dtype=torch.float64, device=DEV) / 2047.0 * case["opd"]
    if case.get("apodization", "gaussian") == "gaussian":
        sg = case["fwhm"] / (2.0 * math.sqrt(2.0 * math.log(2.0)))
        A = torch.exp(-2.0 * (math.pi * sg * L) ** 2)
    else:
        t = 1.0 - (L / case["opd"]) ** 2
        A = 0.045335 + 0.554883 * t ** 2 + 0.399782 * t ** 4
    k = torch.cos(2.0 * math.pi * dv[:, None] * L[None, :]) @ A
    return k / (k.sum() * d)


def _spectra(case, seed, dptmn=True):
    """(R, BT) of the case's scenes, [profiles][channels]."""
    profs, geoms, T_sfc = _scenes(case, seed)
    lists = _lists(case)
    n, n_ch, d, step = _grid_points(case)
    half = math.ceil(16.0 / d)
    den = round(1.0 / d)
    grid = (torch.arange(n, dtype=torch.float64, device=DEV) + round(case["nu_lo"] * den) - half) / den
    chan = case["nu_lo"] + case["dnu"] * torch.arange(n_ch, dtype=torch.float64, device=DEV)
    kern = _ils(case, d)
    y0 = _y0(case, lists) if case["mixing"] else None
    R = torch.stack([_radiance(grid, p, lists, case, g.mu, ts, dptmn, y0).unfold(0, 2 * half + 1, step) @ kern * d
                     for p, g, ts in zip(profs, geoms, T_sfc)])
    return R, torch.where(R > 0.0, C2 * chan / torch.log1p(C1 * chan ** 3 / R), 0.0)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.erf(x / math.sqrt(2.0)))


def exact(case, seed):
    kind = case["kind"]
    if kind == "oe":
        return None
    if kind in ("infer", "train"):
        w, (x_mean, x_sd, y_mean, y_sd), x = _network(case, seed)
        par = [(_t(a).requires_grad_(kind == "train"), _t(b).requires_grad_(kind == "train")) for a, b in w]
        h = (_t(x) - _t(x_mean)) / _t(x_sd)
        for k, (a, b) in enumerate(par):
            h = h @ a.T + b
            h = _gelu(h) if k + 1 < len(par) else h
        if kind == "infer":
            return (h * _t(y_sd) + _t(y_mean)).float().cpu(), None
        t = (_t(_targets(case, seed, (x_mean, x_sd, y_mean, y_sd))) - _t(y_mean)) / _t(y_sd)
        loss = 0.5 * ((h - t) ** 2).mean()
        loss.backward()
        return torch.cat([v.grad.reshape(-1) for ab in par for v in ab]).cpu(), loss.detach().cpu()
    if kind == "xsec":
        g = np.random.Generator(np.random.PCG64(seed))
        T, p, vs = float(g.uniform(190.0, 310.0)), float(10.0 ** g.uniform(-2.5, 0.0)), float(10.0 ** g.uniform(-5.0, -2.0))
        (mol, ll), = _lists(case).items()
        return _line_sum(_t(np.linspace(case["nu_lo"], case["nu_hi"], case["points"])), ll.lines, mol, T, p, vs,
                         method=case["method"]).cpu()
    n = _grid_points(case)[0]
    pairs = LAYERS * case["profiles"] * n * case["lines"] * min(1.0, 50.0 / (case["nu_hi"] - case["nu_lo"]))
    if pairs > 8e10:  # over about 20 seconds
        return None
    R, BT = _spectra(case, seed, dptmn=kind == "forward")
    if kind == "forward":
        return R.cpu(), BT.cpu()
    return (None, BT.cpu()) if kind == "jacobian" else (BT.cpu(), None)
