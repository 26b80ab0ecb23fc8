"""Timed cases: the calls that a fitting program makes, over the sizes it makes them at.

Every case is one call of a public entry point of ``imfit_gb300.ModelObject`` on
a synthetic image (a model with seeded noise).  A case holds

  call    what the program asks for:
            grad       statistic + adjoint gradient (gradient-based minimisers)
            stat       statistics only (differential evolution, chains)
            jtwj       J^T W J, J^T W dev and the statistic (Levenberg-Marquardt)
            cutouts    the same of a set of cutouts of uneven sizes
            plain_stat the FP64 drop-in statistic
            plain_dev  the FP64 drop-in deviates (mpfit's user function)
            plain_fd   the FP64 drop-in statistic and finite-difference gradient
            image      the FP64 drop-in model image (makeimage)
  model   a name of MODELS: the functions of the configuration file
  cols, rows, psf_cols, psf_rows   image and PSF sizes (PSFs are odd)
  batch   parameter vectors of one call; for cutouts, their number
  region, scale   side of an oversampled region in the middle (0: none), its scale
  mask    share of masked pixels
  stat    chi2 | sigma (chi^2 with an error image) | model (model-based errors) | cash | pmlr

``exact`` evaluates the same quantities with torch in 64 bits: the image
functions' formulas, their subsampling rules, a 64-bit FFT convolution, and
automatic differentiation for derivatives.
"""
import math

import numpy as np
import torch

import imfit_gb300
from imfit_gb300 import workloads

D2R = math.pi / 180.0

# functions of each model (all in one function set) -- the bulge, disk, ring,
# bar, nucleus and sky combinations of the repository's workloads and tests
MODELS = {
    "sersic_sky": ["Sersic", "FlatSky"],
    "bulge_disk": ["Sersic", "Exponential"],
    "bulge_disk_sky": ["Sersic", "Exponential", "FlatSky"],
    "ring_sky": ["Sersic", "Exponential", "GaussianRing", "FlatSky"],
    "core_plane": ["Moffat", "Gaussian", "Exponential", "TiltedSkyPlane"],
    "nucleus_sky": ["PointSource", "Sersic", "Exponential", "FlatSky"],
    "edge_on_bar": ["ExponentialDisk3D", "FerrersBar3D"],
}
NAMES = {"Sersic": "PA ell n I_e r_e", "Exponential": "PA ell I_0 h", "FlatSky": "I_sky",
         "GaussianRing": "PA ell A R sigma", "Moffat": "PA ell I_0 fwhm beta", "Gaussian": "PA ell I_0 sigma",
         "TiltedSkyPlane": "I_0 m_x m_y", "PointSource": "I_tot", "ExponentialDisk3D": "PA inc J_0 h n z_0",
         "FerrersBar3D": "PA inc barPA J_0 R_bar q q_z n"}
SUBSAMPLED = {"Sersic": (4.0, 20), "Exponential": (3.0, 20), "Moffat": (3.0, 40), "Gaussian": (3.0, 40)}
PLAIN = ("plain_stat", "plain_dev", "plain_fd", "image")
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _case(name, call, model, cols, rows, psf, batch=1, region=0, scale=0, mask=0.0, stat="chi2"):
    pc, pr = psf if isinstance(psf, tuple) else (psf, psf)
    c = dict(call=call, model=model, cols=cols, rows=rows, psf_cols=pc, psf_rows=pr, batch=batch, region=region,
             scale=scale, mask=mask, stat=stat)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest fits: a postage stamp, where launches and latency are all
        _case("grad_stamp", "grad", "bulge_disk_sky", 40, 31, (13, 15)),
        # one galaxy, one component and the sky: the common single-image fit
        _case("grad_256", "grad", "sersic_sky", 256, 256, 51),
        # a large image with an oversampled centre and a mask, one vector at a time
        _case("grad_1024_region", "grad", "bulge_disk_sky", 1024, 1024, 63, region=40, scale=5, mask=0.1),
        # line-of-sight integrals per pixel
        _case("grad_3d_512", "grad", "edge_on_bar", 512, 512, 35, stat="sigma"),
        # a population with gradients: 256 vectors on one Poisson image
        _case("population_grad", "grad", "ring_sky", 512, 512, 51, batch=256, stat="cash"),
        # a generation of differential evolution: statistics only, ragged sizes
        _case("generation_stat", "stat", "core_plane", 301, 223, (25, 31), batch=104, mask=0.05, stat="pmlr"),
        # a Levenberg-Marquardt evaluation of the large image
        _case("jtwj_1024_region", "jtwj", "bulge_disk_sky", 1024, 1024, 63, region=40, scale=5, mask=0.1),
        # a Levenberg-Marquardt evaluation with a nucleus and model-based errors, odd sizes
        _case("jtwj_nucleus", "jtwj", "nucleus_sky", 203, 171, 35, stat="model"),
        # one lockstep round of many uneven cutouts (48 to 384 px) with their own PSFs
        _case("cutouts_256", "cutouts", "bulge_disk", 384, 384, 63, batch=256, stat="sigma"),
        # the FP64 drop-in under the reference's unchanged solvers
        _case("plain_stat_1024_region", "plain_stat", "bulge_disk_sky", 1024, 1024, 63, region=40, scale=5, mask=0.1),
        _case("plain_fd_256", "plain_fd", "sersic_sky", 256, 256, 51),
        _case("plain_dev_3d_256", "plain_dev", "edge_on_bar", 256, 256, 35, stat="sigma"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(rng, lo, hi):
    return 2 * rng.randint(lo // 2, (hi - 1) // 2) + 1


def draw(rng):
    call = rng.choice(["grad", "grad", "population", "stat", "jtwj", "jtwj", "cutouts", "3d", "plain", "plain"])
    psf = (_odd(rng, 9, 63), _odd(rng, 9, 63))
    if call == "cutouts":
        return _case(None, "cutouts", "bulge_disk", _log(rng, 96, 384), _log(rng, 96, 384), _odd(rng, 25, 63),
                     batch=_log(rng, 6, 256), stat="sigma")
    if call == "3d":
        plain = rng.random() < 0.4
        hi = 256 if plain else 512
        return _case(None, "plain_dev" if plain else "grad", "edge_on_bar", _log(rng, 40, hi), _log(rng, 40, hi),
                     (_odd(rng, 9, 35), _odd(rng, 9, 35)), stat="sigma")
    flat = [m for m in MODELS if m != "edge_on_bar"]
    if call in ("population", "stat"):
        cols, rows = _log(rng, 48, 512), _log(rng, 48, 512)
        batch = min(_log(rng, 4, 256), 256 * 512 * 512 // (cols * rows))
        return _case(None, "grad" if call == "population" else "stat", rng.choice(flat), cols, rows, psf, batch=batch,
                     mask=rng.choice([0.0, 0.05]), stat=rng.choice(["chi2", "cash", "pmlr"]))
    if call == "plain":
        call = rng.choice(PLAIN)
    hi = {"plain_fd": 320}.get(call, 1024)
    cols, rows = _log(rng, 28, hi), _log(rng, 28, hi)
    region = rng.choice([0, 0, 24, 33]) if min(cols, rows) >= 64 and call != "image" else 0
    model = rng.choice(flat)
    if region and model == "nucleus_sky":
        model = "bulge_disk_sky"
    stat = rng.choice(["chi2", "sigma", "model", "pmlr"] if call in ("jtwj", "plain_dev") else ["chi2", "model", "cash"])
    if call == "plain_fd" or call == "image":
        stat = "chi2"
    return _case(None, call, model, cols, rows, psf, region=region, scale=rng.choice([2, 3, 4, 5]) if region else 0,
                 mask=rng.choice([0.0, 0.1]), stat=stat)


def _nparams(model):
    return 2 + sum(len(NAMES[f].split()) for f in MODELS[model])


# ------------------------------------------------------------------ inputs
def _truth(rng, case):
    """A true parameter vector; scales follow the image's smaller side."""
    s = min(case["cols"], case["rows"])
    out = [case["cols"] / 2 + 0.5 + rng.uniform(-0.5, 0.5), case["rows"] / 2 + 0.5 + rng.uniform(-0.5, 0.5)]
    pa, inc = rng.uniform(0, 180), rng.uniform(80, 88)
    for f in MODELS[case["model"]]:
        out += {"Sersic": lambda: [rng.uniform(0, 180), rng.uniform(0.05, 0.5), rng.uniform(1, 4), rng.uniform(20, 60),
                                   max(2.0, s * rng.uniform(0.015, 0.05))],
                "Exponential": lambda: [rng.uniform(0, 180), rng.uniform(0.2, 0.6), rng.uniform(15, 30),
                                        max(3.0, s * rng.uniform(0.04, 0.09))],
                "FlatSky": lambda: [rng.uniform(20, 120)],
                "GaussianRing": lambda: [rng.uniform(0, 180), rng.uniform(0.1, 0.5), rng.uniform(8, 15),
                                         s * rng.uniform(0.1, 0.15), max(1.5, 0.016 * s)],
                "Moffat": lambda: [rng.uniform(0, 180), rng.uniform(0.05, 0.3), rng.uniform(200, 600),
                                   rng.uniform(3, 8), rng.uniform(2.5, 4.5)],
                "Gaussian": lambda: [rng.uniform(0, 180), rng.uniform(0.05, 0.3), rng.uniform(50, 200),
                                     rng.uniform(2, 6)],
                "TiltedSkyPlane": lambda: [rng.uniform(80, 120), rng.uniform(-0.02, 0.02), rng.uniform(-0.02, 0.02)],
                "PointSource": lambda: [rng.uniform(2e3, 2e4)],
                "ExponentialDisk3D": lambda: [pa, inc, 0.5, 40.0 * s / 512, 1.0, max(1.0, 6.0 * s / 512)],
                "FerrersBar3D": lambda: [pa, inc, rng.uniform(0, 180), 0.2, 30.0 * s / 512, 0.4, 0.2667, 2.0]}[f]()
    return np.array(out)


def _perturb(rng, case, truth, frac, pos):
    p = truth * (1 + rng.uniform(-frac, frac, truth.size))
    p[:2] = truth[:2] + rng.uniform(-pos, pos, 2)
    i = 2
    for f in MODELS[case["model"]]:
        for n in NAMES[f].split():
            if n == "ell":
                p[i] = min(p[i], 0.9)
            elif n == "inc":
                p[i] = min(truth[i] + rng.uniform(-2, 2), 89.5)
            elif n in ("PA", "barPA") and case["model"] == "edge_on_bar":
                p[i] = truth[i] + rng.uniform(-3, 3)
            elif n == "n" and f == "FerrersBar3D":
                p[i] = truth[i]
            i += 1
    return p


def _moffat(cols, rows, fwhm, beta, sub=3):
    alpha = fwhm / (2.0 * math.sqrt(2.0 ** (1.0 / beta) - 1.0))
    off = (np.arange(sub) + 0.5) / sub - 0.5
    x = (np.arange(cols)[:, None] + off - (cols - 1) / 2.0).ravel() ** 2
    y = (np.arange(rows)[:, None] + off - (rows - 1) / 2.0).ravel() ** 2
    p = (1.0 + (y[:, None] + x[None, :]) / alpha ** 2) ** -beta
    p = p.reshape(rows, sub, cols, sub).sum(axis=(1, 3))
    return p / p.sum()


class _Inputs:
    """The image, errors, mask, PSFs and parameter vectors of one (case, seed)."""

    def __init__(self, case, seed, cutout=None):
        self.case = case
        rng = np.random.default_rng([20 + int(seed), 0 if cutout is None else cutout + 1])
        self.gain, self.read_noise, self.sky = 4.0, 5.0, 0.0
        if case["stat"] in ("cash", "pmlr"):
            self.gain, self.read_noise = 1.0, 0.0
        fwhm, beta = rng.uniform(2.5, 5.0), rng.uniform(2.5, 4.5)
        if case["model"] == "edge_on_bar":
            beta = 8.0  # close to a Gaussian
        self.psf = _moffat(case["psf_cols"], case["psf_rows"], fwhm, beta)
        self.region = None
        if case["region"]:
            k, half = case["scale"], case["region"] // 2
            x1, y1 = case["cols"] // 2 - half + 1, case["rows"] // 2 - half + 1
            self.region = (x1, x1 + case["region"] - 1, y1, y1 + case["region"] - 1)
            self.os_psf = _moffat(k * case["psf_cols"] | 1, k * case["psf_rows"] | 1, k * fwhm, beta, 1)
        truth = _truth(rng, case)
        n = case["batch"] if cutout is None else 1
        if n > 1:
            self.params = np.stack([_perturb(rng, case, truth, 0.3, 3.0) for _ in range(n)])
        else:
            self.params = _perturb(rng, case, truth, 0.1 if case["model"] != "edge_on_bar" else 0.05, 1.0)[None]
        shape = (case["rows"], case["cols"])
        with torch.no_grad():
            img = _model(self, _lists(self, truth, subsample=False), torch.tensor(truth, device=DEV), 24).cpu().numpy()
        if case["model"] == "edge_on_bar":
            self.sigma = np.full(shape, 5.0)
            self.data = img + rng.normal(0.0, 5.0, shape)
        else:
            e = rng.poisson(np.clip(img, 0, None) * self.gain).astype(np.float64)
            self.data = (e + rng.normal(0.0, 1.0, shape) * self.read_noise) / self.gain
            self.sigma = np.sqrt(np.clip(img, 1, None) / self.gain + (self.read_noise / self.gain) ** 2)
        self.mask = (rng.random(shape) < case["mask"]).astype(np.float64) if case["mask"] else None


def _object(case):
    m = imfit_gb300.ModelObject(0)
    for i, f in enumerate(MODELS[case["model"]]):
        m.add_function(f, i == 0)
    m.finish_functions()
    return m


def _cutout_cases(case, seed):
    """The cutouts' own sizes: sides log-uniform from 48 px to the case's, odd PSFs from 25 px to the case's."""
    rng = np.random.default_rng([11, int(seed)])
    out = []
    for _ in range(case["batch"]):
        side = [int(math.exp(rng.uniform(math.log(48), math.log(case[k] + 1)))) for k in ("cols", "rows")]
        p = 2 * int(rng.integers(12, case["psf_cols"] // 2 + 1)) + 1
        out.append(dict(case, cols=side[0], rows=side[1], psf_cols=p, psf_rows=p, batch=1))
    return out


def prepare(case, seed):
    m = _object(case)
    if case["call"] == "cutouts":
        ins = [_Inputs(c, seed, i) for i, c in enumerate(_cutout_cases(case, seed))]
        m.setup_cutouts([i.data for i in ins], [i.sigma for i in ins], [i.psf for i in ins])
        return m, case, np.concatenate([i.params for i in ins])
    i = _Inputs(case, seed)
    m.add_psf(i.psf)
    m.add_image_data(i.data)
    m.add_image_characteristics(i.gain, i.read_noise, 1.0, 1, i.sky)
    if i.region:
        m.add_oversampled_psf(i.os_psf, case["scale"], i.region)
    if case["stat"] == "sigma":
        m.add_error_vector(i.sigma)
    if i.mask is not None:
        m.add_mask_vector(i.mask)
    if case["stat"] == "model":
        m.use_model_errors()
    elif case["stat"] == "cash":
        m.use_cash()
    elif case["stat"] == "pmlr":
        m.use_pmlr()
    if m.final_setup() != 0:
        raise RuntimeError(m.last_error)
    return m, case, i.params


def _f32(*values):
    """The fast path's results: doubles that hold sums of values evaluated in FP32."""
    return [torch.as_tensor(v, dtype=torch.float32) for v in values]


def run(state):
    m, case, params = state
    call = case["call"]
    if call == "grad":
        if case["batch"] > 1:
            return _f32(*m.batch_statistic_and_gradient(params))
        return _f32(*m.statistic_and_gradient(params[0]))
    if call == "stat":
        return _f32(m.batch_statistic_and_gradient(params, want_grad=False) if case["batch"] > 1
                    else m.fit_statistic_fast(params[0]))
    if call == "jtwj":
        return _f32(*m.jtwj(params[0]))
    if call == "cutouts":
        return _f32(*m.cutouts_jtwj(np.arange(case["batch"]), params))
    if call == "plain_stat":
        return m.get_fit_statistic(params[0])
    if call == "plain_dev":
        return m.compute_deviates(params[0])
    if call == "plain_fd":
        return m.statistic_and_gradient_fd(params[0])
    m.create_model_image(params[0])
    return m.get_model_image()


def work(case):
    """Bytes: the image and its weights once (at the width the path keeps them), parameters and results.
    Flops: per window pixel and component the profile (and its derivatives), the FFT convolutions at
    2.5 N log2 N per real transform, the statistic."""
    if case["call"] == "cutouts":
        cs = [dict(c, call="jtwj") for c in _cutout_cases(case, 0)]
        w = [work(c) for c in cs]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    n, comps = _nparams(case["model"]), len(MODELS[case["model"]])
    px, call = case["cols"] * case["rows"], case["call"]
    width = 8 if call in PLAIN else 4
    grids = [((case["cols"] + case["psf_cols"] - 1) * (case["rows"] + case["psf_rows"] - 1))]
    if case["region"]:
        k, r = case["scale"], case["region"]
        grids.append((k * r + k * case["psf_cols"] - 1) * (k * r + k * case["psf_rows"] - 1))
    # flops per pixel and component of a value and of all derivatives; line-of-sight integrals sum some 60 nodes
    value, deriv = (1200.0, 3600.0) if case["model"] == "edge_on_bar" else (25.0, 50.0)
    flops = 0.0
    for g in grids:
        fft = 5.0 * g * math.log2(g)  # one convolution: a forward and an inverse real transform
        one = g * comps * value + fft + 8.0 * px
        flops += {"grad": one + g * comps * deriv + fft, "jtwj": one + g * comps * deriv + (n - 1) * fft
                  + px * n * (n + 1.0), "plain_fd": (n + 1.0) * one}.get(call, one)
    flops *= case["batch"]
    out = {"grad": n + 1, "stat": 1, "jtwj": n * n + n + 1, "plain_stat": 1, "plain_fd": n + 1}.get(call, px)
    inputs = 0 if call == "image" else 2 * px * width
    return {"bytes": inputs + 8.0 * case["batch"] * (n + (out if out != px else 0)) + (8.0 * px if out == px else 0),
            "flops": flops}


# ------------------------------------------------------------ 64-bit values
def _axes(ins):
    """Pixel coordinates (y, x) of the model window, and of the region's window."""
    def axis(start, step, n):
        return start + step * torch.arange(n, dtype=torch.float64, device=DEV)
    c = ins.case
    win = (axis(1 - (c["psf_rows"] // 2), 1.0, c["rows"] + c["psf_rows"] - 1),
           axis(1 - (c["psf_cols"] // 2), 1.0, c["cols"] + c["psf_cols"] - 1))
    out = [win]
    if ins.region:
        k, (pr, pc), (x1, x2, y1, y2) = c["scale"], ins.os_psf.shape, ins.region
        off = 0.5 / k - 0.5
        out.append((axis(y1 + off - (pr // 2) / k, 1.0 / k, (y2 - y1 + 1) * k + pr - 1),
                    axis(x1 + off - (pc // 2) / k, 1.0 / k, (x2 - x1 + 1) * k + pc - 1)))
    return out


def _slices(case):
    i, out = 2, []
    for f in MODELS[case["model"]]:
        n = len(NAMES[f].split())
        out.append((f, slice(i, i + n)))
        i += n
    return out


def _rotated(p, t, x, y):
    """Offsets along and across the position angle (degrees, from the +y axis)."""
    a = (p[0] + 90.0) * D2R
    dx, dy = x - t[0], y - t[1]
    return dx * torch.cos(a) + dy * torch.sin(a), -dx * torch.sin(a) + dy * torch.cos(a)


def _radius(p, t, x, y):
    xp, yp = _rotated(p, t, x, y)
    ys = yp / (1.0 - p[1])
    return torch.sqrt(xp * xp + ys * ys)


def _moffat_alpha(p):
    return 0.5 * p[3] / torch.sqrt(torch.pow(2.0, 1.0 / p[4]) - 1.0)


def _radial(f, p, r):
    if f == "Sersic":
        n = p[2]
        bn = (2 * n - 0.333333333333333 + 0.009876543209876543 / n + 0.0018028610621203215 / n ** 2
              + 0.00011409410586365319 / n ** 3 - 7.1510122958919723e-05 / n ** 4)  # n > 0.36
        return p[3] * torch.exp(-bn * (torch.pow(r / p[4], 1.0 / n) - 1.0))
    if f == "Exponential":
        return p[2] * torch.exp(-r / p[3])
    if f == "GaussianRing":
        return p[2] * torch.exp(-(r - p[3]) ** 2 / (2 * p[4] ** 2))
    if f == "Gaussian":
        return p[2] * torch.exp(-r * r / (2 * p[3] ** 2))
    return p[2] * torch.pow(1.0 + (r / _moffat_alpha(p)) ** 2, -p[4])


def _lists(ins, theta, subsample=True):
    """Per grid and function, the pixels that are averaged over ns x ns subsamples, by ns."""
    t = torch.as_tensor(theta, dtype=torch.float64, device=DEV)
    out = []
    for y, x in _axes(ins):
        per = []
        for f, sl in _slices(ins.case):
            groups = []
            if subsample and f in SUBSAMPLED:
                inner, small = SUBSAMPLED[f]
                p = t[sl]
                scale = float(_moffat_alpha(p) if f == "Moffat" else p[-1])
                r = _radius(p, t, x[None, :], y[:, None])
                ns = torch.clamp((20 / torch.clamp(r, min=1e-3)).to(torch.int64), max=100)
                ns[r <= inner] = 20
                if scale <= 1.0:
                    ns[r <= 1.0] = min(int(small / scale), 100)
                ns[r >= 10.0] = 1
                for v in torch.unique(ns).tolist():
                    if v > 1:
                        groups.append((v, torch.nonzero(ns.reshape(-1) == v).reshape(-1)))
            per.append(groups)
        out.append(per)
    return out


_DE = {}


def _de_nodes(n):
    """Double-exponential (tanh-sinh) nodes and weights on [0, 1]: distances from both ends without cancellation."""
    if n not in _DE:
        h = 6.4 / (n - 1)
        u = torch.arange(n, dtype=torch.float64) * h - 3.2
        s = 0.5 * math.pi * torch.sinh(u)
        left = 1.0 / (1.0 + torch.exp(-2.0 * s))  # distance from 0
        w = h * 0.25 * math.pi * torch.cosh(u) / torch.cosh(s) ** 2
        _DE[n] = (left.to(DEV), w.to(DEV))
    return _DE[n]


def _integrate(f, a, b, n):
    x, w = _de_nodes(n)
    s = a[..., None] + (b - a)[..., None] * x
    return ((b - a)[..., None] * w * f(s)).sum(-1)


def _line_of_sight(f, p, t, x, y, nodes):
    """The 3-D functions: integrals of the luminosity density along the line of sight, over pieces on
    which it is smooth (the pieces are held fixed in derivatives: the integrand is continuous)."""
    xp, yp = _rotated(p, t, x, y)
    ci, si = torch.cos(p[1] * D2R), torch.sin(p[1] * D2R)

    def depth(s):
        return yp[..., None] * ci + s * si, yp[..., None] * si - s * ci

    if f == "ExponentialDisk3D":
        def density(s):
            yd, zd = depth(s)
            r = torch.sqrt(xp[..., None] ** 2 + yd * yd)
            alpha = 2.0 / p[4]
            u = torch.abs(zd) / (alpha * p[5])
            lnsech = math.log(2.0) - u - torch.log1p(torch.exp(-2.0 * u))
            return p[2] * torch.exp(-r / p[3] + alpha * lnsech)

        lim = 20.0 * p[3].detach()
        with torch.no_grad():
            c, q = ci.detach(), si.detach()
            b1 = torch.minimum(torch.maximum(-yp.detach() * c / q, -lim), lim)
            b2 = torch.minimum(torch.maximum(yp.detach() * q / c, -lim), lim)
            lo, hi = torch.minimum(b1, b2), torch.maximum(b1, b2)
        e = torch.ones_like(lo)
        return sum(_integrate(density, u, v, nodes) for u, v in ((-lim * e, lo), (lo, hi), (hi, lim * e)))

    cb, sb = torch.cos((p[2] + 90.0) * D2R), torch.sin((p[2] + 90.0) * D2R)
    a2 = p[4] ** 2
    b2, c2 = p[5] ** 2 * a2, p[6] ** 2 * a2

    def m2(s):
        yd, zd = depth(s)
        xb, yb = xp[..., None] * cb + yd * sb, -xp[..., None] * sb + yd * cb
        return yb * yb / a2 + xb * xb / b2 + zd * zd / c2

    with torch.no_grad():  # the chord of the ellipsoid: m2 is quadratic in s
        s = torch.tensor([-1.0, 0.0, 1.0], dtype=torch.float64, device=DEV) * p[4]
        v = m2(s.expand(*xp.shape, 3)).detach()
        qa = 0.5 * (v[..., 0] + v[..., 2]) - v[..., 1]
        qb = 0.5 * (v[..., 2] - v[..., 0])
        disc = torch.clamp(qb * qb - 4 * qa * (v[..., 1] - 1.0), min=0.0)
        lo, hi = ((-qb + k * torch.sqrt(disc)) / (2 * qa) * p[4].detach() for k in (-1.0, 1.0))

    def density(s):
        return p[3] * torch.pow(torch.clamp(1.0 - m2(s), min=1e-300), p[7])

    return torch.where(disc > 0, _integrate(density, lo, hi, nodes), torch.zeros_like(xp))


def _grid_image(ins, y, x, groups, t, nodes):
    total = torch.zeros(len(y), len(x), dtype=torch.float64, device=DEV)
    xs, ys = x[None, :], y[:, None]
    for (f, sl), lists in zip(_slices(ins.case), groups):
        p = t[sl]
        if f == "PointSource":
            continue
        if f == "FlatSky":
            total = total + p[0]
        elif f == "TiltedSkyPlane":
            total = total + p[0] + p[1] * (xs - t[0]) + p[2] * (ys - t[1])
        elif f.endswith("3D"):
            rows = max(1, (6 << 20) // (nodes * len(x)))
            total = total + torch.cat([_line_of_sight(f, p, t, xs, ys[i:i + rows], nodes)
                                       for i in range(0, len(y), rows)])
        else:
            v = _radial(f, p, _radius(p, t, xs, ys)).reshape(-1)
            for ns, idx in lists:
                off = (torch.arange(ns, dtype=torch.float64, device=DEV) + 0.5) / ns - 0.5
                px = x[idx % len(x)][:, None, None] + off[None, :, None]
                py = y[idx // len(x)][:, None, None] + off[None, None, :]
                v = torch.index_put(v, (idx,), _radial(f, p, _radius(p, t, px, py)).mean((1, 2)))
            total = total + v.reshape(len(y), len(x))
    return total


def _valid(img, psf):
    k = torch.as_tensor(psf / psf.sum(), dtype=torch.float64, device=DEV)
    full = torch.fft.irfft2(torch.fft.rfft2(img) * torch.fft.rfft2(k, s=img.shape), s=img.shape)
    return full[k.shape[0] - 1:, k.shape[1] - 1:]


def _spline_rows(n, u):
    """Weights (len(u), n) of a natural cubic spline through n unit-spaced knots at positions u."""
    a = np.zeros((n, n))
    d = np.zeros((n, n))
    a[0, 0] = a[-1, -1] = 1.0
    for i in range(1, n - 1):
        a[i, i - 1:i + 2] = 1 / 6, 4 / 6, 1 / 6
        d[i, i - 1:i + 2] = 1.0, -2.0, 1.0
    m = torch.as_tensor(np.linalg.solve(a, d), device=DEV)
    i = torch.clamp(torch.floor(u.detach()).to(torch.int64), 0, n - 2)
    b = (u - i)[:, None]
    e = torch.eye(n, dtype=torch.float64, device=DEV)
    w = (1 - b) * e[i] + b * e[i + 1] + (((1 - b) ** 3 - (1 - b)) * m[i] + (b ** 3 - b) * m[i + 1]) / 6.0
    inside = (u.detach() >= 0) & (u.detach() <= n - 1)
    return torch.where(inside[:, None], w, torch.zeros_like(w))


def _model(ins, lists, t, nodes=160):
    """The model image over the data pixels."""
    c = ins.case
    (y, x), *rest = _axes(ins)
    img = _valid(_grid_image(ins, y, x, lists[0], t, nodes), ins.psf)
    for f, sl in _slices(c):
        if f == "PointSource":  # the PSF, interpolated by a bicubic spline
            def rows(n, m, centre):
                u = torch.arange(1, m + 1, dtype=torch.float64, device=DEV) - centre + (n - 1) / 2.0
                return _spline_rows(n, u)
            psf = torch.as_tensor(ins.psf / ins.psf.sum(), device=DEV)
            img = img + t[sl][0] * (rows(c["psf_rows"], c["rows"], t[1]) @ psf @ rows(c["psf_cols"], c["cols"], t[0]).T)
    if rest:
        (ry, rx), k, (x1, x2, y1, y2) = rest[0], c["scale"], ins.region
        sub = _valid(_grid_image(ins, ry, rx, lists[1], t, nodes), ins.os_psf)
        block = sub.reshape(y2 - y1 + 1, k, x2 - x1 + 1, k).mean((1, 3))
        top = torch.cat([img[y1 - 1:y2, :x1 - 1], block, img[y1 - 1:y2, x2:]], 1)
        img = torch.cat([img[:y1 - 1], top, img[y2:]], 0)
    return img


class _Statistic:
    def __init__(self, ins):
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=DEV)
        self.kind, self.gain, self.sky = ins.case["stat"], ins.gain, ins.sky
        self.rn2 = (ins.read_noise / ins.gain) ** 2
        self.d = t(ins.data)
        good = torch.ones_like(self.d) if ins.mask is None else 1.0 - t(ins.mask)
        self.good = good
        if self.kind == "sigma":
            self.w = good / t(ins.sigma)
        elif self.kind == "chi2":
            self.w = good / torch.sqrt(torch.clamp(self.d + self.sky, min=0.0) / self.gain + self.rn2)
        dv = self.gain * (self.d + self.sky)
        safe = torch.where(dv > 0, dv, torch.ones_like(dv))
        self.extra = torch.where(dv > 0, dv * torch.log(safe) - dv, torch.zeros_like(dv))
        self.dv = dv

    def terms(self, m):
        mv = self.gain * (m + self.sky)
        extra = self.extra if self.kind == "pmlr" else 0.0
        return mv - self.dv * torch.log(mv) + extra

    def deviates(self, m):
        if self.kind in ("sigma", "chi2"):
            return self.w * (self.d - m)
        if self.kind == "model":
            return self.good * (self.d - m) / torch.sqrt((m + self.sky) / self.gain + self.rn2)
        a = 2.0 * torch.abs(self.terms(m))
        return self.good * torch.sqrt(torch.where(a > 0, a, torch.full_like(a, 1e-30)))

    def value(self, m):
        if self.kind in ("cash", "pmlr"):
            return 2.0 * (self.good * self.terms(m)).sum()
        return (self.deviates(m) ** 2).sum()


def _normal_equations(ins):
    """Statistic, J^T J and J^T dev, one tangent at a time."""
    p = torch.tensor(ins.params[0], device=DEV)
    lists, st = _lists(ins, ins.params[0]), _Statistic(ins)
    cols = []
    for j in range(p.numel()):
        e = torch.zeros_like(p)
        e[j] = 1.0
        dev, d = torch.func.jvp(lambda t: st.deviates(_model(ins, lists, t)).reshape(-1), (p,), (e,))
        cols.append(d)
    J = torch.stack(cols, 1)
    return (dev @ dev), J.T @ J, J.T @ dev


def exact(case, seed):
    call = case["call"]
    cpu = lambda v: v.detach().cpu().numpy()
    if call == "cutouts":
        out = [_normal_equations(_Inputs(c, seed, i)) for i, c in enumerate(_cutout_cases(case, seed))]
        return [torch.stack(v).cpu() for v in zip(*out)]
    ins = _Inputs(case, seed)
    if call == "jtwj":
        return [v.cpu() for v in _normal_equations(ins)]
    st = _Statistic(ins)
    S, G = [], []
    for row in ins.params:
        lists = _lists(ins, row)
        t = torch.tensor(row, device=DEV, requires_grad=call in ("grad", "plain_fd"))
        if call == "grad" and case["model"] == "edge_on_bar":
            # the gradient by chunks of rows: the adjoint image first, then each chunk's share of the sum
            with torch.no_grad():
                m = _model(ins, lists, t)
            m.requires_grad_(True)
            s = st.value(m)
            s.backward()
            pad = torch.nn.functional.pad(m.grad, (case["psf_cols"] - 1,) * 2 + (case["psf_rows"] - 1,) * 2)
            rt = _valid(pad, ins.psf[::-1, ::-1])
            (y, x), g = _axes(ins)[0], torch.zeros_like(t)
            for i in range(0, len(y), 16):
                part = _grid_image(ins, y[i:i + 16], x, lists[0], t, 160)
                g += torch.autograd.grad((part * rt[i:i + 16]).sum(), t)[0]
            S.append(float(s.detach()))
            G.append(cpu(g))
            continue
        m = _model(ins, lists, t)
        if call == "plain_dev":
            return cpu(st.deviates(m)).ravel()
        if call == "image":
            return cpu(m)
        s = st.value(m)
        S.append(float(s.detach()))
        if t.requires_grad:
            G.append(cpu(torch.autograd.grad(s, t)[0]))
    if call == "plain_stat":
        return S[0]
    if call == "plain_fd":
        return S[0], G[0]
    if case["batch"] == 1:
        S, G = S[0], G[0] if G else None
    else:
        S, G = np.array(S), np.array(G) if G else None
    return [torch.as_tensor(v, dtype=torch.float64) for v in (S, G) if v is not None]
