"""Workloads of the framework's device path, each through its public entry points.

The correlation of a survey comes first (neighbour lists, work order and
pair accumulation of ``PairEngine``: auto-correlation in both arithmetic
forms, both wavelength grids and both binnings, and the correlation with
quasars), then the continuum fit that makes its deltas (single fits, the whole
Dr16 loop, the warm-start network's forward pass and training step), and the
matrices of a correlation analysis (distortion, metals, Wick covariance) over
kept forest pairs. Inputs are the seeded synthetic surveys of
``picca_gb300.synthetic`` and ``synthetic_spectra`` at the benchmark's density
(50 forests and 75 quasars per square degree).
"""

import math

import numpy as np
import torch

from picca_gb300 import (constants, continuum, dmat, learned, metal, pairs, synthetic,
                         synthetic_spectra, wick)

FORESTS_PER_DEG2 = 50.0
BINS = 50
R_MAX = 200.0
Z_REF = 2.25
#: mean pixels of a synthetic forest (log grid of step 3e-4, 0.8 Angstrom grid)
MEAN_PIXELS = {"log": 185.0, "lin": 545.0}
#: pixels of a raw forest left by the sky and DLA masks
RAW_PIXELS = {"log": 160, "lin": 600}
METAL = "SiIII(1207)"
ALPHA = {"LYA": 2.9, METAL: 1.0}
LEARNING_RATE = 1e-3


def listed():
    return [
        # a healpix or a mock's corner: a call that launches and the last wave count in
        {"name": "auto_patch", "kind": "auto", "forests": 150, "grid": "log",
         "mode": "guard", "binning": "rprt"},
        # the ordinary work: a stretch of the eBOSS-like survey of the benchmark
        {"name": "auto_survey", "kind": "auto", "forests": 12000, "grid": "log",
         "mode": "guard", "binning": "rprt"},
        # DESI-like forests of up to 600 pixels on the 0.8 Angstrom grid
        {"name": "auto_linear_grid", "kind": "auto", "forests": 1501, "grid": "lin",
         "mode": "guard", "binning": "rprt"},
        # --precision fp64, the default of pairs.correlate, and the form that the
        # angular binning and the cuts of r-mu bins run in
        {"name": "auto_fp64", "kind": "auto", "forests": 331, "grid": "log",
         "mode": "fp64", "binning": "rprt"},
        # delta x quasar correlation (100 x 50 bins)
        {"name": "cross_quasars", "kind": "cross", "forests": 9000, "mode": "guard"},
        # one continuum fit of every forest in the default arithmetic of the plugin
        {"name": "fit_fp64", "kind": "fit", "forests": 20011, "grid": "log", "mode": "fp64"},
        # the continuum loop of a survey chunk in the benchmark's arithmetic, deltas included
        {"name": "dr16_loop", "kind": "dr16", "forests": 40000, "grid": "log",
         "mode": "mixed", "iterations": 3},
        # warm-start network: features of every forest and the forward pass
        {"name": "warm_start", "kind": "warm", "forests": 50021, "grid": "log"},
        # one training step of the warm-start network at the default batch
        {"name": "train_step", "kind": "train", "batch": 4096},
        # distortion matrix over kept forest pairs
        {"name": "dmat_pairs", "kind": "dmat", "forests": 500, "reject": 0.95},
        # metal matrix LYA x SiIII(1207), direct and swapped pass
        {"name": "metal_pairs", "kind": "metal", "forests": 500, "reject": 0.95},
        # Wick covariance (T1-T3) of the pairs of a kept forest
        {"name": "wick_pairs", "kind": "wick", "forests": 250, "kept": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["auto", "auto", "auto", "cross", "fit", "dr16", "warm", "train", "dmat",
                       "metal", "wick"])
    if kind == "auto":
        form = rng.choice(["guard", "guard", "guard", "lin", "rmu", "fp64"])
        top = {"guard": 12000, "lin": 1500, "rmu": 4000, "fp64": 330}[form]
        return {"kind": kind, "forests": _log_int(rng, 40, top),
                "grid": "lin" if form == "lin" else "log",
                "mode": "fp64" if form == "fp64" else "guard",
                "binning": "rmu" if form == "rmu" else "rprt"}
    if kind == "cross":
        return {"kind": kind, "forests": _log_int(rng, 100, 9000),
                "mode": rng.choice(["guard", "guard", "fp64"])}
    if kind == "fit":
        mode, grid = rng.choice(["fp64", "mixed"]), rng.choice(["log", "log", "lin"])
        top = 40000 if mode == "mixed" else 20000
        return {"kind": kind, "forests": _log_int(rng, 300, top if grid == "log" else top // 4),
                "grid": grid, "mode": mode}
    if kind == "dr16":
        return {"kind": kind, "forests": _log_int(rng, 2000, 40000), "grid": "log",
                "mode": rng.choice(["mixed", "mixed", "fp64"]), "iterations": rng.randint(2, 3)}
    if kind == "warm":
        return {"kind": kind, "forests": _log_int(rng, 200, 50000),
                "grid": rng.choice(["log", "log", "lin"])}
    if kind == "train":
        return {"kind": kind, "batch": _log_int(rng, 200, 16384)}
    if kind in ("dmat", "metal"):
        return {"kind": kind, "forests": rng.randint(60, 500),
                "reject": round(rng.uniform(0.95, 0.99), 3)}
    return {"kind": kind, "forests": rng.randint(60, 250), "kept": 1}


# -- inputs --------------------------------------------------------------------
def _box(forests):
    side = math.sqrt(forests / FORESTS_PER_DEG2)
    return (150.0, 150.0 + side), (-0.5 * side, 0.5 * side)


def _forests(case, seed):
    ra, dec = _box(case["forests"])
    return synthetic.make_forests(case["forests"], seed, ra, dec, 2.1, 4.0, "inv2",
                                  grid=case.get("grid", "log"))


def _quasars(case, seed):
    ra, dec = _box(case["forests"])
    return synthetic.make_quasars(max(1, int(1.5 * case["forests"])), seed + 1, ra, dec)


def _params(case, fs):
    cross = case["kind"] == "cross"
    rmu = case.get("binning") == "rmu"
    ang_max = synthetic.correlation_ang_max(R_MAX, float(fs.z.min()))
    return pairs.make_params(-R_MAX if cross else 0.0, 1.0 if rmu else R_MAX, R_MAX,
                             2 * BINS if cross else BINS, BINS, ang_max, x_correlation=cross,
                             rmu_binning=rmu)


def _raw(case, seed):
    """Raw forests with a tenth of their pixels masked at random (always the
    same number of pixels left)."""
    grid = synthetic_spectra.Grid()
    if case["grid"] == "lin":
        grid = synthetic_spectra.Grid(step=0.8, wave_solution="lin")
    raw = synthetic_spectra.make_raw_forests(case["forests"], seed, grid=grid)
    total, left = int(raw.pix_offset[-1]), case["forests"] * RAW_PIXELS[case["grid"]]
    keep = np.ones(total, dtype=bool)
    keep[np.random.default_rng(seed + 3).choice(total, total - left, replace=False)] = False
    raw.pix_offset = np.concatenate([[0], np.cumsum(keep)])[raw.pix_offset]
    for name in ("log_lambda", "flux", "ivar", "transmission_correction"):
        setattr(raw, name, getattr(raw, name)[keep])
    return raw


def _num_rows(case):
    """Rows for every healpix that the patch can touch."""
    area = case["forests"] / FORESTS_PER_DEG2
    return int(area / 13.4 + 2.0 * math.sqrt(area) + 9)


def _fit_mode(case):
    return continuum.FIT_MIXED if case["mode"] == "mixed" else continuum.FIT_FP64


def _kept_mask(case, seed, offsets):
    """The kept entries of the neighbour lists: single pairs (random
    rejection) or every neighbour of a few kept forests."""
    rng = np.random.default_rng(seed + 2)
    off = offsets.cpu().numpy()
    if case["kind"] != "wick":
        return rng.random(int(off[-1])) > case["reject"]
    keep = np.zeros(case["forests"], dtype=bool)
    keep[rng.choice(case["forests"], case["kept"], replace=False)] = True
    return np.repeat(keep, np.diff(off))


def _cf1d():
    """A 1D correlation table: 1,000 offsets of 3e-4 in log10(lambda)."""
    k = np.arange(1000)
    ones = np.ones(k.size, dtype=np.int64)
    return {"LLMIN": float(np.log10(3600.0)), "DLL": 3e-4, "v1d": 0.1 + 0.05 * np.sin(k / 60.0),
            "nv1d": ones, "c1d": np.where(k == 0, 1.0, -0.015 * np.exp(-k / 40.0)),
            "nb1d": ones}


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("auto", "cross"):
        fs = _forests(case, seed)
        engine = pairs.PairEngine()
        qs = _quasars(case, seed) if kind == "cross" else None
        return {"kind": kind, "engine": engine, "params": _params(case, fs),
                "num_rows": _num_rows(case),
                "mode": pairs.MODE_FP64 if case["mode"] == "fp64" else pairs.MODE_FP32_GUARD,
                "forests": pairs.DeviceForests(fs),
                "quasars": pairs.DeviceForests(qs) if qs is not None else None}
    if kind in ("fit", "dr16", "warm"):
        raw = _raw(case, seed)
        spectra = continuum.DeviceSpectra(raw, torch.device("cuda"))
        state = {"kind": kind, "spectra": spectra, "grid": raw.grid}
        if kind == "dr16":
            state.update(mode=_fit_mode(case), iterations=case["iterations"])
        else:
            mode = _fit_mode(case) if kind == "fit" else continuum.FIT_MIXED
            state["engine"] = continuum.Dr16Gpu(raw.grid, fit_mode=mode)
        if kind == "warm":
            state["network"] = learned.WarmStartMLP(seed=seed % 1000)
        return state
    if kind == "train":
        gen = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.zeros(case["batch"], learned.FEATURE_STRIDE, device="cuda")
        x[:, :learned.NUM_FEATURES] = 0.5 * torch.randn(case["batch"], learned.NUM_FEATURES,
                                                        device="cuda", generator=gen)
        target = 0.3 * torch.randn(case["batch"], learned.NUM_OUT, device="cuda", generator=gen)
        return {"kind": kind, "network": learned.WarmStartMLP(seed=seed % 1000),
                "x": x.bfloat16(), "target": target}
    fs = _forests(case, seed)
    params = _params(case, fs)
    if kind == "wick":
        engine = wick.WickEngine()
        dev = pairs.DeviceForests(fs, compact=False)
    else:
        engine = metal.MetalEngine() if kind == "metal" else dmat.DmatEngine()
        dev = pairs.DeviceForests(fs)
    offsets, index, _ = engine.engine.neighbours(params, dev)
    mask = _kept_mask(case, seed, offsets)
    state = {"kind": kind, "engine": engine, "params": params, "forests": dev}
    if kind == "wick":
        first, second, num = wick.forest_pairs(dev, offsets, index, mask)
        state["used"] = np.unique(torch.cat([first[:num], second[:num]]).cpu().numpy())
        state["tables"] = wick.OneDTables(_cf1d())
        state["evolution"] = torch.from_numpy(wick.evolution(fs.z, Z_REF, 2.9)).cuda()
    else:
        first, second, num = engine.pair_list(dev, None, offsets, index, mask)
        state["dparams"] = dmat.make_dmat_params(BINS, BINS)
        if kind == "dmat":
            state["side"] = engine.side_arrays(dev, engine.device)
        else:
            cosmo = constants.Cosmo(Om=0.3147, verbose=False)
            state["sides"] = [metal.absorber_pixels(dev, cosmo, name, ALPHA[name])
                              for name in ("LYA", METAL)]
    state["pairs"] = (first, second, num)
    return state


# -- one pass ------------------------------------------------------------------
def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_auto(state):
    engine, params = state["engine"], state["params"]
    dev, other = state["forests"], state.get("quasars")
    cross = other is not None
    offsets, index, total = engine.neighbours(params, dev, other, xcf=cross)
    order, num_work, _ = engine.work_order(dev, other, offsets, index, total, xcf=cross)
    rows = engine.alloc_rows(state["num_rows"], params.num_bins_r_par * params.num_bins_r_trans)
    engine.accumulate(params, dev, other, offsets, index, order, num_work, rows, state["mode"],
                      xcf=cross)
    engine.stats()
    return {"rows": rows, "offsets": offsets}


_run_cross = _run_auto


def _fit_outputs(fit):
    return {k: v for k, v in fit.items() if k != "_keep"}


def _run_fit(state):
    return _fit_outputs(state["engine"].fit(state["spectra"]))


def _run_dr16(state):
    engine = continuum.Dr16Gpu(state["grid"], num_iterations=state["iterations"],
                               fit_mode=state["mode"])
    fit = engine.run(state["spectra"])
    delta, weights = engine.deltas(state["spectra"], fit)
    return {"fit": _fit_outputs(fit), "delta": delta, "weights": weights,
            "mean_cont": engine.mean_cont_y, "eta": engine.eta, "var_lss": engine.var_lss,
            "fudge": engine.fudge, "stack": engine.stack_y}


def _run_warm(state):
    engine, spectra = state["engine"], state["spectra"]
    model, _keep = engine._model()
    feat, a0 = learned.features(engine, spectra, model)
    return {"features": feat, "a0": a0, "y": state["network"].forward_fused(feat)}


def _run_train(state):
    net, target = state["network"], state["target"]
    y, acts = net.forward(state["x"], keep=True)
    loss = net.backward(acts, y, target)
    net.adam_step(lr=LEARNING_RATE)
    return {"y": y, "loss": loss, "grads": net.grads, "params": net.params, "m1": net.m1,
            "m2": net.m2}


def _run_dmat(state):
    engine, params, dparams = state["engine"], state["params"], state["dparams"]
    first, second, num = state["pairs"]
    sums = engine.alloc_sums(params, dparams)
    return engine.accumulate(params, dparams, state["forests"], None, state["side"], None, first,
                             second, num, sums)


def _metal_den():
    return (1 + Z_REF) ** (ALPHA["LYA"] + ALPHA[METAL] - 2)


def _run_metal(state):
    engine, params, dparams = state["engine"], state["params"], state["dparams"]
    first, second, num = state["pairs"]
    lya, si = state["sides"]
    sums = engine.alloc_sums(params, dparams)
    for one, two in ((lya, si), (si, lya)):
        engine.run_pass(params, dparams, _metal_den(), state["forests"], None, one, two, first,
                        second, num, sums)
    return sums


def _run_wick(state):
    engine, params, dev = state["engine"], state["params"], state["forests"]
    first, second, num = state["pairs"]
    arena, offsets, _keep = engine.xi_matrices(dev, state["tables"], state["used"])
    sums = engine.alloc_sums(params.num_bins_r_par * params.num_bins_r_trans)
    zw = state["evolution"]
    return engine.accumulate(params, dev, zw, zw, offsets, arena, first, second, num, sums)


# -- what a pass cannot do without -----------------------------------------------
def _near_fraction(forests, angle_deg):
    """Fraction of pairs of points of a square that are closer than angle."""
    t = angle_deg / math.sqrt(forests / FORESTS_PER_DEG2)
    if t <= 1.0:
        return math.pi * t * t - 8.0 / 3.0 * t**3 + 0.5 * t**4
    return min(1.0, 0.975 + 0.025 * (t - 1.0) / 0.414)


def _candidates(case):
    """Expected candidate pixel pairs of the correlation of a case."""
    n = case["forests"]
    near = _near_fraction(n, 3.2)
    if case["kind"] == "cross":
        return 0.6 * 1.5 * n * n * near * MEAN_PIXELS["log"]
    return 0.5 * n * n * near * MEAN_PIXELS[case.get("grid", "log")] ** 2


def work(case):
    kind = case["kind"]
    if kind in ("auto", "cross"):
        n, cand = case["forests"], _candidates(case)
        nbins = BINS * BINS * (2 if kind == "cross" else 1)
        rows = max(1.0, n / FORESTS_PER_DEG2 / 13.4)
        inputs = n * (MEAN_PIXELS[case.get("grid", "log")] * 40 + 120)
        # 10 flops per candidate (distances, bins, weight), 9 per accepted pair
        return {"bytes": inputs + rows * nbins * 48, "flops": cand * (10 + 9 * 0.55)}
    if kind in ("fit", "dr16", "warm"):
        pixels = case["forests"] * RAW_PIXELS[case["grid"]]
        if kind == "warm":
            layers = sum(a * b for a, b in learned.WarmStartMLP.SHAPES)
            return {"bytes": pixels * 32 + case["forests"] * 16,
                    "flops": 2.0 * layers * case["forests"]}
        passes = case.get("iterations", 1)
        # about 60 flops per pixel and Newton step, five steps a fit
        return {"bytes": passes * (pixels * 40 + case["forests"] * 32) +
                (pixels * 56 if kind == "dr16" else 0), "flops": passes * pixels * 300}
    if kind == "train":
        layers = sum(a * b for a, b in learned.WarmStartMLP.SHAPES)
        return {"bytes": case["batch"] * 170 + layers * 32, "flops": 6.0 * layers * case["batch"]}
    n, pix2 = case["forests"], MEAN_PIXELS["log"] ** 2
    inputs = n * MEAN_PIXELS["log"] * 56
    if kind == "wick":
        units = case["kept"] * 0.5 * n
        listed_pairs = 0.5 * pix2
        return {"bytes": inputs + 3 * (BINS * BINS) ** 2 * 8,
                "flops": units * listed_pairs * listed_pairs}
    kept = 0.5 * n * n * (1 - case["reject"])
    out = (BINS * BINS) ** 2 * 8
    if kind == "metal":
        return {"bytes": inputs + out, "flops": 2 * kept * pix2 * 40}
    # the eta products: about 140 data bins x 140 model bins x 740 terms a pair
    return {"bytes": inputs + out, "flops": kept * (2.0 * 140 * 140 * 740 + 60 * pix2)}


# -- the same in 64 bits -----------------------------------------------------------
def exact(case, seed):
    """What run() returns, by plain torch in 64 bits; None where that takes
    too long."""
    kind = case["kind"]
    if kind in ("auto", "cross"):
        return _exact_rows(case, seed) if _candidates(case) < 4e9 else None
    if kind == "fit":
        return _exact_fit(case, seed)
    if kind == "dr16":
        return None  # three passes of histograms and spline fits
    if kind == "warm":
        return _exact_warm(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    return globals()["_exact_" + kind](case, seed)


def _cuda(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def _angles(fs, f, other):
    dot = (other["x_cart"] * float(fs.x_cart[f]) + other["y_cart"] * float(fs.y_cart[f]) +
           other["z_cart"] * float(fs.z_cart[f]))
    ang = torch.acos(dot.clamp(-1.0, 1.0))
    dra, ddec = other["ra"] - float(fs.ra[f]), other["dec"] - float(fs.dec[f])
    flat = torch.sqrt(ddec**2 + (float(fs.cos_dec[f]) * dra) ** 2)
    tiny = 2.0 / 3600.0 * math.pi / 180.0
    return torch.where((dra.abs() < tiny) & (ddec.abs() < tiny), flat, ang)


def _sky(fs):
    return {k: _cuda(getattr(fs, k)) for k in ("x_cart", "y_cart", "z_cart", "ra", "dec")}


def _pixels(fs):
    return {k: _cuda(getattr(fs, k)) for k in ("z", "r_comov", "dist_m", "weights", "delta",
                                               "log_lambda")}


def _exact_rows(case, seed):
    fs = _forests(case, seed)
    cross, rmu = case["kind"] == "cross", case.get("binning") == "rmu"
    p = _params(case, fs)
    n_p, n_t = p.num_bins_r_par, p.num_bins_r_trans
    nbins, num_rows = n_p * n_t, _num_rows(case)
    out = torch.zeros(5, num_rows, nbins, dtype=torch.float64, device="cuda")
    pix, off = _pixels(fs), fs.pix_offset
    if cross:
        qs = _quasars(case, seed)
        sky = _sky(qs)
        two = {"z": _cuda(qs.z_qso), "r_comov": _cuda(qs.obj_r_comov),
               "dist_m": _cuda(qs.obj_dist_m), "weights": _cuda(qs.obj_weight)}
        start2, size2 = torch.arange(qs.num, device="cuda"), torch.ones(qs.num, device="cuda",
                                                                        dtype=torch.int64)
    else:
        sky, two = _sky(fs), pix
        start2, size2 = _cuda(off[:-1]), _cuda(np.diff(off))
    for f in range(fs.num):
        ang = _angles(fs, f, sky)
        near = ang < p.ang_max
        if not cross:
            near &= sky["ra"] < float(fs.ra[f])
        g = torch.nonzero(near).flatten()
        n1 = int(off[f + 1] - off[f])
        if g.numel() == 0 or n1 == 0:
            continue
        sizes = size2[g]
        first = torch.repeat_interleave(start2[g] - (torch.cumsum(sizes, 0) - sizes), sizes)
        j = first + torch.arange(first.numel(), device="cuda")
        half = torch.repeat_interleave(ang[g] / 2, sizes)
        one = {k: v[off[f]:off[f + 1], None] for k, v in pix.items()}
        r_par = (one["r_comov"] - two["r_comov"][j]) * torch.cos(half)
        r_trans = (one["dist_m"] + two["dist_m"][j]) * torch.sin(half)
        if rmu:
            r_trans = torch.sqrt(r_trans**2 + r_par**2)
            r_par = r_par / r_trans
        if not cross:
            r_par = r_par.abs()
        ok = (r_par < p.r_par_max) & (r_trans < p.r_trans_max)
        ok &= (r_par > p.r_par_min) if cross else (r_par >= p.r_par_min)
        w12 = one["weights"] * two["weights"][j]
        d12 = one["delta"] * w12 if cross else one["delta"] * w12 * two["delta"][j]
        z = (one["z"] + two["z"][j]) / 2
        bins = (torch.floor(r_trans / p.r_trans_max * n_t) +
                n_t * torch.floor((r_par - p.r_par_min) / (p.r_par_max - p.r_par_min) * n_p))
        bins = bins[ok].long()
        w = w12[ok]
        row = out[:, int(fs.row[f])]
        for k, v in enumerate((w, d12[ok], r_par[ok] * w, r_trans[ok] * w, z[ok] * w)):
            row[k] += torch.bincount(bins, weights=v, minlength=nbins)
    return {"rows": [v.reshape(-1) for v in out] + [None], "offsets": None}


def _padded(case, seed):
    """Spectra of a case as padded [forests, pixels] FP64 arrays."""
    raw = _raw(case, seed)
    npix = torch.as_tensor(np.diff(raw.pix_offset), device="cuda")
    have = torch.arange(int(npix.max()), device="cuda")[None, :] < npix[:, None]
    out = {"have": have, "z_qso": _cuda(raw.z_qso)}
    for k in ("log_lambda", "flux", "ivar", "transmission_correction"):
        v = torch.zeros(have.shape, dtype=torch.float64, device="cuda")
        v[have] = _cuda(getattr(raw, k))
        out[k] = v
    rest = raw.grid.log_lambda_rest_frame_grid
    zp1 = torch.log10(1 + out["z_qso"])[:, None]
    out["x"] = (out["log_lambda"] - (rest[0] + zp1)) / (rest[-1] - rest[0])
    return raw, out


def _exact_fit(case, seed):
    """Damped Newton on sum (f - C)^2 / D + log D with C = a + b x and
    D = 1 / ivar + 0.1 C^2 (the model a new loop starts from)."""
    _, s = _padded(case, seed)
    use = (s["ivar"] > 0) & s["have"]
    iv = torch.where(use, s["ivar"], 1.0)
    f, x, mc = s["flux"], s["x"], s["transmission_correction"]

    def terms(a, b):
        c = (a[:, None] + b[:, None] * x) * mc
        d = 1.0 / iv + 0.1 * c * c
        dd, d2d, r = 0.2 * c, 0.2, f - c
        val = r * r / d + torch.log(d)
        g = -2 * r / d - (r / d) ** 2 * dd + dd / d
        h = (2 / d + 4 * r / d * dd / d + 2 * (r / d) ** 2 * dd * dd / d - (r / d) ** 2 * d2d +
             d2d / d - (dd / d) ** 2)
        ja, jb = mc, x * mc
        return [torch.where(use, v, 0.0).sum(1) for v in
                (val, g * ja, g * jb, h * ja * ja, h * ja * jb, h * jb * jb)]

    a = (torch.where(use, f * iv, 0.0)).sum(1) / torch.where(use, iv, 0.0).sum(1)
    b = torch.zeros_like(a)
    cur = terms(a, b)
    for _ in range(40):
        det = cur[3] * cur[5] - cur[4] ** 2
        scale = torch.maximum(cur[3].abs(), cur[5].abs())
        da = -(cur[5] * cur[1] - cur[4] * cur[2]) / det
        db = -(cur[3] * cur[2] - cur[4] * cur[1]) / det
        bad = ~((det > 0) & (cur[3] > 0)) | (da * cur[1] + db * cur[2] >= 0)
        da, db = torch.where(bad, -cur[1] / scale, da), torch.where(bad, -cur[2] / scale, db)
        slope = da * cur[1] + db * cur[2]
        t = torch.ones_like(a)
        for _ in range(12):
            new = terms(a + t * da, b + t * db)
            worse = ~(new[0] <= cur[0] + 1e-4 * t * slope)
            if not bool(worse.any()):
                break
            t = torch.where(worse, t / 2, t)
        better = new[0] <= cur[0]
        a, b = torch.where(better, a + t * da, a), torch.where(better, b + t * db, b)
        cur = terms(a, b)
    cont = (a[:, None] + b[:, None] * x) * mc
    bad = ((cont < 0) & s["have"]).any(1)
    nan = torch.full_like(a, math.nan)
    return {"zero_point": torch.where(bad, nan, a), "slope": torch.where(bad, nan, b),
            "chi2": torch.where(bad, nan, cur[0]), "ndata": None, "status": None,
            "iterations": None, "continuum": cont[s["have"]]}


def _layers(net):
    """(weights, bias) of each layer in FP64, the weights as the BF16 products see them."""
    out, at = [], 0
    for fan_in, fan_out in net.SHAPES:
        w = net.params[at:at + fan_in * fan_out].bfloat16().double().view(fan_in, fan_out)
        at += fan_in * fan_out
        out.append((w, net.params[at:at + fan_out].double()))
        at += fan_out
    return out


def _exact_warm(case, seed):
    """The features are BF16 results of their own; a0 and the network on the
    features of the pass are computed numbers."""
    _, s = _padded(case, seed)
    iv = torch.where(s["have"], s["ivar"], 0.0)
    state = prepare(case, seed)
    model, _keep = state["engine"]._model()
    feat, _ = learned.features(state["engine"], state["spectra"], model)
    h = feat.double()[:, :learned.NUM_FEATURES]
    layers = _layers(state["network"])
    for k, (w, bias) in enumerate(layers):
        h = h @ w + bias
        if k + 1 < len(layers):
            h = torch.nn.functional.gelu(h)
    return {"features": None, "a0": (s["flux"] * iv).sum(1) / iv.sum(1), "y": h}


def _exact_train(case, seed):
    state = prepare(case, seed)
    net, m = state["network"], case["batch"]
    layers = _layers(net)
    leaves = [t.clone().requires_grad_(True) for pair in layers for t in pair]
    h = state["x"].double()[:, :learned.NUM_FEATURES]
    for k in range(len(layers)):
        h = h @ leaves[2 * k] + leaves[2 * k + 1]
        if k + 1 < len(layers):
            h = torch.nn.functional.gelu(h)
    loss = ((h - state["target"].double()) ** 2).sum() / m
    grads = torch.autograd.grad(loss, leaves)
    g = torch.cat([v.reshape(-1) for v in grads])
    m1, m2 = 0.1 * g, 0.001 * g * g
    params = net.params.double() - LEARNING_RATE * (m1 / 0.1) / (torch.sqrt(m2 / 0.001) + 1e-8)
    return {"y": h.detach(), "loss": loss.detach().reshape(1), "grads": g, "params": params,
            "m1": m1, "m2": m2}


def _pair_geometry(fs, f, g):
    """cos and sin of half the angle between two forests."""
    dot = (fs.x_cart[f] * fs.x_cart[g] + fs.y_cart[f] * fs.y_cart[g] +
           fs.z_cart[f] * fs.z_cart[g])
    half = math.acos(min(1.0, max(-1.0, dot))) / 2
    return math.cos(half), math.sin(half)


def _bin(r_par, r_trans):
    """Bin of r_par, r_trans (0 to R_MAX, BINS bins each) and whether it is in range."""
    bp, bt = torch.floor(r_par / R_MAX * BINS), torch.floor(r_trans / R_MAX * BINS)
    return (bt + BINS * bp).long(), (r_par < R_MAX) & (r_trans < R_MAX)


def _kept_pairs(case, seed):
    first, second, num = prepare(case, seed)["pairs"]
    return list(zip(first[:num].tolist(), second[:num].tolist()))


def _new_sums(*names):
    nb = BINS * BINS
    return {k: torch.zeros(nb * nb if k in ("dmat", "t1", "t2", "t3") else nb,
                           dtype=torch.float64, device="cuda") for k in names}


def _exact_metal(case, seed):
    fs = _forests(case, seed)
    cosmo = constants.Cosmo(Om=0.3147, verbose=False)
    pix, off, nb = _pixels(fs), fs.pix_offset, BINS * BINS
    out = _new_sums("weights_dmat", "dmat", "r_par_eff", "r_trans_eff", "z_eff", "weight_eff")
    z_qso = np.repeat(fs.z_qso, np.diff(off))
    sides = []
    for name in ("LYA", METAL):
        z = 10**fs.log_lambda / constants.ABSORBER_IGM[name] - 1
        sides.append({"r": _cuda(cosmo.get_r_comov(z)), "d": _cuda(cosmo.get_dist_m(z)),
                      "z": _cuda(z), "f": _cuda((1 + z) ** (ALPHA[name] - 1)),
                      "w": _cuda(np.where(z < z_qso, fs.weights, 0.0))})
    for f, g in _kept_pairs(case, seed):
        c, s = _pair_geometry(fs, f, g)
        a, b = slice(off[f], off[f + 1]), slice(off[g], off[g + 1])
        bins, ok0 = _bin(((pix["r_comov"][a, None] - pix["r_comov"][b]) * c).abs(),
                         (pix["dist_m"][a, None] + pix["dist_m"][b]) * s)
        for one, two in (sides, sides[::-1]):
            w = one["w"][a, None] * two["w"][b]
            out["weights_dmat"].index_add_(0, bins[ok0], w[ok0])
            rp = ((one["r"][a, None] - two["r"][b]) * c).abs()
            rt = (one["d"][a, None] + two["d"][b]) * s
            model, ok = _bin(rp, rt)
            ok &= ok0
            m, wz = model[ok], (w * one["f"][a, None] * two["f"][b] / _metal_den())[ok]
            out["dmat"].index_add_(0, bins[ok] * nb + m, wz)
            z = (one["z"][a, None] + two["z"][b]) / 2
            for key, v in (("r_par_eff", rp[ok] * wz), ("r_trans_eff", rt[ok] * wz),
                           ("z_eff", z[ok] * wz), ("weight_eff", wz)):
                out[key].index_add_(0, m, v)
    return out


def _exact_dmat(case, seed):
    fs = _forests(case, seed)
    pix, off, nb = _pixels(fs), fs.pix_offset, BINS * BINS
    out = _new_sums("weights_dmat", "dmat", "r_par_eff", "r_trans_eff", "z_eff", "weight_eff")
    dmat_2d = out["dmat"].view(nb, nb)
    evolution = ((1 + pix["z"]) / (1 + Z_REF)) ** 1.9
    for f, g in _kept_pairs(case, seed):
        c, s = _pair_geometry(fs, f, g)
        a, b = slice(off[f], off[f + 1]), slice(off[g], off[g + 1])
        rp = ((pix["r_comov"][a, None] - pix["r_comov"][b]) * c).abs()
        rt = (pix["dist_m"][a, None] + pix["dist_m"][b]) * s
        bins, ok = _bin(rp, rt)
        i, j = torch.nonzero(ok, as_tuple=True)
        if i.numel() == 0:
            continue
        bins = bins[ok]
        w1, w2 = pix["weights"][a], pix["weights"][b]
        d1 = pix["log_lambda"][a] - (pix["log_lambda"][a] * w1).sum() / w1.sum()
        d2 = pix["log_lambda"][b] - (pix["log_lambda"][b] * w2).sum() / w2.sum()
        # mean and slope weights of each pixel in the projection of its forest
        m1, s1 = w1 / w1.sum(), w1 * d1 / (w1 * d1 * d1).sum()
        m2, s2 = w2 / w2.sum(), w2 * d2 / (w2 * d2 * d2).sum()
        zf = evolution[a][i] * evolution[b][j]
        w12 = w1[i] * w2[j]
        z = (pix["z"][a][i] + pix["z"][b][j]) / 2
        for key, v in (("weights_dmat", w12), ("weight_eff", w12), ("r_par_eff", w12 * rp[ok]),
                       ("r_trans_eff", w12 * rt[ok]), ("z_eff", w12 * z)):
            out[key].index_add_(0, bins, v)
        used, k = torch.unique(bins, return_inverse=True)
        nu, n1, n2 = used.numel(), w1.numel(), w2.numel()

        def spread(cols, col, v):
            t = torch.zeros(nu * cols, dtype=torch.float64, device="cuda")
            return t.index_add_(0, k * cols + col, v).view(nu, cols)

        one = torch.zeros_like(i)
        d = torch.diag(spread(1, one, w12 * zf).flatten())
        for value, eta in ((w12, m1[i] * m2[j]), (w12 * d2[j], m1[i] * s2[j]),
                           (w12 * d1[i], s1[i] * m2[j]), (w12 * d1[i] * d2[j], s1[i] * s2[j])):
            d += spread(1, one, value) @ spread(1, one, zf * eta).T
        d -= spread(n1, i, w12) @ spread(n1, i, zf * m2[j]).T
        d -= spread(n2, j, w12) @ spread(n2, j, zf * m1[i]).T
        d -= spread(n1, i, w12 * d2[j]) @ spread(n1, i, zf * s2[j]).T
        d -= spread(n2, j, w12 * d1[i]) @ spread(n2, j, zf * s1[i]).T
        dmat_2d[used[:, None], used] += d
    return out


def _exact_wick(case, seed):
    fs = _forests(case, seed)
    pix, off, nb = _pixels(fs), fs.pix_offset, BINS * BINS
    table = _cf1d()
    log_lambda = table["LLMIN"] + table["DLL"] * np.arange(1000)
    out = _new_sums("weights_wick", "t1", "t2", "t3")
    zw = ((1 + pix["z"]) / (1 + Z_REF)) ** 1.9

    def nearest(x, y, v):
        bounds = _cuda(x[1:] / 2 + x[:-1] / 2)
        return _cuda(y)[torch.searchsorted(bounds, v.contiguous())]

    def matrix(sl):
        ll, w = pix["log_lambda"][sl], pix["weights"][sl]
        var = nearest(log_lambda, table["v1d"], ll)
        xi = nearest(log_lambda - table["LLMIN"], table["c1d"], (ll[:, None] - ll).abs())
        x = w[:, None] * w * xi * torch.sqrt(var[:, None] * var)
        return x * (1 - torch.eye(ll.numel(), dtype=torch.float64, device="cuda"))

    for f, g in _kept_pairs(case, seed):
        c, s = _pair_geometry(fs, f, g)
        a, b = slice(off[f], off[f + 1]), slice(off[g], off[g + 1])
        bins, ok = _bin(((pix["r_comov"][a, None] - pix["r_comov"][b]) * c).abs(),
                        (pix["r_comov"][a, None] + pix["r_comov"][b]) * s)
        i, j = torch.nonzero(ok, as_tuple=True)
        if i.numel() == 0:
            continue
        bins = bins[ok]
        w12 = pix["weights"][a][i] * pix["weights"][b][j]
        out["weights_wick"].index_add_(0, bins, w12)
        out["t1"].index_add_(0, bins * (nb + 1), w12 * zw[a][i] * zw[b][j])
        used, k = torch.unique(bins, return_inverse=True)
        n1, n2 = ok.shape
        member = torch.zeros(used.numel(), n1, n2, dtype=torch.float64, device="cuda")
        member[k, i, j] = 1.0
        x1, x2 = matrix(a), matrix(b)
        right = member @ x2                            # sum over the partners in forest 2
        left = torch.einsum("ik,pkj->pij", x1, member)  # and in forest 1
        c1, c2 = pix["weights"][a] * zw[a], pix["weights"][b] * zw[b]
        t2 = (torch.einsum("pij,qij->pq", right * c1[:, None], member) +
              torch.einsum("pij,qij->pq", left * c2, member))
        t3 = right.reshape(used.numel(), -1) @ left.reshape(used.numel(), -1).T
        for key, v in (("t2", t2), ("t3", t3)):
            out[key].view(nb, nb)[used[:, None], used] += v
    out["num_pairs_wick"] = None
    return out
