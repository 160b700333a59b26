"""The histograms of a Dr16 iteration do not depend on the order of their
terms: the same bits from forests in another order and from a second loop
on the same spectra. Their values against numpy's FP64 sums, with weights in
each of the ranges of the fixed-point sums and beyond (two-float terms: 1e-12
of the sum of the terms' magnitudes)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _grid(wave):
    from picca_gb300 import synthetic_spectra
    return synthetic_spectra.Grid(step=3e-4 if wave == "log" else 0.8, wave_solution=wave)


def _spectra(num, wave, seed=5):
    from picca_gb300 import continuum, synthetic_spectra
    raw = synthetic_spectra.make_raw_forests(num, seed, grid=_grid(wave))
    return raw, continuum.DeviceSpectra(raw, torch.device("cuda"))


def _permuted(raw, order):
    from picca_gb300 import continuum, synthetic_spectra
    off = raw.pix_offset
    pick = np.concatenate([np.arange(off[f], off[f + 1]) for f in order])
    out = synthetic_spectra.RawForests(
        pix_offset=np.concatenate([[0], np.cumsum(np.diff(off)[order])]), z_qso=raw.z_qso[order],
        los_id=raw.los_id[order], grid=raw.grid,
        **{k: getattr(raw, k)[pick] for k in ("log_lambda", "flux", "ivar",
                                              "transmission_correction")})
    return continuum.DeviceSpectra(out, torch.device("cuda"))


@pytest.mark.parametrize("parts", [dict(), dict(delta_stack=False), dict(mean_cont=False,
                                                                        var_stats=False)])
@pytest.mark.parametrize("wave", ["log", "lin"])
def test_order(wave, parts):
    from picca_gb300 import continuum
    raw, spectra = _spectra(3000, wave)
    other = _permuted(raw, np.random.default_rng(1).permutation(raw.num))
    got = []
    for s in (spectra, other, spectra):
        eng = continuum.Dr16Gpu(raw.grid, fit_mode=continuum.FIT_MIXED)
        got.append(eng._stacks(s, eng.fit(s), **parts))
    for sums in got[1:]:
        for key, value in got[0].items():
            assert np.array_equal(value, sums[key]), key


@pytest.mark.parametrize("wave", ["log", "lin"])
def test_loop(wave):
    from picca_gb300 import continuum
    _, spectra = _spectra(4000, wave)
    runs = []
    for _ in range(2):
        eng = continuum.Dr16Gpu(_grid(wave), num_iterations=3,
                                fit_mode=continuum.FIT_MIXED)
        fit = eng.run(spectra)
        delta, weights = eng.deltas(spectra, fit)
        runs.append([v.cpu().numpy() for v in (
            fit["zero_point"], fit["slope"], fit["chi2"], fit["iterations"], fit["continuum"],
            delta, weights)] + [eng.mean_cont_y, eng.eta, eng.var_lss, eng.fudge, eng.stack_y])
    for k, (a, b) in enumerate(zip(*runs)):
        assert np.array_equal(a, b, equal_nan=True), k


@pytest.mark.parametrize("eta", [1.0, 1e-6, 1e-16, 1e10, 1e18, 1e26])
def test_values(eta):
    from picca_gb300 import continuum
    raw, spectra = _spectra(800, "log")
    eng = continuum.Dr16Gpu(raw.grid)
    fit = eng.fit(spectra)
    eng.eta = np.full_like(eng.eta, eta)
    eng.var_lss = np.zeros_like(eng.var_lss)
    sums = eng._stacks(spectra, fit)
    out = continuum.fit_results_to_host(fit)
    npix = np.diff(raw.pix_offset)
    use = np.repeat(out["status"] == 0, npix) & (raw.ivar > 0)
    cont, iv, ratio = out["continuum"][use], raw.ivar[use], raw.flux[use] / out["continuum"][use]
    weight = iv * cont**2 / eta
    ll = raw.log_lambda[use]
    rest = raw.grid.find_bins(ll - np.repeat(np.log10(1 + raw.z_qso), npix)[use],
                              raw.grid.log_lambda_rest_frame_grid)
    obs = raw.grid.find_bins(ll, raw.grid.log_lambda_grid)
    for key, bins, term in (("mc_num", rest, ratio * weight), ("mc_w", rest, weight),
                            ("s_num", obs, ratio * weight), ("s_w", obs, weight)):
        n = sums[key].size
        want = np.bincount(bins, term, n)
        scale = np.bincount(bins, np.abs(term), n)
        assert scale.sum() > 0
        assert np.all(np.abs(sums[key] - want) <= 1e-12 * scale), key
