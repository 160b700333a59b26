"""The FP64 continuum fit where its forms can go wrong: forests around 32, 224
(the short form's limit) and 1,024 pixels, mixed in one call and fitted through
an index list, masked pixels, a forest without a usable pixel, orders 0 and 1,
with and without a fudge term. Against the FP64 oracle's chi2 at the point that
comes back (1e-11 relative, sums of a thousand FP64 terms), whose gradient
vanishes there (1e-6 of the gradient's own terms, what a step of 1e-10 of the
scale leaves)."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _raw(lengths, seed):
    from picca_gb300 import synthetic_spectra
    grid = synthetic_spectra.Grid(step=0.8, wave_solution="lin")
    raw = synthetic_spectra.make_raw_forests(len(lengths), seed, grid=grid, z_lo=2.9, z_hi=3.4)
    rng = np.random.default_rng(seed)
    cols = {k: [] for k in ("log_lambda", "flux", "ivar", "transmission_correction")}
    for f, n in enumerate(lengths):
        o = int(raw.pix_offset[f])
        have = int(raw.pix_offset[f + 1]) - o
        take = o + np.sort(rng.integers(0, have, n))  # repeats where the forest is shorter
        for k in cols:
            cols[k].append(getattr(raw, k)[take])
        bad = rng.random(n) < 0.1
        cols["ivar"][-1] = np.where(bad, 0.0, cols["ivar"][-1])
    cols["ivar"][-1][:] = 0.0
    for k, v in cols.items():
        setattr(raw, k, np.concatenate(v))
    raw.pix_offset = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    return raw


@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("fudge", [0.0, 1e-3])
def test_lengths(order, fudge):
    from picca_gb300 import continuum
    lengths = [5, 31, 32, 33, 64, 223, 224, 225, 256, 500, 1023, 1024, 100]
    raw = _raw(lengths, 4)
    eng = continuum.Dr16Gpu(raw.grid, order=order, fit_mode=continuum.FIT_FP64)
    x = eng.var_x
    eng.eta, eng.var_lss = 1.0 + 0.1 * np.sin(9 * x), 0.1 + 0.02 * np.cos(7 * x)
    eng.fudge = np.full_like(x, fudge)
    eng.mean_cont_y = 1.0 + 0.2 * np.sin(30 * eng.mean_cont_x)
    spectra = continuum.DeviceSpectra(raw, eng.device)
    fit = eng.fit(spectra)
    index = torch.tensor([11, 2, 7, 12, 0, 5], dtype=torch.int32)
    part = eng.fit(spectra, index=index)
    pick = index.long().cuda()
    for key in ("zero_point", "slope", "chi2", "ndata", "status", "iterations"):
        assert torch.equal(torch.nan_to_num(part[key].double()[pick], nan=-1.0),
                           torch.nan_to_num(fit[key].double()[pick], nan=-1.0)), key
    out = continuum.fit_results_to_host(fit)
    assert list(out["status"][:-1]) == [0] * (len(lengths) - 1)
    from scipy.interpolate import interp1d
    eta, vlss, fud = (interp1d(x, y, kind="cubic", fill_value="extrapolate")
                      for y in (eng.eta, eng.var_lss, eng.fudge))
    mean = interp1d(eng.mean_cont_x, eng.mean_cont_y, fill_value="extrapolate")
    rest = raw.grid.log_lambda_rest_frame_grid
    for f in range(len(lengths) - 1):
        sl = slice(raw.pix_offset[f], raw.pix_offset[f + 1])
        ll, flux, iv = raw.log_lambda[sl], raw.flux[sl], raw.ivar[sl]
        zp1 = np.log10(1 + raw.z_qso[f])
        mc = mean(ll - zp1) * raw.transmission_correction[sl]
        u = (ll - rest[0] - zp1) / (rest[-1] - rest[0])
        a, b = out["zero_point"][f], out["slope"][f]
        cont = (b * u + a) * mc
        assert np.allclose(out["continuum"][sl], cont, rtol=1e-12, atol=0)
        ok = iv > 0
        c, i = cont[ok], iv[ok]
        d = eta(ll[ok]) / i + vlss(ll[ok]) * c**2 + fud(ll[ok]) * i * c**4
        r = flux[ok] - c
        terms = r * r / d + np.log(d)
        assert abs(out["chi2"][f] - terms.sum()) <= 1e-11 * np.abs(terms).sum()
        dd = 2 * vlss(ll[ok]) * c + 4 * fud(ll[ok]) * i * c**3
        g = -2 * r / d - (r / d) ** 2 * dd + dd / d
        for jac in (mc[ok], u[ok] * mc[ok])[:order + 1]:
            assert abs((g * jac).sum()) <= 1e-6 * np.abs(g * jac).sum()
        assert out["ndata"][f] == ok.sum()
